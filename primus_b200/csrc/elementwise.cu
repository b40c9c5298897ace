// Memory-bound training ops for sm_100a: RoPE, SwiGLU (plain / routing-prob weighted / clamped), cross-entropy (fused
// softmax + gradient, vocab-parallel capable), AdamW on flat buffers, L2-norm / scale helpers, MoE row movement.  (RMSNorm:
// csrc/rmsnorm.cu.)
//
// All kernels move 16 bytes per thread per access and keep fp32 math in registers; each is one
// pass over its operands except where a row statistic forces a second read (which hits L1/L2).
//
// Reference call sites these replace: TE fused RoPE and bias-SwiGLU (primus/backends/megatron/patches/te_patches/
// fused_bias_swiglu_patches.py:21), swiglu_with_probs (primus_turbo.py:1954-1980), clamped SwiGLU
// (primus/backends/megatron/core/fusions/fused_bias_swiglu.py:25-100), TE cross-entropy fusion
// and FusedAdam (primus/backends/megatron/patches/torch_fused_adam_patches.py:40-88).
#include "div_invariant.h"
#include "vec.cuh"

namespace {

using pb::Bf8;
using pb::bf8_to_f;
using pb::block_max;
using pb::block_sum;
using pb::div_invariant;
using pb::f_to_bf8;

// ------------------------------------------------------------------ logit soft-capping
// forward: y = cap * tanh(x / cap) (in place when y == x); backward: dx = dy * (1 - (y / cap)^2) from the saved output.
// Replaces the reference's Triton `fused_softcap_kernel` (primus/backends/megatron/core/extensions/logits_processor.py:13-37).
__global__ void softcap_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, long nvec,
                                   float cap, float inv_cap) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nvec; i += (long)gridDim.x * blockDim.x) {
    float f[8];
    bf8_to_f(reinterpret_cast<const Bf8*>(x)[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = cap * tanhf(f[j] * inv_cap);
    reinterpret_cast<Bf8*>(y)[i] = f_to_bf8(f);
  }
}
__global__ void softcap_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ dx, long nvec, float inv_cap) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nvec; i += (long)gridDim.x * blockDim.x) {
    float g[8], f[8];
    bf8_to_f(reinterpret_cast<const Bf8*>(dy)[i], g);
    bf8_to_f(reinterpret_cast<const Bf8*>(y)[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float t = f[j] * inv_cap;
      g[j] *= (1.f - t * t);
    }
    reinterpret_cast<Bf8*>(dx)[i] = f_to_bf8(g);
  }
}

// ------------------------------------------------------------------ RoPE (rotate-half), in place
// x: [T, heads, d] with row pitch ld; rotates the first rot_dim channels of every head.
// pos[t] selects the row of the cos/sin tables ([max_pos, rot_dim/2] fp32). sign=-1 for backward.
// A thread owns 8 channel pairs of ROPE_HEADS neighbouring heads of a token: their 2 x ROPE_HEADS 16-byte loads are in
// flight together and share one read of the cos / sin entries.
template <int ROPE_HEADS>
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos, const float* __restrict__ cos_t,
            const float* __restrict__ sin_t, long T, int heads, int d, int rot_dim, long ld, float sign) {
  PB_GRID_WAIT();
  const int half = rot_dim / 2;
  const int vec_per_head = half / 8;
  const int per_token = vec_per_head * ((heads + ROPE_HEADS - 1) / ROPE_HEADS);
  const long idx = blockIdx.x * 256L + threadIdx.x;
  const long t = idx / per_token;
  if (t >= T) return;
  const int r = (int)(idx - t * per_token);
  const int v = r % vec_per_head, h0 = r / vec_per_head * ROPE_HEADS;
  const int p = pos ? pos[t] : (int)t;
  __nv_bfloat16* base = x + t * ld + (long)h0 * d + v * 8;
  Bf8 a[ROPE_HEADS], b[ROPE_HEADS];
#pragma unroll
  for (int i = 0; i < ROPE_HEADS; ++i)
    if (h0 + i < heads) {
      a[i] = *reinterpret_cast<Bf8*>(base + (long)i * d);
      b[i] = *reinterpret_cast<Bf8*>(base + (long)i * d + half);
    }
  float c[8], s[8];
  const float* cp = cos_t + (long)p * half + v * 8;
  const float* sp = sin_t + (long)p * half + v * 8;
  *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cp);
  *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cp + 4);
  *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(sp);
  *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(sp + 4);
#pragma unroll
  for (int i = 0; i < ROPE_HEADS; ++i)
    if (h0 + i < heads) {
      float fa[8], fb[8], oa[8], ob[8];
      bf8_to_f(a[i], fa);
      bf8_to_f(b[i], fb);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sn = s[j] * sign;
        oa[j] = fa[j] * c[j] - fb[j] * sn;
        ob[j] = fb[j] * c[j] + fa[j] * sn;
      }
      *reinterpret_cast<Bf8*>(base + (long)i * d) = f_to_bf8(oa);
      *reinterpret_cast<Bf8*>(base + (long)i * d + half) = f_to_bf8(ob);
    }
}

// gated-unit activations: kind 0 = SiLU (SwiGLU), 1 = tanh-approximated GELU (GEGLU)
__device__ __forceinline__ float gate_act(float g, int kind, float& dact) {
  if (kind == 0) {
    const float sig = pb::fast_sigmoid(g);
    dact = sig * (1.f + g * (1.f - sig));
    return g * sig;
  }
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float t = tanhf(k0 * (g + k1 * g * g * g));
  dact = 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * k0 * (1.f + 3.f * k1 * g * g);
  return 0.5f * g * (1.f + t);
}

// ------------------------------------------------------------------ SwiGLU
// in: [T, 2I] = [gate | up]; out[T, I] = act(min(g,clamp)) * clip(u,+-clamp) * prob[t]; KIND: gate_act.
// The kernels are bound by memory: a thread takes 16-byte vectors of `in`, the grid's threads apart (the backward two at a time:
// 8192 x 14336 224 -> 186 us, 128 x 7168 30 -> 8; the forward gains nothing from a second one, 109 and 117), and steps from one
// to the next by the quotient and remainder of that distance (dt rows, dv vectors) instead of a 64-bit division each.  The
// backward with the gradient of the probabilities takes a warp per row (40896 x 768 62 -> 56 us with three vectors in flight).
template <int KIND, bool CLAMP>
__device__ __forceinline__ void swiglu_fwd_vec(const Bf8& g, const Bf8& u, float p, float clamp, Bf8& out) {
  float fg[8], fu[8], o[8];
  bf8_to_f(g, fg);
  bf8_to_f(u, fu);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float gg = fg[j], uu = fu[j];
    if (CLAMP) {
      gg = fminf(gg, clamp);
      uu = fminf(fmaxf(uu, -clamp), clamp);
    }
    float unused;
    o[j] = gate_act(gg, KIND, unused) * uu * p;
  }
  out = f_to_bf8(o);
}
// ... og, ou: gradients of gate and up; act: what the forward gave; returns the sum of dy * act / p
template <int KIND, bool CLAMP>
__device__ __forceinline__ float swiglu_bwd_vec(const Bf8& g, const Bf8& u, const Bf8& dy, float p, float clamp, float dp, Bf8& dg,
                                                Bf8& du, Bf8& act) {
  float fg[8], fu[8], fd[8], og[8], ou[8], oa[8];
  bf8_to_f(g, fg);
  bf8_to_f(u, fu);
  bf8_to_f(dy, fd);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float gg = fg[j], uu = fu[j];
    float gmask = 1.f, umask = 1.f;
    if (CLAMP) {
      if (gg > clamp) { gg = clamp; gmask = 0.f; }
      if (uu > clamp) { uu = clamp; umask = 0.f; }
      if (uu < -clamp) { uu = -clamp; umask = 0.f; }
    }
    float dsl;
    const float sl = gate_act(gg, KIND, dsl);
    dp += fd[j] * sl * uu;
    const float d = fd[j] * p;
    og[j] = d * uu * dsl;
    ou[j] = d * sl;
    if (CLAMP) {
      og[j] *= gmask;
      ou[j] *= umask;
    }
    oa[j] = sl * uu * p;
  }
  dg = f_to_bf8(og);
  du = f_to_bf8(ou);
  act = f_to_bf8(oa);
  return dp;
}

struct VecWalk {                        // a thread's vectors: row t, vector v of vpr
  long t;
  int v, vpr;
  __device__ __forceinline__ VecWalk(int vpr_) : vpr(vpr_) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    t = i / (unsigned)vpr_;
    v = (int)(i - (unsigned)t * (unsigned)vpr_);
  }
  __device__ __forceinline__ void next(int dt, int dv) {
    t += dt;
    v += dv;
    if (v >= vpr) { v -= vpr; ++t; }
  }
};

template <int KIND, bool CLAMP>
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ in, const float* __restrict__ probs, __nv_bfloat16* __restrict__ out, long T,
                  int I, float clamp, int dt, int dv) {
  PB_GRID_WAIT();
  for (VecWalk w(I / 8); w.t < T; w.next(dt, dv)) {
    const Bf8* row = reinterpret_cast<const Bf8*>(in + w.t * 2L * I) + w.v;
    Bf8 o;
    swiglu_fwd_vec<KIND, CLAMP>(row[0], row[I / 8], probs ? probs[w.t] : 1.f, clamp, o);
    reinterpret_cast<Bf8*>(out + w.t * (long)I)[w.v] = o;
  }
}

// din[T,2I] from dy[T,I]; act (optional, may be dy itself): the forward's output again, for a weight gradient that did not keep it
// (a pass of its own reads `in` once more; 8192 x 14336: 224 + 113 us in two passes, 234 in one).
template <int KIND, bool CLAMP>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* __restrict__ in, const float* __restrict__ probs,
                  __nv_bfloat16* __restrict__ din, __nv_bfloat16* act, long T, int I, float clamp, int dt, int dv) {
  PB_GRID_WAIT();
  VecWalk w(I / 8);
  while (w.t < T) {
    Bf8 g[2], u[2], d[2];
    float p[2];
    long t[2];
    int v[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      t[k] = w.t;
      v[k] = w.v;
      if (t[k] < T) {
        const Bf8* row = reinterpret_cast<const Bf8*>(in + t[k] * 2L * I) + v[k];
        g[k] = row[0];
        u[k] = row[I / 8];
        d[k] = reinterpret_cast<const Bf8*>(dy + t[k] * (long)I)[v[k]];
        p[k] = probs ? probs[t[k]] : 1.f;
      }
      w.next(dt, dv);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (t[k] < T) {
        Bf8 a;
        swiglu_bwd_vec<KIND, CLAMP>(g[k], u[k], d[k], p[k], clamp, 0.f, g[k], u[k], a);
        Bf8* row = reinterpret_cast<Bf8*>(din + t[k] * 2L * I) + v[k];
        row[0] = g[k];
        row[I / 8] = u[k];
        if (act) reinterpret_cast<Bf8*>(act + t[k] * (long)I)[v[k]] = a;
      }
  }
}

// ... and dprobs[t] = sum_i dy * act(g) * u: a warp per row, three vectors of a lane in flight
template <int KIND, bool CLAMP>
__global__ void __launch_bounds__(256)
swiglu_bwd_probs_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* __restrict__ in, const float* __restrict__ probs,
                        __nv_bfloat16* __restrict__ din, __nv_bfloat16* act, float* __restrict__ dprobs, long T, int I, float clamp) {
  PB_GRID_WAIT();
  const int vpr = I / 8, lane = threadIdx.x & 31;
  const long num_warps = ((long)gridDim.x * blockDim.x) >> 5;
  for (long t = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5; t < T; t += num_warps) {
    const float p = probs ? probs[t] : 1.f;
    const Bf8 *rg = reinterpret_cast<const Bf8*>(in + t * 2L * I), *ru = rg + vpr, *rd = reinterpret_cast<const Bf8*>(dy + t * (long)I);
    Bf8 *og = reinterpret_cast<Bf8*>(din + t * 2L * I), *ou = og + vpr, *oa = act ? reinterpret_cast<Bf8*>(act + t * (long)I) : nullptr;
    float dp = 0.f;
    for (int v0 = lane; v0 < vpr; v0 += 96) {
      Bf8 g[3], u[3], d[3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (v0 + 32 * k < vpr) {
          g[k] = rg[v0 + 32 * k];
          u[k] = ru[v0 + 32 * k];
          d[k] = rd[v0 + 32 * k];
        }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (v0 + 32 * k < vpr) {
          Bf8 a;
          dp = swiglu_bwd_vec<KIND, CLAMP>(g[k], u[k], d[k], p, clamp, dp, g[k], u[k], a);
          og[v0 + 32 * k] = g[k];
          ou[v0 + 32 * k] = u[k];
          if (oa) oa[v0 + 32 * k] = a;
        }
    }
    dp = pb::warp_sum(dp);
    if (lane == 0) dprobs[t] = dp;
  }
}

// ------------------------------------------------------------------ cross entropy
// Phase 1: per-row local max, sum(exp(x - max)) and the target logit when the label falls into
// this rank's vocabulary slice [vocab_start, vocab_start + V).
constexpr int CE_THREADS = 1024;
__global__ void __launch_bounds__(CE_THREADS)
ce_stats_kernel(const __nv_bfloat16* __restrict__ logits, const long* __restrict__ labels,
                float* __restrict__ row_max, float* __restrict__ row_sumexp,
                float* __restrict__ tgt_logit, int V, long ld, int vocab_start) {
  __shared__ float red[32];
  const long row = blockIdx.x;
  const Bf8* lr = reinterpret_cast<const Bf8*>(logits + row * ld);
  const int nv = V / 8;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < nv; i += CE_THREADS) {
    float f[8];
    bf8_to_f(lr[i], f);
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > m) {
      s *= __expf(m - lm);
      m = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
  }
  const float gm = block_max<CE_THREADS>(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  s = block_sum<CE_THREADS>(s, red);
  if (threadIdx.x == 0) {
    row_max[row] = gm;
    row_sumexp[row] = s;
    const long lab = labels[row] - vocab_start;
    tgt_logit[row] = (lab >= 0 && lab < V) ? __bfloat162float(logits[row * ld + lab]) : 0.f;
  }
}

// Phase 2: logits <- (softmax - onehot) * gscale[row]  (in place), given the global log-sum-exp.
__global__ void __launch_bounds__(CE_THREADS)
ce_grad_kernel(__nv_bfloat16* __restrict__ logits, const long* __restrict__ labels,
               const float* __restrict__ lse, const float* __restrict__ gscale, int V, long ld,
               int vocab_start) {
  const long row = blockIdx.x;
  Bf8* lr = reinterpret_cast<Bf8*>(logits + row * ld);
  const int nv = V / 8;
  const float l = lse[row];
  const float sc = gscale[row];
  const long lab = labels[row] - vocab_start;
  for (int i = threadIdx.x; i < nv; i += CE_THREADS) {
    float f[8];
    bf8_to_f(lr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(f[j] - l);
      if ((long)i * 8 + j == lab) p -= 1.f;
      f[j] = p * sc;
    }
    lr[i] = f_to_bf8(f);
  }
}

// Single-rank fused form: loss[row] = lse - target, gradient written in place.  A CTA takes a row, sums it and reads it again.
// What bounded it was instructions (80 % of the issue slots at 1480 x 128256, half of the memory's rate), so two values go into one
// packed operation wherever there is one, the exponentials' care for denormals is left to vectors that have any, and the target
// to its owner before and after the loop.  Then it is the memory, twice the logits as long as the second reading comes from L2:
//   HOLD = 0: four rows per SM under way, which have to fit into L2;
//   HOLD > 0: two, of whose vectors a thread keeps its first HOLD (all there: V >= 8 THREADS HOLD) in shared memory, and results
//   leave by stores that make way in L2.
// us, before and now: 4096 x 128256 494 -> 358, 1024 x 202048 226 -> 176, 4096 x 50304 223 -> 153, 4096 x 32000 153 -> 94, 768 x
// 32000 39 -> 27, 20000 x 1000 173 -> 75.  (A CTA per SM that stays, with its row and the next ones' start in a ring of
// asynchronous copies: 450 us for the first, as its SM moves nothing between sums and gradient.)
constexpr int CE_HOLD = 6;
template <int THREADS, int CTAS, int HOLD, int U>
__global__ void __launch_bounds__(THREADS, CTAS)
ce_fused_kernel(__nv_bfloat16* __restrict__ logits, const long* __restrict__ labels, const float* __restrict__ gscale,
                float* __restrict__ loss, int V, long ld) {
  PB_GRID_WAIT();
  extern __shared__ __align__(16) uint8_t held_raw[];
  __shared__ float2 red[THREADS / 32];
  constexpr float LOG2E = 1.4426950408889634f;
  const int tid = threadIdx.x, nv = V / 8;
  const long row = blockIdx.x;
  uint4* held = reinterpret_cast<uint4*>(held_raw) + tid;                // [HOLD][thread]
  uint4* lr = reinterpret_cast<uint4*>(logits + row * ld);
  const uint64_t one2 = pb::pack_f32x2(1.f, 1.f), log2e2 = pb::pack_f32x2(LOG2E, LOG2E);
  // (f + neg) log2(e) of a word's two values
  auto scaled = [&](uint32_t w, uint64_t neg) {
    const uint64_t f = pb::pack_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return pb::mul_f32x2(pb::fma_f32x2(f, one2, neg), log2e2);
  };
  float m = -3.402823466e38f;    // (finite: nothing but -inf so far adds 0, not a NaN)
  uint64_t s2 = 0;               // sums of the even and the odd values' exp(f - m)
  auto sum = [&](const uint4 v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const float lm = pb::max_bf16x2(pb::max2_bf16x2(pb::max2_bf16x2(w[0], w[1]), pb::max2_bf16x2(w[2], w[3])));
    if (lm > m) {
      const float c = pb::fast_exp2((m - lm) * LOG2E);
      s2 = pb::mul_f32x2(s2, pb::pack_f32x2(c, c));
      m = lm;
    }
    const uint64_t neg = pb::pack_f32x2(-m, -m);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float a, b;
      pb::unpack_f32x2(scaled(w[q], neg), a, b);
      s2 = pb::fma_f32x2(pb::pack_f32x2(pb::fast_exp2(a), pb::fast_exp2(b)), one2, s2);
    }
  };
  int i = tid;
#pragma unroll 1
  for (int h = 0; h < HOLD; h += U) {
    uint4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) v[k] = __ldcs(lr + i + k * THREADS);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      held[(h + k) * THREADS] = v[k];
      sum(v[k]);
    }
    i += U * THREADS;
  }
  for (; i < nv; i += THREADS) sum(lr[i]);
  const long lab = labels[row];
  const float sc = gscale[row];
  float s, s1;
  pb::unpack_f32x2(s2, s, s1);
  const float wm = pb::warp_max(m);
  s = pb::warp_sum((s + s1) * pb::fast_exp2((m - wm) * LOG2E));
  if ((tid & 31) == 0) red[tid >> 5] = make_float2(wm, s);
  __syncthreads();
  const float2 r = red[tid & (THREADS / 32 - 1)];
  const float gm = pb::warp_max(r.x);
  s = r.y * pb::fast_exp2((r.x - gm) * LOG2E);
  // (logf: mean error of the loss against 64 bits 3.0e-7 at 512 x 8192, 2.8e-7 at 128 x 128256; with __logf 3.6e-7 and 4.0e-7)
  const float l = gm + logf(pb::warp_sum((tid & 31) < THREADS / 32 ? s : 0.f));
  // the target's logit belongs to the thread that will write its vector
  const bool has_label = lab >= 0 && lab < V, own_label = has_label && tid == (int)(lab / 8) % THREADS;
  float t = l;
  if (own_label) t = __bfloat162float(logits[row * ld + lab]);
  if (has_label ? own_label : tid == 0) loss[row] = l - t;
  const uint64_t neg = pb::pack_f32x2(-l, -l), sc2 = pb::pack_f32x2(sc, sc);
  const float low = l - 86.f;    // exp(-86) is a normal number
  auto grad = [&](const uint4 v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float p[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) pb::unpack_f32x2(scaled(w[q], neg), p[2 * q], p[2 * q + 1]);
    if (pb::min_bf16x2(pb::min2_bf16x2(pb::min2_bf16x2(w[0], w[1]), pb::min2_bf16x2(w[2], w[3]))) > low) {
#pragma unroll
      for (int j = 0; j < 8; ++j) p[j] = pb::fast_exp2(p[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) asm("ex2.approx.f32 %0, %0;" : "+f"(p[j]));
    }
    uint32_t g[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float a, b;
      pb::unpack_f32x2(pb::mul_f32x2(pb::pack_f32x2(p[2 * q], p[2 * q + 1]), sc2), a, b);
      g[q] = pb::pack_bf16x2(a, b);
    }
    if (HOLD) __stcs(lr + i, make_uint4(g[0], g[1], g[2], g[3]));
    else lr[i] = make_uint4(g[0], g[1], g[2], g[3]);
  };
  i = tid;
#pragma unroll 2
  for (int h = 0; h < HOLD; ++h, i += THREADS) grad(held[h * THREADS]);
  for (; i < nv; i += THREADS) grad(HOLD ? __ldcs(lr + i) : lr[i]);
  if (own_label) logits[row * ld + lab] = __float2bfloat16_rn((__expf(t - l) - 1.f) * sc);
}

// out[0] = sum of x[i] * w[i], in a fixed order (the loss of a micro-batch from its tokens')
__global__ void __launch_bounds__(1024)
weighted_sum_kernel(const float* __restrict__ x, const float* __restrict__ w, long n, float* __restrict__ out) {
  PB_GRID_WAIT();
  __shared__ float red[32];
  float s = 0.f;
  for (long i = threadIdx.x; i < n; i += 1024) s += x[i] * w[i];
  s = block_sum<1024>(s, red);
  if (threadIdx.x == 0) out[0] = s;
}

// ------------------------------------------------------------------ optimizer / flat-buffer helpers
// AdamW over a flat shard. grads are multiplied by *grad_scale (device scalar: clip coefficient x
// 1/loss-scale). When *skip != 0 (non-finite gradients found) nothing is updated.
__device__ __forceinline__ void load4(const float* p, float* o) {
  *reinterpret_cast<float4*>(o) = *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float* o) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(p);
  const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ void store4(float* p, const float* o) {
  *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(o);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float* o) {
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(p);
  h[0] = __floats2bfloat162_rn(o[0], o[1]);
  h[1] = __floats2bfloat162_rn(o[2], o[3]);
}
__device__ __forceinline__ void store1(float* p, float o) { *p = o; }
__device__ __forceinline__ void store1(__nv_bfloat16* p, float o) { *p = __float2bfloat16(o); }

// The two bias corrections are the same for all elements; dividing by them with the general division made the update bound
// by its three divisions (699 us for 126 M elements, against 589 us this way; 582 us without the care that div_invariant
// takes of numerators near the subnormals).
__device__ __forceinline__ void adamw_update(float& p, float& m, float& v, float g, float lr, float beta1, float beta2,
                                             float eps, float wd, float bc1, float bc2, float ic1, float ic2) {
  m = beta1 * m + (1.f - beta1) * g;
  v = beta2 * v + (1.f - beta2) * g * g;
  const float mh = div_invariant(m, bc1, ic1);
  const float vh = div_invariant(v, bc2, ic2);
  p = p * (1.f - lr * wd) - lr * mh / (sqrtf(vh) + eps);
}

// GradT: fp32 or bf16 gradients; StateT: fp32 or bf16 moments (precision-aware optimizer: the moments can be kept in
// bf16 to halve their memory; the arithmetic is fp32 either way and the master weights stay fp32).
template <typename GradT, typename StateT>
__global__ void adamw_kernel(float* __restrict__ master, StateT* __restrict__ m, StateT* __restrict__ v,
                             const GradT* __restrict__ grad, __nv_bfloat16* __restrict__ param_out,
                             long n, float lr, float beta1, float beta2, float eps, float wd,
                             float bc1, float bc2, float ic1, float ic2, const float* __restrict__ grad_scale,
                             const int* __restrict__ skip) {
  if (skip && *skip) return;
  const float gs = grad_scale ? *grad_scale : 1.f;
  for (long i = (blockIdx.x * (long)blockDim.x + threadIdx.x) * 4; i < n;
       i += (long)gridDim.x * blockDim.x * 4) {
    float p[4], mm[4], vv[4], g[4];
    const bool full = i + 4 <= n;
    if (full) {
      load4(master + i, p);
      load4(m + i, mm);
      load4(v + i, vv);
      load4(grad + i, g);
    } else {
      for (int j = 0; j < 4; ++j) {
        const bool in = i + j < n;
        p[j] = in ? master[i + j] : 0.f;
        mm[j] = in ? (float)m[i + j] : 0.f;
        vv[j] = in ? (float)v[i + j] : 0.f;
        g[j] = in ? (float)grad[i + j] : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) adamw_update(p[j], mm[j], vv[j], g[j] * gs, lr, beta1, beta2, eps, wd, bc1, bc2, ic1, ic2);
    if (full) {
      store4(master + i, p);
      store4(m + i, mm);
      store4(v + i, vv);
      if (param_out) store4(param_out + i, p);
    } else {
      for (int j = 0; j < 4 && i + j < n; ++j) {
        master[i + j] = p[j];
        store1(m + i + j, mm[j]);
        store1(v + i + j, vv[j]);
        if (param_out) param_out[i + j] = __float2bfloat16(p[j]);
      }
    }
  }
}

// AdamW over up to ADAMW_SEGS buckets in one launch (between launches the SMs run empty, 4 us each: 126 M elements in four buckets
// 587 us in four launches, 560 in one).  A bucket is cut into ranges with their own weight-decay multiplier and learning
// rate (norm gains without decay between matrices with it: one launch per range left the SMs idle around every small one);
// range r starts at starts[r] (element 0 first, all multiples of 4) and uses wd * mult[r] and lrs.v[group[r]].  A CTA takes
// a contiguous chunk whose first range the host has looked up; its threads walk on from there, after their loads are issued.
// The chunks go from the last to the first: the gradients that the norm, just before, read last are still in L2.
constexpr int ADAMW_CHUNK = 8192, ADAMW_SEGS = 32;
struct AdamWRates {
  float v[4];
};
struct AdamWSeg {                       // a bucket; the first of its chunks in the launch
  float* master;
  void *m, *v;
  const void* grad;
  __nv_bfloat16* param_out;
  long n;
  const int* first;
  const long* starts;
  const float* mult;
  const int* group;
  int R;
  unsigned chunk0;
};
struct AdamWSegs {
  AdamWSeg seg[ADAMW_SEGS];
  int count;
};
template <typename GradT, typename StateT>
__global__ void __launch_bounds__(256, 5)
adamw_ranges_kernel(const __grid_constant__ AdamWSegs segs, AdamWRates lrs, float beta1, float beta2, float eps, float wd,
                    float bc1, float bc2, float ic1, float ic2, const float* __restrict__ grad_scale,
                    const int* __restrict__ skip) {
  PB_GRID_WAIT();
  if (skip && *skip) return;
  const unsigned chunk = gridDim.x - 1 - blockIdx.x;
  int k = segs.count - 1;
  while (segs.seg[k].chunk0 > chunk) --k;
  const AdamWSeg& sg = segs.seg[k];
  float* __restrict__ master = sg.master;
  StateT *__restrict__ m = (StateT*)sg.m, *__restrict__ v = (StateT*)sg.v;
  const GradT* __restrict__ grad = (const GradT*)sg.grad;
  __nv_bfloat16* __restrict__ param_out = sg.param_out;
  const long n = sg.n;
  const long* __restrict__ starts = sg.starts;
  const float* __restrict__ mult = sg.mult;
  const int* __restrict__ group = sg.group;
  const int R = sg.R;
  const long c0 = (long)(chunk - sg.chunk0) * ADAMW_CHUNK, c1 = min(n, c0 + ADAMW_CHUNK);
  int r = sg.first[chunk - sg.chunk0];
  const float gs = grad_scale ? *grad_scale : 1.f;
  long end = r + 1 < R ? starts[r + 1] : n;
  float lr = lrs.v[group[r]], rwd = wd * mult[r];
  for (long i = c0 + threadIdx.x * 4; i < c1; i += 256 * 4) {
    float p[4], mm[4], vv[4], g[4];
    const bool full = i + 4 <= n;
    if (full) {
      load4(master + i, p);
      load4(m + i, mm);
      load4(v + i, vv);
      load4(grad + i, g);
    } else {
      for (int j = 0; j < 4; ++j) {
        const bool in = i + j < n;
        p[j] = in ? master[i + j] : 0.f;
        mm[j] = in ? (float)m[i + j] : 0.f;
        vv[j] = in ? (float)v[i + j] : 0.f;
        g[j] = in ? (float)grad[i + j] : 0.f;
      }
    }
    if (i >= end) {
      do {
        ++r;
        end = r + 1 < R ? starts[r + 1] : n;
      } while (i >= end);
      lr = lrs.v[group[r]];
      rwd = wd * mult[r];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) adamw_update(p[j], mm[j], vv[j], g[j] * gs, lr, beta1, beta2, eps, rwd, bc1, bc2, ic1, ic2);
    if (full) {
      store4(master + i, p);
      store4(m + i, mm);
      store4(v + i, vv);
      store4(param_out + i, p);
    } else {
      for (int j = 0; j < 4 && i + j < n; ++j) {
        master[i + j] = p[j];
        store1(m + i + j, mm[j]);
        store1(v + i + j, vv[j]);
        param_out[i + j] = __float2bfloat16(p[j]);
      }
    }
  }
}

// partial[b] = sum of squares handled by block b (deterministic two-stage reduction).  The order of the additions is fixed
// and part of the result (the clip coefficient, and with it the whole optimizer state, moves with the last bit of the norm):
// SUMSQ_CHAINS serial sums, chain j over the elements j, j + SUMSQ_CHAINS, ... in turn; the 512 chains of a block meet in
// a butterfly over 32 neighbours (distances 16, 8, 4, 2, 1) and one over the 16 results.
// What bounds it is the bytes in flight.  A thread therefore owns PER neighbouring chains, whose elements are one 16-byte
// load, with U of them issued before the first is added, and a block is 512 / PER threads; the butterfly steps whose
// distance is below PER are additions inside a thread.  A start off a 16-byte boundary takes element loads, in the same
// order.
constexpr int SUMSQ_BLOCKS = 1184, SUMSQ_BLOCK_CHAINS = 512;
constexpr long SUMSQ_CHAINS = (long)SUMSQ_BLOCKS * SUMSQ_BLOCK_CHAINS;

__device__ __forceinline__ void sumsq_unpack(const float* p, float (&f)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  f[0] = q.x; f[1] = q.y; f[2] = q.z; f[3] = q.w;
}
__device__ __forceinline__ void sumsq_unpack(const __nv_bfloat16* p, float (&f)[8]) {
  bf8_to_f(*reinterpret_cast<const Bf8*>(p), f);
}

constexpr int SUMSQ_SEGS = 32;
struct SumsqSegs {                      // tensors of one launch: SUMSQ_BLOCKS blocks and partial sums each
  const void* x[SUMSQ_SEGS];
  long n[SUMSQ_SEGS];
};

template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(SUMSQ_BLOCK_CHAINS * sizeof(T) / 16)
sumsq_partial_kernel(const __grid_constant__ SumsqSegs segs, float* __restrict__ partial) {
  PB_GRID_WAIT();
  constexpr int PER = 16 / sizeof(T), THREADS = SUMSQ_BLOCK_CHAINS / PER, LANES = 32 / PER, U = 8;
  __shared__ float red[16];
  const T* __restrict__ x = (const T*)segs.x[blockIdx.x / SUMSQ_BLOCKS];
  const long n = segs.n[blockIdx.x / SUMSQ_BLOCKS];
  const long j0 = (long)(blockIdx.x % SUMSQ_BLOCKS) * SUMSQ_BLOCK_CHAINS + threadIdx.x * PER;
  float s[PER] = {};
  long i = j0;
  if (ALIGNED) {
    for (; i + (U - 1) * SUMSQ_CHAINS + PER <= n; i += U * SUMSQ_CHAINS) {
      float f[U][PER];
#pragma unroll
      for (int u = 0; u < U; ++u) sumsq_unpack(x + i + u * SUMSQ_CHAINS, f[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < PER; ++e) s[e] += f[u][e] * f[u][e];
    }
    for (; i + PER <= n; i += SUMSQ_CHAINS) {
      float f[PER];
      sumsq_unpack(x + i, f);
#pragma unroll
      for (int e = 0; e < PER; ++e) s[e] += f[e] * f[e];
    }
  }
  for (; i < n; i += SUMSQ_CHAINS) {
#pragma unroll
    for (int e = 0; e < PER; ++e)
      if (i + e < n) {
        const float f = (float)x[i + e];
        s[e] += f * f;
      }
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < PER; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
#pragma unroll
  for (int o = PER / 2; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < o; ++e) s[e] += s[e + o];
  if (threadIdx.x % LANES == 0) red[threadIdx.x / LANES] = s[0];
  __syncthreads();
  if (threadIdx.x < 32) {
    const float r = pb::warp_sum(threadIdx.x < 16 ? red[threadIdx.x] : 0.f);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
  }
}
// coef = min(1, max_norm / (sqrt(sumsq) + 1e-6)) * extra
// skip (optional): set to whether the step is left out, because the sum is not finite (check) or above `spike` (if positive).
// In a kernel because as operations of their own the checks are eight launches for one number.
struct ClipArgs {
  float max_norm, extra;
  float *coef, *norm_out;
  int *skip, check;
  float spike;
};
__device__ __forceinline__ void clip_coef(float sumsq, const ClipArgs& a) {
  const float nrm = sqrtf(sumsq);
  if (a.skip) a.skip[0] = (a.check && !isfinite(sumsq)) || (a.spike > 0.f && sumsq > a.spike);
  if (a.norm_out) a.norm_out[0] = nrm;
  float c = 1.f;
  if (a.max_norm > 0.f) c = fminf(1.f, a.max_norm / (nrm + 1e-6f));
  a.coef[0] = c * a.extra;
}
__global__ void clip_coef_kernel(const float* sumsq, ClipArgs args) {
  PB_GRID_WAIT();
  clip_coef(sumsq[0], args);
}

// out[0] (+)= sum(partial) of each of `segs` tensors in turn; nonfinite[0] |= !isfinite(sum); with args.coef the clip
// coefficient of that sum, where nothing else is to be added to it.
__global__ void __launch_bounds__(512) sumsq_final_kernel(const float* __restrict__ partial, int segs,
                                                         float* __restrict__ out, int accumulate,
                                                         int* __restrict__ nonfinite, ClipArgs args) {
  PB_GRID_WAIT();
  constexpr int B = 4;                  // tensors at a time
  __shared__ float red[B][16], total[B];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float r = accumulate && threadIdx.x == 0 ? out[0] : 0.f;
  for (int k0 = 0; k0 < segs; k0 += B) {
    float s[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      s[k] = 0.f;
      if (k0 + k < segs)
        for (int i = threadIdx.x; i < SUMSQ_BLOCKS; i += 512) s[k] += partial[(long)(k0 + k) * SUMSQ_BLOCKS + i];
    }
#pragma unroll
    for (int k = 0; k < B; ++k) {
      s[k] = pb::warp_sum(s[k]);
      if (lane == 0) red[k][warp] = s[k];
    }
    __syncthreads();
    if (warp < B) {
      const float t = pb::warp_sum(lane < 16 ? red[warp][lane] : 0.f);
      if (lane == 0) total[warp] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int k = 0; k < B && k0 + k < segs; ++k) r += total[k];
  }
  if (threadIdx.x == 0) {
    out[0] = r;
    if (nonfinite && !isfinite(r)) *nonfinite = 1;
    if (args.coef) clip_coef(r, args);
  }
}

__global__ void scale_f32_kernel(float* __restrict__ x, long n, float s) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    x[i] *= s;
}
__global__ void cast_f32_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}
// dst(fp32) += src(bf16)   (flat; used to fold bf16 gradients into fp32 main grads)
__global__ void add_bf16_into_f32_kernel(float* __restrict__ dst, const __nv_bfloat16* __restrict__ src, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] += __bfloat162float(src[i]);
}
// embedding backward: dW[token[t], :] += dy[t, :]  (fp32 atomics)
__global__ void embedding_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const long* __restrict__ tokens,
                                     float* __restrict__ dw, long T, int H, int vocab_start, int vocab) {
  PB_GRID_WAIT();
  const long total = T * (H / 2);
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const long t = idx / (H / 2);
    const int c = (idx % (H / 2)) * 2;
    const long tok = tokens[t] - vocab_start;
    if (tok < 0 || tok >= vocab) continue;
    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dy + t * H + c));
    atomicAdd(dw + tok * H + c, g.x);
    atomicAdd(dw + tok * H + c + 1, g.y);
  }
}

inline int grid_for(long work_items, int threads, int cap = 148 * 16) {
  long g = (work_items + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

}  // namespace

#define PB_CHECK_LAUNCH() return (int)cudaGetLastError()

extern "C" {

int pb_rope(void* x, const int* pos, const float* cos_t, const float* sin_t, long T, int heads, int d,
            int rot_dim, long ld, int backward, cudaStream_t s) {
  if (rot_dim % 16 || ld % 8 || d % 8) return -2;
  // four heads per thread where that still gives every SM 1024 threads, else one head, for the parallelism
  const long vecs = T * (rot_dim / 16), four = vecs * ((heads + 3) / 4), one = vecs * heads;
  if (one <= 0) return 0;
  const float sign = backward ? -1.f : 1.f;
  if (four >= 148 * 1024L)
    pbh::launch_dependent(rope_kernel<4>, (unsigned)((four + 255) / 256), 256, 0, s, (__nv_bfloat16*)x, pos, cos_t, sin_t, T, heads,
        d, rot_dim, ld, sign);
  else
    pbh::launch_dependent(rope_kernel<1>, (unsigned)((one + 255) / 256), 256, 0, s, (__nv_bfloat16*)x, pos, cos_t, sin_t, T, heads,
        d, rot_dim, ld, sign);
  PB_CHECK_LAUNCH();
}

int pb_softcap_fwd(const void* x, void* y, long n, float cap, cudaStream_t s) {
  if (n % 8 || cap <= 0.f) return -2;
  if (n == 0) return 0;
  softcap_fwd_kernel<<<grid_for(n / 8, 256), 256, 0, s>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n / 8, cap,
                                                         1.f / cap);
  PB_CHECK_LAUNCH();
}

int pb_softcap_bwd(const void* dy, const void* y, void* dx, long n, float cap, cudaStream_t s) {
  if (n % 8 || cap <= 0.f) return -2;
  if (n == 0) return 0;
  softcap_bwd_kernel<<<grid_for(n / 8, 256), 256, 0, s>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)y,
                                                         (__nv_bfloat16*)dx, n / 8, 1.f / cap);
  PB_CHECK_LAUNCH();
}

// kind: 0 SiLU gate (SwiGLU), 1 tanh-GELU gate (GEGLU)
#define PB_SWIGLU_KERNEL(name) \
  (kind == 0 ? (clamp > 0.f ? name<0, true> : name<0, false>) : (clamp > 0.f ? name<1, true> : name<1, false>))
int pb_swiglu_fwd(const void* in, const float* probs, void* out, long T, int I, float clamp, int kind, cudaStream_t s) {
  if (I % 8) return -2;
  if (T == 0 || I == 0) return 0;
  const int blocks = grid_for(T * (I / 8), 256), step = blocks * 256;
  auto kern = PB_SWIGLU_KERNEL(swiglu_fwd_kernel);
  pbh::launch_dependent(kern, blocks, 256, 0, s, (const __nv_bfloat16*)in, probs, (__nv_bfloat16*)out, T, I, clamp, step / (I / 8),
      step % (I / 8));
  PB_CHECK_LAUNCH();
}

// act (or null): receives what pb_swiglu_fwd gives, and may be dy itself
int pb_swiglu_bwd_act(const void* dy, const void* in, const float* probs, void* din, float* dprobs, void* act, long T, int I,
                      float clamp, int kind, cudaStream_t s) {
  if (I % 8) return -2;
  if (T == 0) return 0;
  if (dprobs) {
    auto kern = PB_SWIGLU_KERNEL(swiglu_bwd_probs_kernel);
    pbh::launch_dependent(kern, grid_for(T * 32, 256), 256, 0, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)in, probs,
        (__nv_bfloat16*)din, (__nv_bfloat16*)act, dprobs, T, I, clamp);
  } else if (I > 0) {
    const int blocks = grid_for(T * (I / 8), 512, 148 * 8), step = blocks * 256;
    auto kern = PB_SWIGLU_KERNEL(swiglu_bwd_kernel);
    pbh::launch_dependent(kern, blocks, 256, 0, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)in, probs, (__nv_bfloat16*)din,
        (__nv_bfloat16*)act, T, I, clamp, step / (I / 8), step % (I / 8));
  }
  PB_CHECK_LAUNCH();
}
int pb_swiglu_bwd(const void* dy, const void* in, const float* probs, void* din, float* dprobs, long T,
                  int I, float clamp, int kind, cudaStream_t s) {
  return pb_swiglu_bwd_act(dy, in, probs, din, dprobs, nullptr, T, I, clamp, kind, s);
}
#undef PB_SWIGLU_KERNEL

int pb_ce_stats(const void* logits, const long* labels, float* row_max, float* row_sumexp, float* tgt,
                long rows, int V, long ld, int vocab_start, cudaStream_t s) {
  if (V % 8 || ld % 8) return -2;
  if (rows == 0) return 0;
  ce_stats_kernel<<<(unsigned)rows, CE_THREADS, 0, s>>>((const __nv_bfloat16*)logits, labels, row_max,
                                                       row_sumexp, tgt, V, ld, vocab_start);
  PB_CHECK_LAUNCH();
}

int pb_ce_grad(void* logits, const long* labels, const float* lse, const float* gscale, long rows, int V,
               long ld, int vocab_start, cudaStream_t s) {
  if (V % 8 || ld % 8) return -2;
  if (rows == 0) return 0;
  ce_grad_kernel<<<(unsigned)rows, CE_THREADS, 0, s>>>((__nv_bfloat16*)logits, labels, lse, gscale, V, ld,
                                                      vocab_start);
  PB_CHECK_LAUNCH();
}

int pb_ce_fused(void* logits, const long* labels, const float* gscale, float* loss, long rows, int V,
                long ld, cudaStream_t s) {
  if (V % 8 || ld % 8) return -2;
  if (rows == 0) return 0;
  __nv_bfloat16* l = (__nv_bfloat16*)logits;
  // (us, four rows and two: V = 32000 94 and 123, 50304 153 and 165, 65536 209 and 204, 81920 277 and 235, 128256 480 and 358)
  if (V <= 57344) {
    pbh::launch_dependent(ce_fused_kernel<512, 4, 0, 1>, (unsigned)rows, 512, 0, s, l, labels, gscale, loss, V, ld);
  } else {
    static std::atomic<bool> allowed[pbh::MAX_DEVICES];
    auto kern = ce_fused_kernel<1024, 2, CE_HOLD, 3>;
    constexpr int BYTES = CE_HOLD * 1024 * 16;
    if (int rc = pbh::allow_shared_memory(kern, BYTES, allowed)) return rc;
    pbh::launch_dependent(kern, (unsigned)rows, 1024, BYTES, s, l, labels, gscale, loss, V, ld);
  }
  PB_CHECK_LAUNCH();
}

int pb_weighted_sum(const float* x, const float* w, float* out, long n, cudaStream_t s) {
  pbh::launch_dependent(weighted_sum_kernel, 1, 1024, 0, s, x, w, n, out);
  PB_CHECK_LAUNCH();
}

// state_is_bf16: the moments m, v are bf16 tensors (else fp32).
int pb_adamw_ex(float* master, void* m, void* v, const void* grad, int grad_is_bf16, int state_is_bf16,
                void* param_out, long n, float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2,
                const float* grad_scale, const int* skip, cudaStream_t s) {
  if (n == 0) return 0;
  const int g = grid_for((n + 3) / 4, 256, 148 * 8);
  __nv_bfloat16* po = (__nv_bfloat16*)param_out;
#define PB_ADAMW(GT, ST)                                                                                          \
  adamw_kernel<GT, ST><<<g, 256, 0, s>>>(master, (ST*)m, (ST*)v, (const GT*)grad, po, n, lr, beta1, beta2, eps, wd, \
                                         bc1, bc2, (float)(1.0 / bc1), (float)(1.0 / bc2), grad_scale, skip)
  if (grad_is_bf16 && state_is_bf16) PB_ADAMW(__nv_bfloat16, __nv_bfloat16);
  else if (grad_is_bf16) PB_ADAMW(__nv_bfloat16, float);
  else if (state_is_bf16) PB_ADAMW(float, __nv_bfloat16);
  else PB_ADAMW(float, float);
#undef PB_ADAMW
  PB_CHECK_LAUNCH();
}

// `count` buckets: bucket i is the eleven 64-bit values table[11 i ..] (host memory), addresses of master, m, v, grad, param_out
// (bf16), then n, addresses of first, starts, mult and group, and R.  Its ranges r = 0 .. R - 1 start at starts[r] (device, int64;
// starts[0] = 0, ascending multiples of 4) and use weight decay wd * mult[r] and learning rate lr[group[r]]; first[c]: the range
// that element c * pb_adamw_ranges_chunk() lies in.  hyper (host): four learning rates, beta1, beta2, eps, wd, and the two bias
// corrections.
int pb_adamw_ranges_chunk() { return ADAMW_CHUNK; }

int pb_adamw_ranges(const long* table, int count, const float* hyper, int grad_is_bf16, int state_is_bf16,
                    const float* grad_scale, const int* skip, cudaStream_t s) {
  for (int i = 0; i < count; ++i)
    if (table[11 * i + 5] < 0 || (table[11 * i + 5] && (table[11 * i + 10] <= 0 || !table[11 * i + 4]))) return -2;
  const AdamWRates lrs{{hyper[0], hyper[1], hyper[2], hyper[3]}};
  const float beta1 = hyper[4], beta2 = hyper[5], eps = hyper[6], wd = hyper[7], bc1 = hyper[8], bc2 = hyper[9];
  for (int i = 0; i < count;) {
    AdamWSegs segs;
    segs.count = 0;
    long chunks = 0;
    for (; i < count && segs.count < ADAMW_SEGS; ++i) {
      const long* t = table + 11 * i;
      if (t[5] == 0) continue;
      const long add = (t[5] + ADAMW_CHUNK - 1) / ADAMW_CHUNK;
      if (chunks + add > 2147483647L) break;
      segs.seg[segs.count++] = AdamWSeg{(float*)t[0], (void*)t[1], (void*)t[2], (const void*)t[3], (__nv_bfloat16*)t[4], t[5],
                                        (const int*)t[6], (const long*)t[7], (const float*)t[8], (const int*)t[9], (int)t[10],
                                        (unsigned)chunks};
      chunks += add;
    }
    if (chunks == 0) {
      if (i < count) return -2;                        // a bucket of more chunks than a grid has blocks
      break;
    }
#define PB_ADAMW(GT, ST)                                                                                                      \
  pbh::launch_dependent(adamw_ranges_kernel<GT, ST>, (unsigned)chunks, 256, 0, s, segs, lrs, beta1, beta2, eps, wd, bc1, bc2, \
      (float)(1.0 / bc1), (float)(1.0 / bc2), grad_scale, skip)
    if (grad_is_bf16 && state_is_bf16) PB_ADAMW(__nv_bfloat16, __nv_bfloat16);
    else if (grad_is_bf16) PB_ADAMW(__nv_bfloat16, float);
    else if (state_is_bf16) PB_ADAMW(float, __nv_bfloat16);
    else PB_ADAMW(float, float);
#undef PB_ADAMW
    const int rc = (int)cudaGetLastError();
    if (rc) return rc;
  }
  return 0;
}

int pb_adamw(float* master, float* m, float* v, const void* grad, int grad_is_bf16, void* param_out,
             long n, float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2,
             const float* grad_scale, const int* skip, cudaStream_t s) {
  return pb_adamw_ex(master, m, v, grad, grad_is_bf16, 0, param_out, n, lr, beta1, beta2, eps, wd, bc1, bc2, grad_scale,
                     skip, s);
}

int pb_sumsq_num_partials() { return SUMSQ_BLOCKS; }

namespace {
int sumsq_many(const long* table, int count, int is_bf16, float* scratch, float* out, int accumulate, int* nonfinite,
               const ClipArgs& clip, cudaStream_t s) {
  bool aligned = true;
  for (int i = 0; i < count; ++i) aligned = aligned && table[2 * i] % 16 == 0;
  for (int i = 0; i < count; i += SUMSQ_SEGS) {
    SumsqSegs segs;
    const int n = count - i < SUMSQ_SEGS ? count - i : SUMSQ_SEGS;
    for (int k = 0; k < n; ++k) {
      segs.x[k] = (const void*)table[2 * (i + k)];
      segs.n[k] = table[2 * (i + k) + 1];
    }
#define PB_SUMSQ(T, A) \
  pbh::launch_dependent(sumsq_partial_kernel<T, A>, n * SUMSQ_BLOCKS, SUMSQ_BLOCK_CHAINS * sizeof(T) / 16, 0, s, segs, \
      scratch + (long)i * SUMSQ_BLOCKS)
    if (is_bf16) { if (aligned) PB_SUMSQ(__nv_bfloat16, true); else PB_SUMSQ(__nv_bfloat16, false); }
    else { if (aligned) PB_SUMSQ(float, true); else PB_SUMSQ(float, false); }
#undef PB_SUMSQ
    const int rc = (int)cudaGetLastError();
    if (rc) return rc;
  }
  pbh::launch_dependent(sumsq_final_kernel, 1, 512, 0, s, scratch, count, out, accumulate, nonfinite, clip);
  return (int)cudaGetLastError();
}
}  // namespace

// out[0] (+)= sum(x^2). scratch: fp32 [pb_sumsq_num_partials()].
int pb_sumsq(const void* x, int is_bf16, long n, float* scratch, float* out, int accumulate,
             int* nonfinite, cudaStream_t s) {
  const long table[2] = {(long)x, n};
  return sumsq_many(table, 1, is_bf16, scratch, out, accumulate, nonfinite, ClipArgs{}, s);
}

// out[0] (+)= the sums of squares of `count` tensors of one type, added in turn as by as many pb_sumsq calls; table (host): address
// and number of elements of each.  scratch: fp32 [count, pb_sumsq_num_partials()].  coef (or null): then what pb_clip_coef
// gives for out[0].  (126 M fp32 values in four tensors: 99 + 12 us in eight launches and two more for the coefficient, 88 + 6 in two.)
int pb_grad_norm(const long* table, int count, int is_bf16, float* scratch, float* out, int accumulate, float max_norm, float extra,
                 float* coef, float* norm_out, int* skip, int check, float spike, cudaStream_t s) {
  if (count <= 0) return -2;
  return sumsq_many(table, count, is_bf16, scratch, out, accumulate, nullptr,
                    ClipArgs{max_norm, extra, coef, norm_out, skip, check, spike}, s);
}

int pb_clip_coef(const float* sumsq, float max_norm, float extra, float* coef, float* norm_out, int* skip, int check,
                 float spike, cudaStream_t s) {
  pbh::launch_dependent(clip_coef_kernel, 1, 1, 0, s, sumsq, ClipArgs{max_norm, extra, coef, norm_out, skip, check, spike});
  PB_CHECK_LAUNCH();
}

int pb_scale_f32(float* x, long n, float sc, cudaStream_t s) {
  if (n == 0) return 0;
  scale_f32_kernel<<<grid_for(n, 256), 256, 0, s>>>(x, n, sc);
  PB_CHECK_LAUNCH();
}
int pb_cast_f32_bf16(const float* x, void* y, long n, cudaStream_t s) {
  if (n == 0) return 0;
  cast_f32_bf16_kernel<<<grid_for(n, 256), 256, 0, s>>>(x, (__nv_bfloat16*)y, n);
  PB_CHECK_LAUNCH();
}
int pb_add_bf16_into_f32(float* dst, const void* src, long n, cudaStream_t s) {
  if (n == 0) return 0;
  add_bf16_into_f32_kernel<<<grid_for(n, 256), 256, 0, s>>>(dst, (const __nv_bfloat16*)src, n);
  PB_CHECK_LAUNCH();
}
int pb_embedding_bwd(const void* dy, const long* tokens, float* dw, long T, int H, int vocab_start,
                     int vocab, cudaStream_t s) {
  if (H % 2) return -2;
  if (T == 0) return 0;
  pbh::launch_dependent(embedding_bwd_kernel, grid_for(T * (H / 2), 256), 256, 0, s, (const __nv_bfloat16*)dy, tokens, dw, T, H,
      vocab_start, vocab);
  PB_CHECK_LAUNCH();
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// MoE token movement.
//   moe_gather_rows : out[r, :] = x[src[r], :] (* scale[r])   (src[r] < 0 -> zero row: expert padding)
//   moe_combine_rows: out[t, :] = sum_k y[pos[t, k], :]        (pos < 0 skipped)  -- the un-weighted top-k
//                     combine (routing probabilities are applied inside the expert activation) and, read
//                     the other way round, the backward of the gather.
// A warp moves rows with 16-byte accesses.  Replaces the permutation kernels of
// primus/backends/transformer_engine/pytorch/common/triton/permutation.py:189-305.
namespace {

// What bounds both is the loads in flight, and those are a matter of the warps on an SM as much as of the vectors that a lane
// asks for: eight vectors per lane at 64 and more registers were slower than two at 32 to 40.  A warp takes ROWS neighbouring
// rows (tokens) at a time, several where a row is a vector per lane or less, and VECS vectors of each per lane.
template <int ROWS, int VECS>
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ src, const float* __restrict__ scale,
                       __nv_bfloat16* __restrict__ out, long R, int H, const int* __restrict__ limit_rows) {
  PB_GRID_WAIT();
  const int lane = threadIdx.x & 31;
  const long warp_global = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const long num_warps = ((long)gridDim.x * blockDim.x) >> 5;
  const int nv = H / 8;
  const long end = limit_rows ? min(R, (long)*limit_rows) : R;
  for (long r0 = warp_global * ROWS; r0 < end; r0 += num_warps * ROWS) {
    int s[ROWS];
    float sc[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) s[i] = r0 + i < end ? src[r0 + i] : -1;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) sc[i] = scale && s[i] >= 0 ? scale[r0 + i] : 1.f;
    for (int base = lane; base < nv; base += 32 * VECS) {
      Bf8 t[ROWS][VECS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int u = 0; u < VECS; ++u) {
          const int v = base + u * 32;
          if (s[i] < 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) t[i][u].v[j] = __floats2bfloat162_rn(0.f, 0.f);
          } else if (v < nv) {
            t[i][u] = reinterpret_cast<const Bf8*>(x + (long)s[i] * H)[v];
          }
        }
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int u = 0; u < VECS; ++u) {
          const int v = base + u * 32;
          if (v >= nv || r0 + i >= end) continue;
          if (scale) {
            float f[8];
            bf8_to_f(t[i][u], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= sc[i];
            t[i][u] = f_to_bf8(f);
          }
          reinterpret_cast<Bf8*>(out + (r0 + i) * H)[v] = t[i][u];
        }
    }
  }
}

// All COPIES copies of a token at once, summed in copy order: a vector's sum needs its registers only while it is stored.
template <int COPIES, int ROWS, int VECS, int CTAS>
__global__ void __launch_bounds__(256, CTAS)
moe_combine_all_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ pos, __nv_bfloat16* __restrict__ out, long T, int H) {
  PB_GRID_WAIT();
  const int lane = threadIdx.x & 31;
  const long warp_global = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const long num_warps = ((long)gridDim.x * blockDim.x) >> 5;
  const int nv = H / 8;
  for (long t0 = warp_global * ROWS; t0 < T; t0 += num_warps * ROWS) {
    int p[ROWS][COPIES];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int k = 0; k < COPIES; ++k) p[i][k] = t0 + i < T ? pos[(t0 + i) * COPIES + k] : -1;
    for (int base = lane; base < nv; base += 32 * VECS) {
      Bf8 a[ROWS][VECS][COPIES];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int u = 0; u < VECS; ++u)
#pragma unroll
          for (int k = 0; k < COPIES; ++k)
            if (p[i][k] >= 0 && base + u * 32 < nv) a[i][u][k] = reinterpret_cast<const Bf8*>(y + (long)p[i][k] * H)[base + u * 32];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int u = 0; u < VECS; ++u) {
          if (t0 + i >= T || base + u * 32 >= nv) continue;
          float acc[8] = {};
#pragma unroll
          for (int k = 0; k < COPIES; ++k) {
            if (p[i][k] < 0) continue;
            float f[8];
            bf8_to_f(a[i][u][k], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += f[j];
          }
          reinterpret_cast<Bf8*>(out + (t0 + i) * H)[base + u * 32] = f_to_bf8(acc);
        }
    }
  }
}

// COPIES of a token's topk copies at a time, summed in copy order.
template <int COPIES, int ROWS, int VECS>
__global__ void __launch_bounds__(256)
moe_combine_rows_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ pos, __nv_bfloat16* __restrict__ out,
                        long T, int topk, int H) {
  PB_GRID_WAIT();
  const int lane = threadIdx.x & 31;
  const long warp_global = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const long num_warps = ((long)gridDim.x * blockDim.x) >> 5;
  const int nv = H / 8;
  for (long t0 = warp_global * ROWS; t0 < T; t0 += num_warps * ROWS) {
    for (int base = lane; base < nv; base += 32 * VECS) {
      float acc[ROWS][VECS][8] = {};
      for (int k0 = 0; k0 < topk; k0 += COPIES) {
        int p[ROWS][COPIES];
        Bf8 a[ROWS][COPIES][VECS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int k = 0; k < COPIES; ++k) p[i][k] = k0 + k < topk && t0 + i < T ? pos[(t0 + i) * topk + k0 + k] : -1;
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int k = 0; k < COPIES; ++k)
#pragma unroll
            for (int u = 0; u < VECS; ++u)
              if (p[i][k] >= 0 && base + u * 32 < nv)
                a[i][k][u] = reinterpret_cast<const Bf8*>(y + (long)p[i][k] * H)[base + u * 32];
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int k = 0; k < COPIES; ++k)
#pragma unroll
            for (int u = 0; u < VECS; ++u)
              if (p[i][k] >= 0 && base + u * 32 < nv) {
                float f[8];
                bf8_to_f(a[i][k][u], f);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][u][j] += f[j];
              }
      }
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int u = 0; u < VECS; ++u)
          if (t0 + i < T && base + u * 32 < nv)
            reinterpret_cast<Bf8*>(out + (t0 + i) * H)[base + u * 32] = f_to_bf8(acc[i][u]);
    }
  }
}

// CTAs of eight warps for `warps` warps' work (one pass over most layers; more loop)
inline unsigned moe_grid(long warps) { return (unsigned)grid_for(warps * 32, 256, 1 << 16); }

}  // namespace

extern "C" int pb_moe_gather_rows(const void* x, const int* src, const float* scale, void* out, long R, int H,
                                  const int* limit_rows, cudaStream_t s) {
  if (H % 8) return -2;
  if (R == 0) return 0;
#define PB_GATHER(ROWS, VECS)                                                                           \
  pbh::launch_dependent(moe_gather_rows_kernel<ROWS, VECS>, moe_grid((R + ROWS - 1) / ROWS), 256, 0, s, \
      (const __nv_bfloat16*)x, src, scale, (__nv_bfloat16*)out, R, H, limit_rows)
  // (us, B200, before and now: 4096 tokens of 2048, 64 experts, eight copies 51 -> 43; 65536 of 256, two copies 44 -> 22)
  if (H <= 256 && R >= 8192) PB_GATHER(4, 1); else PB_GATHER(1, 2);
#undef PB_GATHER
  return (int)cudaGetLastError();
}

extern "C" int pb_moe_combine_rows(const void* y, const int* pos, void* out, long T, int topk, int H,
                                   cudaStream_t s) {
  if (H % 8) return -2;
  if (T == 0) return 0;
#define PB_COMBINE_ALL(COPIES, ROWS, VECS, CTAS)                                                  \
  pbh::launch_dependent(moe_combine_all_kernel<COPIES, ROWS, VECS, CTAS>, moe_grid((T + ROWS - 1) / ROWS), 256, 0, s, \
      (const __nv_bfloat16*)y, pos, (__nv_bfloat16*)out, T, H)
#define PB_COMBINE(COPIES, ROWS, VECS)                                                            \
  pbh::launch_dependent(moe_combine_rows_kernel<COPIES, ROWS, VECS>, moe_grid((T + ROWS - 1) / ROWS), 256, 0, s, \
      (const __nv_bfloat16*)y, pos, (__nv_bfloat16*)out, T, topk, H)
  // (us, B200, before and now: 16384 tokens of 2048, one copy 31 -> 24; 65536 of 256, two copies 35 -> 17; 4096 of 2048,
  // eight copies 35 -> 29).  Fewer than 148 x 16 warps leave the SMs short of loads unless each asks for more of them: 1024
  // tokens of 4096, eight copies 18 us against 23.
  if (topk == 1) PB_COMBINE_ALL(1, 1, 4, 6);
  else if (topk == 2) { if (H <= 512) PB_COMBINE_ALL(2, 2, 1, 6); else PB_COMBINE_ALL(2, 1, 4, 4); }
  else if (T < 148 * 16) PB_COMBINE(4, 1, 2);
  else if (H <= 256) { if (T < 16384) PB_COMBINE(4, 1, 1); else PB_COMBINE(1, 1, 1); }
  else PB_COMBINE(2, 1, 2);
#undef PB_COMBINE_ALL
#undef PB_COMBINE
  return (int)cudaGetLastError();
}
