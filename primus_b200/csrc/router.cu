// Fused MoE router: score function + (group-limited) top-k + probability normalisation + per-expert token
// counts in one pass over the logits, and the matching backward.  One warp per token; the token's scores
// live in shared memory (E <= 1024).
//
//   softmax, pre_softmax  : full = softmax(l); choose on full;  p_j = full[i_j]
//   softmax, post         : full = softmax(l); choose on l;     p   = softmax(l[i_1..i_k])
//   sigmoid (+ bias)      : full = sigmoid(l); choose on full + bias; p_j = full[i_j] / (sum_j full[i_j] + 1e-20) (k > 1)
//   group-limited         : experts are split into G groups, only the best `group_topk` groups stay eligible
//                           (group score = max, or the sum of the two best entries when a bias is used)
//   p *= scaling_factor;  counts[e] += 1 for every selected expert.
// `full` (fp32 [T, E]) is written for the load-balancing losses and the backward.
//
// Tokens are counted per CTA in shared memory and added once per expert: 32768 atomics on 64 counters of two cache lines were most of
// the kernel (4096 tokens, 64 experts, eight each: 22 us, now 11).  The usual load-balancing loss, coeff * E * sum_e f_e P_e with
// f_e = counts[e] / (T k) and P_e the mean of full[:, e], comes from the same scores: every CTA leaves the sums of its tokens, and
// aux_loss_kernel adds them in a fixed order; its gradient joins the router's backward.
//
// Replaces `fused_group_topk_routing_with_aux_score` and the router's softmax / top-k op chain
// (primus/backends/megatron/core/transformer/moe/router.py:24-134).
#include "common.cuh"

namespace {

constexpr int WARPS = 8;

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax warp_argmax(float v, int i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) {
      v = ov;
      i = oi;
    }
  }
  return {v, i};
}

template <typename TIn>
__device__ __forceinline__ float to_f(TIn x);
template <>
__device__ __forceinline__ float to_f<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

// One token: everything but the counts.  sel_i: the expert that lane j < k selected.
template <typename TIn>
__device__ __forceinline__ int route_token(const TIn* __restrict__ logits, const float* __restrict__ bias, int t, int E, int k,
                                           int sigmoid, int pre_softmax, int num_groups, int group_topk, float scale,
                                           float* __restrict__ probs, int* __restrict__ idx, long* __restrict__ idx64,
                                           float* __restrict__ full, float* sc, float* ch) {
  // sc [0,E): full scores; ch [0,E): selection scores
  const int lane = threadIdx.x & 31;
  const TIn* lrow = logits + (long)t * E;

  float m = -INFINITY;
  for (int e = lane; e < E; e += 32) {
    const float l = to_f<TIn>(lrow[e]);
    ch[e] = l;
    m = fmaxf(m, l);
  }
  m = pb::warp_max(m);
  if (!sigmoid) {
    float s = 0.f;
    for (int e = lane; e < E; e += 32) {
      const float ex = __expf(ch[e] - m);
      sc[e] = ex;
      s += ex;
    }
    s = pb::warp_sum(s);
    const float inv = 1.f / s;
    for (int e = lane; e < E; e += 32) {
      const float f = sc[e] * inv;
      sc[e] = f;
      if (pre_softmax) ch[e] = f;
    }
  } else {
    for (int e = lane; e < E; e += 32) {
      const float f = 1.f / (1.f + __expf(-ch[e]));
      sc[e] = f;
      ch[e] = bias ? f + bias[e] : f;
    }
  }
  for (int e = lane; e < E; e += 32) full[(long)t * E + e] = sc[e];
  __syncwarp();

  if (num_groups > 1 && group_topk > 0 && group_topk < num_groups) {
    // lane g owns groups g, g + 32, ... (num_groups <= 64 in practice)
    const int gs = E / num_groups;
    float gscore[2] = {-INFINITY, -INFINITY};
    for (int gi = 0; gi < 2; ++gi) {
      const int g = lane + gi * 32;
      if (g < num_groups) {
        float b1 = -INFINITY, b2 = -INFINITY;
        for (int j = 0; j < gs; ++j) {
          const float v = ch[g * gs + j];
          if (v > b1) { b2 = b1; b1 = v; } else if (v > b2) { b2 = v; }
        }
        gscore[gi] = (bias && gs > 1) ? b1 + b2 : b1;
      }
    }
    unsigned long long keep = 0ull;  // bit g: group stays eligible
    for (int it = 0; it < group_topk; ++it) {
      float v = gscore[0];
      int i = lane;
      if (gscore[1] > v) { v = gscore[1]; i = lane + 32; }
      const ArgMax am = warp_argmax(v, i);
      keep |= 1ull << am.i;
      if ((am.i & 31) == lane) gscore[am.i >> 5] = -INFINITY;
    }
    for (int e = lane; e < E; e += 32)
      if (!((keep >> (e / gs)) & 1ull)) ch[e] = -INFINITY;
    __syncwarp();
  }

  // Every lane proposes the best of its experts that are still free, the first of them if none has a score (NaN and -inf count as
  // none: a diverged row, or fewer eligible experts than k).  As k <= E, one always is free: the k selections are distinct experts
  // whatever the row holds, and scores that are no numbers go on into the probabilities.
  float sel_p = 0.f;   // lane j < k keeps the j-th selection
  int sel_i = 0;
  unsigned taken = 0;  // bit n: expert lane + 32 n
  for (int j = 0; j < k; ++j) {
    float v = -INFINITY;
    int i = 0x7fffffff;
    for (int e = lane, n = 0; e < E; e += 32, ++n) {
      const float c = ch[e];
      if (!((taken >> n) & 1u) && (c > v || i == 0x7fffffff)) { v = fmaxf(c, -INFINITY); i = e; }
    }
    i = warp_argmax(v, i).i;
    if (lane == j) {
      sel_i = i;
      sel_p = (!sigmoid && !pre_softmax) ? ch[i] : sc[i];
    }
    if (lane == (i & 31)) taken |= 1u << (i >> 5);
  }
  const bool act = lane < k;
  if (!sigmoid && !pre_softmax) {
    // softmax over the selected logits
    float mm = act ? sel_p : -INFINITY;
    mm = pb::warp_max(mm);
    const float ex = act ? __expf(sel_p - mm) : 0.f;
    const float s = pb::warp_sum(ex);
    sel_p = ex / s;
  } else if (sigmoid && k > 1) {
    const float s = pb::warp_sum(act ? sel_p : 0.f);
    sel_p = sel_p / (s + 1e-20f);
  }
  if (act) {
    probs[(long)t * k + lane] = sel_p * scale;
    idx[(long)t * k + lane] = sel_i;
    if (idx64) idx64[(long)t * k + lane] = sel_i;
  }
  return sel_i;
}

// counts (or null): [E], added to; score_sums (or null): [gridDim.x, E], the sums of full over the CTA's tokens.
template <typename TIn>
__global__ void __launch_bounds__(WARPS * 32)
router_fwd_kernel(const TIn* __restrict__ logits, const float* __restrict__ bias, int T, int E, int k, int sigmoid,
                  int pre_softmax, int num_groups, int group_topk, float scale, float* __restrict__ probs,
                  int* __restrict__ idx, long* __restrict__ idx64, float* __restrict__ full, int* __restrict__ counts,
                  float* __restrict__ score_sums) {
  PB_GRID_WAIT();
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * WARPS + warp;
  float* sc = smem + warp * 2 * E;
  int* hist = reinterpret_cast<int*>(smem + WARPS * 2 * E);
  for (int e = threadIdx.x; e < E; e += WARPS * 32) hist[e] = 0;
  __syncthreads();
  if (t < T) {
    const int sel = route_token<TIn>(logits, bias, t, E, k, sigmoid, pre_softmax, num_groups, group_topk, scale, probs, idx, idx64,
                                     full, sc, sc + E);
    if (lane < k) atomicAdd(hist + sel, 1);
  }
  __syncthreads();
  const int tokens = min(WARPS, T - blockIdx.x * WARPS);
  for (int e = threadIdx.x; e < E; e += WARPS * 32) {
    if (counts && hist[e]) atomicAdd(counts + e, hist[e]);
    if (score_sums) {
      float s = 0.f;
      for (int w = 0; w < tokens; ++w) s += smem[w * 2 * E + e];
      score_sums[(long)blockIdx.x * E + e] = s;
    }
  }
}

// aux = factor * sum_e counts[e] / (T k) * (sum over `blocks` rows of score_sums[:, e]) / T.  A CTA owns 32 experts, its 16 thread
// rows every 16th row of sums; the last CTA to finish (`done`, zero before) adds the CTAs' terms in their order.
constexpr int AUX_COLS = 32, AUX_ROWS = 16;
__global__ void __launch_bounds__(AUX_COLS * AUX_ROWS)
aux_loss_kernel(const float* __restrict__ score_sums, const int* __restrict__ counts, int blocks, int T, int E, int k, float factor,
                int* __restrict__ done, volatile float* __restrict__ terms, float* __restrict__ aux) {
  PB_GRID_WAIT();
  __shared__ float red[AUX_ROWS][AUX_COLS + 1];
  const int c = threadIdx.x % AUX_COLS, g = threadIdx.x / AUX_COLS, e = blockIdx.x * AUX_COLS + c;
  float s = 0.f;
  if (e < E) {
#pragma unroll 8
    for (int b = g; b < blocks; b += AUX_ROWS) s += score_sums[(long)b * E + e];
  }
  red[g][c] = s;
  __syncthreads();
#pragma unroll
  for (int step = AUX_ROWS / 2; step > 0; step >>= 1) {
    if (g < step) red[g][c] += red[g + step][c];
    __syncthreads();
  }
  if (threadIdx.x >= 32) return;
  float term = e < E ? (float)counts[e] / ((float)T * (float)k) * (red[0][c] / (float)T) : 0.f;
  term = pb::warp_sum(term);
  if (threadIdx.x != 0) return;
  terms[blockIdx.x] = term;
  __threadfence();
  if (atomicAdd(done, 1) != (int)gridDim.x - 1) return;
  __threadfence();
  float total = 0.f;
  for (int i = 0; i < (int)gridDim.x; ++i) total += terms[i];
  aux[0] = factor * total;
}

// dlogits [T, E] from dprobs [T, k], dfull [T, E] (may be null), saved full / idx / probs.  daux (or null): the gradient of the
// load-balancing loss, whose own with respect to full[t, e] is aux_factor * f_e / T.
template <typename TOut>
__global__ void __launch_bounds__(WARPS * 32)
router_bwd_kernel(const float* __restrict__ dprobs, const float* __restrict__ dfull, const float* __restrict__ full,
                  const int* __restrict__ idx, const float* __restrict__ probs, int T, int E, int k, int sigmoid,
                  int pre_softmax, float scale, const float* __restrict__ daux, const int* __restrict__ counts, float aux_factor,
                  TOut* __restrict__ dlogits) {
  PB_GRID_WAIT();
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * WARPS + warp;
  if (t >= T) return;
  float* g = smem + warp * E;  // gradient w.r.t. the full scores
  const float da = daux ? *daux * aux_factor : 0.f;
  for (int e = lane; e < E; e += 32) {
    float d = dfull ? dfull[(long)t * E + e] : 0.f;
    if (daux) d += da * ((float)counts[e] / ((float)T * (float)k)) / (float)T;
    g[e] = d;
  }
  __syncwarp();
  const bool act = lane < k;
  const int my_i = act ? idx[(long)t * k + lane] : 0;
  const float dp = act ? dprobs[(long)t * k + lane] * scale : 0.f;   // gradient w.r.t. the unscaled probability
  const float p = act ? probs[(long)t * k + lane] / scale : 0.f;
  const float* frow = full + (long)t * E;
  TOut* drow = dlogits + (long)t * E;
  if (!sigmoid) {
    float extra = 0.f;  // direct logit gradient of the selected entries (post-softmax normalisation)
    if (pre_softmax) {
      if (act) g[my_i] += dp;
    } else {
      const float dot = pb::warp_sum(dp * p);
      extra = p * (dp - dot);
    }
    __syncwarp();
    float dot = 0.f;
    for (int e = lane; e < E; e += 32) dot += g[e] * frow[e];
    dot = pb::warp_sum(dot);
    for (int e = lane; e < E; e += 32) g[e] = frow[e] * (g[e] - dot);
    __syncwarp();
    if (!pre_softmax && act) g[my_i] += extra;
    __syncwarp();
    for (int e = lane; e < E; e += 32) drow[e] = (TOut)g[e];
  } else {
    const float f = act ? frow[my_i] : 0.f;
    float df = dp;
    if (k > 1) {
      const float S = pb::warp_sum(f) + 1e-20f;
      const float dot = pb::warp_sum(dp * f);
      df = dp / S - dot / (S * S);
    }
    if (act) g[my_i] += df;
    __syncwarp();
    for (int e = lane; e < E; e += 32) {
      const float fe = frow[e];
      drow[e] = (TOut)(g[e] * fe * (1.f - fe));
    }
  }
}

}  // namespace

extern "C" {

// logits: [T, E] bf16 (in_bf16 != 0) or fp32.  bias: fp32 [E] or null.  idx64 (or null): idx as 64-bit values.  counts: int [E]
// accumulated (may be null).  score_sums (or null): fp32 [ceil(T / 8), E].
static int router_fwd(const void* logits, int in_bf16, const float* bias, int T, int E, int k, int sigmoid, int pre_softmax,
                      int num_groups, int group_topk, float scale, float* probs, int* idx, long* idx64, float* full, int* counts,
                      float* score_sums, cudaStream_t s) {
  if (E > 1024 || k > 32 || k < 1 || k > E || (num_groups > 1 && (E % num_groups || num_groups > 64))) return -2;
  const int blocks = (T + WARPS - 1) / WARPS;
  const size_t smem = (size_t)(WARPS * 2 + 1) * E * sizeof(float);
  if (smem > 48 * 1024) {
    static std::atomic<bool> allowed[2][pbh::MAX_DEVICES];
    const int rc = in_bf16 ? pbh::allow_shared_memory(router_fwd_kernel<__nv_bfloat16>, 68 * 1024, allowed[0])
                           : pbh::allow_shared_memory(router_fwd_kernel<float>, 68 * 1024, allowed[1]);
    if (rc) return rc;
  }
  if (in_bf16)
    pbh::launch_dependent(router_fwd_kernel<__nv_bfloat16>, blocks, WARPS * 32, smem, s,
        reinterpret_cast<const __nv_bfloat16*>(logits), bias, T, E, k, sigmoid, pre_softmax, num_groups, group_topk,
        scale, probs, idx, idx64, full, counts, score_sums);
  else
    pbh::launch_dependent(router_fwd_kernel<float>, blocks, WARPS * 32, smem, s, reinterpret_cast<const float*>(logits), bias, T, E,
        k, sigmoid, pre_softmax, num_groups, group_topk, scale, probs, idx, idx64, full, counts, score_sums);
  return (int)cudaGetLastError();
}
int pb_router_fwd(const void* logits, int in_bf16, const float* bias, int T, int E, int k, int sigmoid, int pre_softmax,
                  int num_groups, int group_topk, float scale, float* probs, int* idx, float* full, int* counts,
                  cudaStream_t s) {
  return router_fwd(logits, in_bf16, bias, T, E, k, sigmoid, pre_softmax, num_groups, group_topk, scale, probs, idx, nullptr, full,
                    counts, nullptr, s);
}

// pb_router_fwd with counts stored instead of added, and 64-bit copies of the indices.  ws: 32-bit words, E counts and 33 more.
// aux (or null): fp32, receives aux_factor * sum_e f_e P_e; score_sums: fp32 [ceil(T / 8), E], its scratch.
int pb_moe_route(const void* logits, int in_bf16, const float* bias, int T, int E, int k, int sigmoid, int pre_softmax,
                 int num_groups, int group_topk, float scale, float* probs, int* idx, long* idx64, float* full, int* ws,
                 float* aux, float* score_sums, float aux_factor, cudaStream_t s) {
  if (E > 1024 || E < 1) return -2;
  const cudaError_t e = cudaMemsetAsync(ws, 0, (size_t)(E + 1) * sizeof(int), s);
  if (e != cudaSuccess) return (int)e;
  if (T == 0) return aux ? (int)cudaMemsetAsync(aux, 0xff, sizeof(float), s) : 0;      // the mean of nothing
  const int rc = router_fwd(logits, in_bf16, bias, T, E, k, sigmoid, pre_softmax, num_groups, group_topk, scale, probs, idx, idx64, full,
                            ws, aux ? score_sums : nullptr, s);
  if (rc || !aux) return rc;
  pbh::launch_dependent(aux_loss_kernel, (E + AUX_COLS - 1) / AUX_COLS, AUX_COLS * AUX_ROWS, 0, s, score_sums, ws,
      (T + WARPS - 1) / WARPS, T, E, k, aux_factor, ws + E, reinterpret_cast<float*>(ws + E + 1), aux);
  return (int)cudaGetLastError();
}

// dlogits: bf16 (out_bf16 != 0) or fp32.  daux (or null), counts and aux_factor: as the loss of pb_moe_route was made.
int pb_router_bwd(const float* dprobs, const float* dfull, const float* full, const int* idx, const float* probs, int T,
                  int E, int k, int sigmoid, int pre_softmax, float scale, const float* daux, const int* counts, float aux_factor,
                  int out_bf16, void* dlogits, cudaStream_t s) {
  if (E > 1024 || k > 32) return -2;
  if (T == 0) return 0;
  const int blocks = (T + WARPS - 1) / WARPS;
  const size_t smem = (size_t)WARPS * E * sizeof(float);
  if (out_bf16)
    pbh::launch_dependent(router_bwd_kernel<__nv_bfloat16>, blocks, WARPS * 32, smem, s, dprobs, dfull, full, idx, probs, T, E, k,
        sigmoid, pre_softmax, scale, daux, counts, aux_factor, (__nv_bfloat16*)dlogits);
  else
    pbh::launch_dependent(router_bwd_kernel<float>, blocks, WARPS * 32, smem, s, dprobs, dfull, full, idx, probs, T, E, k, sigmoid,
        pre_softmax, scale, daux, counts, aux_factor, (float*)dlogits);
  return (int)cudaGetLastError();
}

}  // extern "C"
