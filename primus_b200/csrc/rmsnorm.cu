// RMSNorm for sm_100a: forward (optional fused residual add) and backward (optional residual gradient).
//
// Rows range from 64 channels (per-head norms: hundreds of thousands of rows) to 16384.  A group of LPR lanes owns a row
// and every lane VPL 16-byte vectors of it, so that short rows share a warp and long ones spread over a CTA, and no lane
// idles at the widths models use (powers of two; other multiples of 8 leave the last vectors of some lanes empty).
//
// Reference call sites these replace: rmsnorm / fused residual norm
// (primus/backends/megatron/core/extensions/primus_turbo.py:1697-1700, fused_residual_rmsnorm.py).
#include "vec.cuh"

namespace {

using pb::Bf8;
using pb::bf8_to_f;
using pb::f_to_bf8;

// Sum over the LPR lanes of a row group; every lane of the group gets it.  LPR > 32: one slot per warp in `red`, which
// the caller does not reuse before another barrier.
template <int LPR>
__device__ __forceinline__ float group_sum(float v, float* red) {
  if (LPR <= 32) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  v = pb::warp_sum(v);
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[warp] = v;
  __syncthreads();
  const float* r = red + warp / (LPR / 32) * (LPR / 32);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < LPR / 32; ++i) s += r[i];
  return s;
}

// ------------------------------------------------------------------ forward
// y = (x [+ res]) * rstd * w ; optionally writes the summed residual stream to xsum.  RPG rows per group: their loads
// are issued together, so a lane has RPG * VPL (about four) 16-byte loads per operand in flight whatever the row length.
// Values stay packed in registers between the two passes: every operand is read from memory once.
template <int LPR, int VPL, int RPG, int THREADS>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ xsum, float* __restrict__ rstd_out, long rows, int H, long ldx,
                   long ldy, float eps) {
  PB_GRID_WAIT();
  __shared__ float red[THREADS / 32];
  const int lane = threadIdx.x % LPR;
  const long row0 = (blockIdx.x * (long)(THREADS / LPR) + threadIdx.x / LPR) * RPG;
  const int nv = H / 8;
  Bf8 v[RPG][VPL], wv[VPL];
  float ss[RPG];
#pragma unroll
  for (int r = 0; r < RPG; ++r)
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (row0 + r < rows && lane + k * LPR < nv)
        v[r][k] = reinterpret_cast<const Bf8*>(x + (row0 + r) * ldx)[lane + k * LPR];
  if (res != nullptr) {
    Bf8 q[RPG][VPL];
#pragma unroll
    for (int r = 0; r < RPG; ++r)
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (row0 + r < rows && lane + k * LPR < nv)
          q[r][k] = reinterpret_cast<const Bf8*>(res + (row0 + r) * ldx)[lane + k * LPR];
#pragma unroll
    for (int r = 0; r < RPG; ++r)
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (row0 + r < rows && lane + k * LPR < nv) {
          float f[8], g[8];
          bf8_to_f(v[r][k], f);
          bf8_to_f(q[r][k], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += g[j];
          v[r][k] = f_to_bf8(f);  // normalise exactly what later layers will read
          reinterpret_cast<Bf8*>(xsum + (row0 + r) * ldx)[lane + k * LPR] = v[r][k];
        }
  }
#pragma unroll
  for (int k = 0; k < VPL; ++k)
    if (lane + k * LPR < nv) wv[k] = reinterpret_cast<const Bf8*>(w)[lane + k * LPR];
#pragma unroll
  for (int r = 0; r < RPG; ++r) {
    ss[r] = 0.f;
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (row0 + r < rows && lane + k * LPR < nv) {
        float f[8];
        bf8_to_f(v[r][k], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[r] += f[j] * f[j];
      }
  }
#pragma unroll
  for (int r = 0; r < RPG; ++r) {
    const float rstd = rsqrtf(group_sum<LPR>(ss[r], red) / H + eps);
    if (row0 + r >= rows) continue;   // (RPG is 1 where group_sum holds a barrier)
    if (lane == 0 && rstd_out) rstd_out[row0 + r] = rstd;
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (lane + k * LPR < nv) {
        float f[8], g[8];
        bf8_to_f(v[r][k], f);
        bf8_to_f(wv[k], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        reinterpret_cast<Bf8*>(y + (row0 + r) * ldy)[lane + k * LPR] = f_to_bf8(f);
      }
  }
}

// Many long rows: CTAs that stay, THREADS threads a row, whose loads run `stages` rows ahead of the row sums through the threads' own
// slots of shared memory, as in the backward; a CTA per row spends its life waiting for its loads, then for its sum (16384 x
// 8192 with residual 183 us, this 172, without 121 and 89; 8192 x 4096 50 and 46, 30 and 23; 1300 x 8192 19 and 14).  Sums in the
// order of the kernel above.  (Three rows ahead or eight CTAs per SM are no faster: 8192 x 5120 63 us against 56.)
// Rows of up to 2048 want twice the CTAs, pay from 16 rows per SM on and without residual: 4096 x 2048 14.3 -> 12.3 us, 16384 x 2048
// 34.8 -> 28.7, 8192 x 1536 18.5 -> 15.4, 2000 x 2048 9.2 -> 10.2; with residual 52.2 -> 53.2 and 24.6 -> 24.6.
constexpr int FWD_STAGES = 2;
inline bool fwd_ring(long rows, int H, bool residual) {
  return H > 2048 ? rows >= 148 * 8 : H > 1024 && !residual && rows >= 148 * 16;
}
template <int VPT, int THREADS, bool RES>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_ring_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                        const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                        __nv_bfloat16* __restrict__ xsum, float* __restrict__ rstd_out, long rows, int H, long ldx,
                        long ldy, float eps) {
  PB_GRID_WAIT();
  extern __shared__ __align__(16) uint8_t ring_raw[];
  __shared__ float red[2][THREADS / 32];
  constexpr int OPS = RES ? 2 : 1;
  Bf8* ring = reinterpret_cast<Bf8*>(ring_raw) + threadIdx.x;      // [stage][operand][k][thread]
  const int tid = threadIdx.x, nv = H / 8;
  auto fetch = [&](long row, int st) {
    if (row < rows) {
      Bf8* slot = ring + st * (OPS * VPT * THREADS);
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        const int i = tid + k * THREADS;
        if (i < nv) {
          pb::cp_async_16(slot + k * THREADS, reinterpret_cast<const Bf8*>(x + row * ldx) + i);
          if (RES) pb::cp_async_16(slot + (VPT + k) * THREADS, reinterpret_cast<const Bf8*>(res + row * ldx) + i);
        }
      }
    }
    pb::cp_async_commit();   // also when empty: the wait below counts groups
  };
  long row = blockIdx.x;
#pragma unroll
  for (int st = 0; st < FWD_STAGES; ++st) fetch(row + (long)st * gridDim.x, st);
  Bf8 wv[VPT];
#pragma unroll
  for (int k = 0; k < VPT; ++k)
    if (tid + k * THREADS < nv) wv[k] = reinterpret_cast<const Bf8*>(w)[tid + k * THREADS];
  int st = 0, flip = 0;
  for (; row < rows; row += gridDim.x, flip ^= 1) {
    pb::cp_async_wait<FWD_STAGES - 1>();
    const Bf8* slot = ring + st * (OPS * VPT * THREADS);
    Bf8 v[VPT];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (tid + k * THREADS < nv) {
        float f[8];
        v[k] = slot[k * THREADS];
        bf8_to_f(v[k], f);
        if (RES) {
          float g[8];
          bf8_to_f(slot[(VPT + k) * THREADS], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += g[j];
          v[k] = f_to_bf8(f);  // normalise exactly what later layers will read
          reinterpret_cast<Bf8*>(xsum + row * ldx)[tid + k * THREADS] = v[k];
          bf8_to_f(v[k], f);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    ss = pb::warp_sum(ss);
    if ((tid & 31) == 0) red[flip][tid >> 5] = ss;
    __syncthreads();           // (the slots of `red` alternate: one barrier a row)
    fetch(row + (long)FWD_STAGES * gridDim.x, st);   // the slot's values are in registers
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) ss += red[flip][i];
    const float rstd = rsqrtf(ss / H + eps);
    if (tid == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (tid + k * THREADS < nv) {
        float f[8], g[8];
        bf8_to_f(v[k], f);
        bf8_to_f(wv[k], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        reinterpret_cast<Bf8*>(y + row * ldy)[tid + k * THREADS] = f_to_bf8(f);
      }
    if (++st == FWD_STAGES) st = 0;
  }
}

template <int VPT, int THREADS, int CTAS, bool RES>
int launch_rmsnorm_fwd_ring(cudaStream_t s, const __nv_bfloat16* x, const __nv_bfloat16* res, const __nv_bfloat16* w, __nv_bfloat16* y,
                            __nv_bfloat16* xsum, float* rstd, long rows, int H, long ldx, long ldy, float eps) {
  constexpr int BYTES = FWD_STAGES * (RES ? 2 : 1) * VPT * THREADS * 16;
  constexpr int PER_SM = 220 * 1024 / BYTES;
  static_assert(PER_SM >= 1, "shared memory");
  auto kern = rmsnorm_fwd_ring_kernel<VPT, THREADS, RES>;
  static std::atomic<bool> allowed[pbh::MAX_DEVICES];
  const int rc = pbh::allow_shared_memory(kern, BYTES, allowed);
  if (rc) return rc;
  pbh::launch_dependent(kern, (unsigned)(pbh::sm_count() * (PER_SM < CTAS ? PER_SM : CTAS)), THREADS, BYTES, s, x, res, w, y, xsum,
                        rstd, rows, H, ldx, ldy, eps);
  return 0;
}

template <typename... Args>
void launch_rmsnorm_fwd(long rows, int H, cudaStream_t s, Args... args) {
  const int nv = H / 8;
#define PB_NORM_FWD(LPR, VPL, RPG, THREADS)                                                             \
  pbh::launch_dependent(rmsnorm_fwd_kernel<LPR, VPL, RPG, THREADS>, \
      (unsigned)((rows + (THREADS / LPR) * RPG - 1) / ((THREADS / LPR) * RPG)), THREADS, 0, s, args...)
  // Few rows do not fill the SMs with four rows (or two, or a row per warp) per group: spread them (768 rows of 256: 3.0 -> 2.2
  // us).  The lines lie where both forms take the same time; 64 lanes of four vectors hold for 1032 to 2048 channels at any
  // number of rows (500 rows of 2048 3.2 us, with 256 lanes of one vector 3.5), 256 lanes of eight above 8192 (4096 rows of
  // 12288 76 us, with 512 lanes of four 85).
  const bool few = rows * nv < 148 * 2048L;
  if (nv <= 8) { if (few) PB_NORM_FWD(8, 1, 1, 128); else PB_NORM_FWD(8, 1, 4, 128); }
  else if (nv <= 16) { if (few) PB_NORM_FWD(16, 1, 1, 128); else PB_NORM_FWD(16, 1, 4, 128); }
  else if (nv <= 32) { if (few) PB_NORM_FWD(32, 1, 1, 128); else PB_NORM_FWD(32, 1, 4, 128); }
  else if (nv <= 64) { if (few) PB_NORM_FWD(32, 2, 1, 128); else PB_NORM_FWD(32, 2, 2, 128); }
  else if (nv <= 128 && rows * nv >= 148 * 256L) PB_NORM_FWD(32, 4, 1, 128);
  else if (nv <= 256) PB_NORM_FWD(64, 4, 1, 128);
  else if (nv <= 512) PB_NORM_FWD(128, 4, 1, 128);
  else if (nv <= 1024) PB_NORM_FWD(256, 4, 1, 256);
  else PB_NORM_FWD(256, 8, 1, 256);
#undef PB_NORM_FWD
}

// ------------------------------------------------------------------ backward
// dx = rstd * (dy*w) - x * rstd^3 * mean(dy*w*x)  (+ dres when given)
// dx2 (optional) receives dx once more: first gradients of two leaves, which autograd would have to copy otherwise (a layer used
// by itself; inside a model the two inputs are no leaves).  16384 x 8192: a second store 41 us, the copy 83 us.
// y (optional) receives the normalised rows again, for the weight gradient of a linear layer that followed the norm and does not
// store its input: x and rstd are here already, and a pass of its own reads x once more (8192 x 4096 with
// residual: 50 + 23 us in two passes, 58 in one; 4096 x 2048 21 + 12 and 23).
// dw partial sums per CTA go to `partial` [gridDim.x, H]; rmsnorm_dw_reduce_kernel folds them.

// word j of a vector as two fp32 values and back
__device__ __forceinline__ uint64_t widen(const Bf8& b, int j) {
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&b.v[j]);
  return pb::pack_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ void narrow(uint64_t f, Bf8& b, int j) {
  float lo, hi;
  pb::unpack_f32x2(f, lo, hi);
  b.v[j] = __floats2bfloat162_rn(lo, hi);
}

// Rows of up to 1024 channels: LPR <= 32 lanes per row, no barrier in the loop, RPG rows per group in flight.  The dw
// sums of a CTA's groups meet in shared memory at the end.
// PACKED: two channels per fp32 instruction (the same bits; us without and with: 262144 x 192 91 -> 83, 262144 x 128 52 -> 48, 32768 x 512
// with residual 33.8 -> 31.7, 32768 x 1024 52 -> 46).  Rows of more than 512 with a residual hold too much for register pairs: 16384 x
// 1024 36 -> 40.
template <bool PACKED>
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  if (PACKED) return pb::mul_f32x2(a, b);
  float a0, a1, b0, b1;
  pb::unpack_f32x2(a, a0, a1);
  pb::unpack_f32x2(b, b0, b1);
  return pb::pack_f32x2(a0 * b0, a1 * b1);
}
template <bool PACKED>
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  if (PACKED) return pb::fma_f32x2(a, b, c);
  float a0, a1, b0, b1, c0, c1;
  pb::unpack_f32x2(a, a0, a1);
  pb::unpack_f32x2(b, b0, b1);
  pb::unpack_f32x2(c, c0, c1);
  return pb::pack_f32x2(fmaf(a0, b0, c0), fmaf(a1, b1, c1));
}
template <int LPR, int VPL, int RPG, bool Y, bool PACKED>
__global__ void __launch_bounds__(256, 2)
rmsnorm_bwd_short_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                         const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                         const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                         __nv_bfloat16* __restrict__ dx2, __nv_bfloat16* __restrict__ y, float* __restrict__ partial, long rows,
                         int H, long ldx, long lddy) {
  PB_GRID_WAIT();
  constexpr int GROUPS = 256 / LPR;
  __shared__ float4 sums[GROUPS][LPR * VPL * 2];
  const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR;
  const int nv = H / 8;
  Bf8 wv[VPL];
  uint64_t dw[VPL][4];
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
#pragma unroll
    for (int j = 0; j < 4; ++j) dw[k][j] = 0;
    if (lane + k * LPR < nv) wv[k] = reinterpret_cast<const Bf8*>(w)[lane + k * LPR];
  }
  const long stride = (long)gridDim.x * GROUPS * RPG;
  // the loop bound is the CTA's first row: all lanes of a warp run the same number of iterations (shuffles inside)
  for (long base = (long)blockIdx.x * GROUPS * RPG; base < rows; base += stride) {
    const long row0 = base + grp * RPG;
    Bf8 vx[RPG][VPL], vg[RPG][VPL], vr[RPG][VPL];
    float rs[RPG];
#pragma unroll
    for (int r = 0; r < RPG; ++r) {
      rs[r] = 0.f;
      if (row0 + r < rows) rs[r] = rstd[row0 + r];
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (row0 + r < rows && lane + k * LPR < nv) {
          vx[r][k] = reinterpret_cast<const Bf8*>(x + (row0 + r) * ldx)[lane + k * LPR];
          vg[r][k] = reinterpret_cast<const Bf8*>(dy + (row0 + r) * lddy)[lane + k * LPR];
          if (dres) vr[r][k] = reinterpret_cast<const Bf8*>(dres + (row0 + r) * ldx)[lane + k * LPR];
        }
    }
#pragma unroll
    for (int r = 0; r < RPG; ++r) {
      const uint64_t rs2 = pb::pack_f32x2(rs[r], rs[r]);
      float dot = 0.f;
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (row0 + r < rows && lane + k * LPR < nv) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t px = widen(vx[r][k], j), pg = widen(vg[r][k], j), pw = widen(wv[k], j);
            dw[k][j] = fma2<PACKED>(mul2<PACKED>(pg, px), rs2, dw[k][j]);
            float x0, x1, d0, d1;
            pb::unpack_f32x2(px, x0, x1);
            pb::unpack_f32x2(mul2<PACKED>(pg, pw), d0, d1);
            dot = fmaf(d0, x0, dot);
            dot = fmaf(d1, x1, dot);
          }
        }
      dot = group_sum<LPR>(dot, nullptr);
      const float c = dot * rs[r] * rs[r] * rs[r] / H;
      const uint64_t c2 = pb::pack_f32x2(-c, -c);
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (row0 + r < rows && lane + k * LPR < nv) {
          Bf8 ob, yv;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t px = widen(vx[r][k], j), pw = widen(wv[k], j);
            float o0, o1, r0 = 0.f, r1 = 0.f;
            pb::unpack_f32x2(fma2<PACKED>(mul2<PACKED>(widen(vg[r][k], j), pw), rs2, mul2<PACKED>(px, c2)), o0, o1);
            if (Y) narrow(mul2<PACKED>(mul2<PACKED>(px, rs2), pw), yv, j);
            if (dres) {
              pb::unpack_f32x2(widen(vr[r][k], j), r0, r1);
              o0 += r0;
              o1 += r1;
            }
            ob.v[j] = __floats2bfloat162_rn(o0, o1);
          }
          if (Y) reinterpret_cast<Bf8*>(y + (row0 + r) * ldx)[lane + k * LPR] = yv;
          reinterpret_cast<Bf8*>(dx + (row0 + r) * ldx)[lane + k * LPR] = ob;
          if (dx2) reinterpret_cast<Bf8*>(dx2 + (row0 + r) * ldx)[lane + k * LPR] = ob;
        }
    }
  }
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float4 v;
      pb::unpack_f32x2(dw[k][2 * q], v.x, v.y);
      pb::unpack_f32x2(dw[k][2 * q + 1], v.z, v.w);
      sums[grp][(lane + k * LPR) * 2 + q] = v;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nv * 2; i += 256) {
    float4 t = sums[0][i];
#pragma unroll
    for (int g = 1; g < GROUPS; ++g) {
      const float4 u = sums[g][i];
      t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
    }
    reinterpret_cast<float4*>(partial + (long)blockIdx.x * H)[i] = t;
  }
}

// Longer rows: one CTA per row, persistent over rows blockIdx.x, blockIdx.x + gridDim.x, ...  Every thread keeps a ring
// of STAGES rows of its own vectors in shared memory, filled by its own 16-byte cp.async copies, so loads run several
// rows ahead of the block reductions without holding registers; the reduction is the only barrier of a row (its slots
// alternate).  Two channels share an fp32 instruction but for the row sum, whose order stands, and the residual, whose packed
// addend would spill: us with single values and now, 16384 x 8192 with residual 175 -> 165, 8192 x 4096 52.2 -> 50.2 and 44 -> 42
// without, 16384 x 2048 without 50 -> 46.
template <int VPT, int THREADS, bool RES, bool Y>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   __nv_bfloat16* __restrict__ dx2, __nv_bfloat16* __restrict__ y, float* __restrict__ partial, long rows, int H,
                   long ldx, long lddy, int stages) {
  PB_GRID_WAIT();
  extern __shared__ __align__(16) uint8_t ring_raw[];
  __shared__ float red[2][THREADS / 32];
  constexpr int OPS = RES ? 3 : 2;
  Bf8* ring = reinterpret_cast<Bf8*>(ring_raw);   // [stage][operand][k][thread]
  const int tid = threadIdx.x;
  const int nv = H / 8;
  Bf8 wv[VPT];
  uint64_t dw[VPT][4];
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
#pragma unroll
    for (int j = 0; j < 4; ++j) dw[k][j] = 0;
    if (tid + k * THREADS < nv) wv[k] = reinterpret_cast<const Bf8*>(w)[tid + k * THREADS];
  }
  auto fetch = [&](long row, int st) {
    if (row < rows) {
      Bf8* slot = ring + (long)st * OPS * VPT * THREADS + tid;
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        const int i = tid + k * THREADS;
        if (i < nv) {
          pb::cp_async_16(slot + k * THREADS, reinterpret_cast<const Bf8*>(x + row * ldx) + i);
          pb::cp_async_16(slot + (VPT + k) * THREADS, reinterpret_cast<const Bf8*>(dy + row * lddy) + i);
          if (RES) pb::cp_async_16(slot + (2 * VPT + k) * THREADS, reinterpret_cast<const Bf8*>(dres + row * ldx) + i);
        }
      }
    }
    pb::cp_async_commit();   // also when empty: the wait below counts groups
  };
  // two ring sizes: the wait needs a constant
  auto wait_oldest = [&]() {
    if (stages == 4) pb::cp_async_wait<3>();
    else pb::cp_async_wait<1>();
  };
  long row = blockIdx.x;
  for (int st = 0; st < stages; ++st) fetch(row + (long)st * gridDim.x, st);
  float rs = row < rows ? rstd[row] : 0.f;
  int st = 0, flip = 0;
  for (; row < rows; row += gridDim.x) {
    const long next = row + gridDim.x;
    const float rs_next = next < rows ? rstd[next] : 0.f;
    wait_oldest();
    const Bf8* slot = ring + (long)st * OPS * VPT * THREADS + tid;
    Bf8 vx[VPT], vg[VPT], vr[VPT];
    const uint64_t rs2 = pb::pack_f32x2(rs, rs);
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (tid + k * THREADS < nv) {
        vx[k] = slot[k * THREADS];
        vg[k] = slot[(VPT + k) * THREADS];
        if (RES) vr[k] = slot[(2 * VPT + k) * THREADS];
        Bf8 yv;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint64_t px = widen(vx[k], j), pg = widen(vg[k], j), pw = widen(wv[k], j);
          dw[k][j] = pb::fma_f32x2(pb::mul_f32x2(pg, px), rs2, dw[k][j]);
          float x0, x1, d0, d1;
          pb::unpack_f32x2(px, x0, x1);
          pb::unpack_f32x2(pb::mul_f32x2(pg, pw), d0, d1);
          dot = fmaf(d0, x0, dot);
          dot = fmaf(d1, x1, dot);
          if (Y) narrow(pb::mul_f32x2(pb::mul_f32x2(px, rs2), pw), yv, j);
        }
        if (Y) reinterpret_cast<Bf8*>(y + row * ldx)[tid + k * THREADS] = yv;
      }
    dot = pb::warp_sum(dot);
    if ((tid & 31) == 0) red[flip][tid >> 5] = dot;
    __syncthreads();
    // the slot's values are in registers (the sum above used them; vr is pinned by the barrier's memory clobber)
    fetch(row + (long)stages * gridDim.x, st);
    dot = 0.f;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) dot += red[flip][i];
    const float c = dot * rs * rs * rs / H;
    const uint64_t c2 = pb::pack_f32x2(-c, -c);
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (tid + k * THREADS < nv) {
        Bf8 ob;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint64_t gw = pb::mul_f32x2(widen(vg[k], j), widen(wv[k], j)), px = widen(vx[k], j);
          float o0, o1, r0 = 0.f, r1 = 0.f;
          pb::unpack_f32x2(pb::fma_f32x2(gw, rs2, pb::mul_f32x2(px, c2)), o0, o1);
          if (RES) pb::unpack_f32x2(widen(vr[k], j), r0, r1);
          ob.v[j] = RES ? __floats2bfloat162_rn(o0 + r0, o1 + r1) : __floats2bfloat162_rn(o0, o1);
        }
        reinterpret_cast<Bf8*>(dx + row * ldx)[tid + k * THREADS] = ob;
        if (RES && dx2) reinterpret_cast<Bf8*>(dx2 + row * ldx)[tid + k * THREADS] = ob;
      }
    rs = rs_next;
    flip ^= 1;
    if (++st == stages) st = 0;
  }
#pragma unroll
  for (int k = 0; k < VPT; ++k)
    if (tid + k * THREADS < nv) {
      float4* p = reinterpret_cast<float4*>(partial + (long)blockIdx.x * H + (long)(tid + k * THREADS) * 8);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float4 v;
        pb::unpack_f32x2(dw[k][2 * q], v.x, v.y);
        pb::unpack_f32x2(dw[k][2 * q + 1], v.z, v.w);
        p[q] = v;
      }
    }
}

// CTAs (= partial rows) of the backward: two per SM, fewer when there are fewer rows
constexpr int BWD_MAX_PARTIALS = 296;

// CTAs that `rows` rows of H channels keep busy, out of at most P.  Every CTA's partial row costs the reduction as much as a row
// of the CTA's own, so few rows take one CTA per SM, and short ones (a warp or less per row) one per eight rows: 200 rows of
// 128 4.5 us instead of 5.9, 290 of 1536 5.5 instead of 6.4.
inline bool bwd_row_per_warp(long rows, int H) { return H <= 512 || (H <= 1024 && rows >= 148 * 16); }
inline int bwd_ctas(int P, long rows, int H) {
  long n = P;
  if (bwd_row_per_warp(rows, H)) { if (rows < 148 * 16) n = (rows + 7) / 8 < 148 ? (rows + 7) / 8 : 148; }
  else if (rows <= 148 * 4) n = 148;
  return (int)(n < P ? n : P);
}

template <int VPT, int THREADS, bool RES, bool Y>
int launch_rmsnorm_bwd_ring(int P, cudaStream_t s, const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w,
                            const float* rstd, const __nv_bfloat16* dres, __nv_bfloat16* dx, __nv_bfloat16* dx2,
                            __nv_bfloat16* y, float* partial, long rows, int H, long ldx, long lddy) {
  constexpr int STAGE = (RES ? 3 : 2) * VPT * THREADS * 16;
  // four rows ahead where two CTAs of an SM then still fit into its shared memory, else two
  constexpr int STAGES = 4 * STAGE <= 100 * 1024 ? 4 : 2;
  auto kern = rmsnorm_bwd_kernel<VPT, THREADS, RES, Y>;
  static std::atomic<bool> allowed[pbh::MAX_DEVICES];
  const int rc = pbh::allow_shared_memory(kern, STAGES * STAGE, allowed);
  if (rc) return rc;
  pbh::launch_dependent(kern, P, THREADS, STAGES * STAGE, s, dy, x, w, rstd, dres, dx, dx2, y, partial, rows, H, ldx, lddy, STAGES);
  return (int)cudaGetLastError();
}

int launch_rmsnorm_bwd(int P, cudaStream_t s, const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w,
                       const float* rstd, const __nv_bfloat16* dres, __nv_bfloat16* dx, __nv_bfloat16* dx2, __nv_bfloat16* y,
                       float* partial, long rows, int H, long ldx, long lddy) {
  const int nv = H / 8;
#define PB_NORM_BWD_SHORT(LPR, VPL, RPG)                                                                               \
  {                                                                                                                    \
    auto kern = VPL == 4 && dres                                                                                       \
                    ? (y ? rmsnorm_bwd_short_kernel<LPR, VPL, RPG, (LPR > 8), VPL != 4>                                \
                         : rmsnorm_bwd_short_kernel<LPR, VPL, RPG, false, VPL != 4>)                                   \
                    : (y ? rmsnorm_bwd_short_kernel<LPR, VPL, RPG, (LPR > 8), true>                                    \
                         : rmsnorm_bwd_short_kernel<LPR, VPL, RPG, false, true>);                                      \
    pbh::launch_dependent(kern, P, 256, 0, s, dy, x, w, rstd, dres, dx, dx2, y, partial, rows, H, ldx, lddy);                   \
    return (int)cudaGetLastError();                                                                                    \
  }
#define PB_NORM_BWD_RING(VPT, THREADS, RES, Y) \
  launch_rmsnorm_bwd_ring<VPT, THREADS, RES, Y>(P, s, dy, x, w, rstd, dres, dx, dx2, y, partial, rows, H, ldx, lddy)
#define PB_NORM_BWD(VPT, THREADS)                                                                                  \
  return dres ? (y ? PB_NORM_BWD_RING(VPT, THREADS, true, true) : PB_NORM_BWD_RING(VPT, THREADS, true, false))     \
              : (y ? PB_NORM_BWD_RING(VPT, THREADS, false, true) : PB_NORM_BWD_RING(VPT, THREADS, false, false))
  const bool few = rows * nv < 148 * 512L * 4;   // (two CTAs of 256 threads per SM)
  if (nv <= 8) { if (few) PB_NORM_BWD_SHORT(8, 1, 1) else PB_NORM_BWD_SHORT(8, 1, 4) }
  if (nv <= 16) { if (few) PB_NORM_BWD_SHORT(16, 1, 1) else PB_NORM_BWD_SHORT(16, 1, 4) }
  if (nv <= 32) { if (few) PB_NORM_BWD_SHORT(32, 1, 1) else PB_NORM_BWD_SHORT(32, 1, 4) }
  if (nv <= 64) PB_NORM_BWD_SHORT(32, 2, 2)
  // (a row per warp leaves most warps without one up to some two thousand rows: 40 rows of 1024 4.8 us with a row per CTA, 6.7
  // with a row per warp, 1500 rows 8.3 and 9.7 us, 8192 rows 19.4 and 18.8 us)
  if (bwd_row_per_warp(rows, H)) PB_NORM_BWD_SHORT(32, 4, 1)
  if (nv <= 256) PB_NORM_BWD(1, 256);
  if (nv <= 512) PB_NORM_BWD(2, 256);
  if (nv <= 1024) PB_NORM_BWD(4, 256);
  PB_NORM_BWD(4, 512);
#undef PB_NORM_BWD
#undef PB_NORM_BWD_RING
#undef PB_NORM_BWD_SHORT
}

// ------------------------------------------------------------------ per-head norms of q and k in a packed QKV tensor
// qkv [T, (hq + 2 hkv) * d] = [q heads | k heads | v heads]: every q and k head is normalised with its own gain (wq / wk),
// v heads are copied, and the result is packed the same way, so that nothing is sliced, copied or concatenated around the
// norms.  ROPE: the q and k heads are then rotated (rotate-half in their first rot_dim channels, as rope_kernel does it), which as
// passes of its own reads and writes them once more in each direction.
// A group of LPR lanes owns a head row and a lane two 16-byte vectors of it, those that rotate with one another: no exchange but
// the row's sum, and the pair shares its table entries, which stay for the rows of one token that a group takes in turn.  (One
// vector per lane, twice the shuffles and three times the instructions: 4096 x 32 / 4 x 128 forward with rotation 29 us, two
// passes 39, this 23; backward 57, 64 and 50.)
struct Rope {
  const int* pos;                       // row of the tables, or null: the token's number
  const float *cos_t, *sin_t;           // [positions, rot_dim / 2]
  int rot_dim;
};
struct HeadLane {                       // a lane's two vectors of a head row of d channels
  int a, b;
  bool ina, inb, turns;
  template <bool ROPE>
  static __device__ __forceinline__ HeadLane make(int lane, int d, int rot_dim) {
    const int nv = d / 8, half8 = ROPE ? rot_dim / 16 : (nv + 1) / 2;
    HeadLane l;
    l.turns = ROPE && lane < half8;
    l.a = lane < half8 ? lane : 2 * half8 + 2 * (lane - half8);
    l.b = lane < half8 ? lane + half8 : l.a + 1;
    l.ina = l.a < nv;
    l.inb = l.b < nv;
    return l;
  }
};
struct HeadRow {                        // a head row; stepping to the next costs no division
  long t;
  int h, heads;
  __device__ __forceinline__ HeadRow(long row, int heads_) : heads(heads_) {
    t = row >> 32 ? row / heads_ : (long)((unsigned)row / (unsigned)heads_);
    h = (int)(row - t * heads_);
  }
  __device__ __forceinline__ void next() {
    if (++h == heads) { h = 0; ++t; }
  }
};
// the entries of token t for the lane's pair
__device__ __forceinline__ void rope_entries(const Rope& rp, long t, int lane, float (&c)[8], float (&s)[8]) {
  const long at = ((long)(rp.pos ? rp.pos[t] : (int)t) * (rp.rot_dim / 16) + lane) * 8;
#pragma unroll
  for (int j = 0; j < 8; j += 4) {
    *reinterpret_cast<float4*>(c + j) = *reinterpret_cast<const float4*>(rp.cos_t + at + j);
    *reinterpret_cast<float4*>(s + j) = *reinterpret_cast<const float4*>(rp.sin_t + at + j);
  }
}
__device__ __forceinline__ void rope_pair(Bf8& a, Bf8& b, const float (&c)[8], const float (&s)[8], float sign) {
  float fa[8], fb[8], oa[8], ob[8];
  bf8_to_f(a, fa);
  bf8_to_f(b, fb);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sn = s[j] * sign;
    oa[j] = fa[j] * c[j] - fb[j] * sn;
    ob[j] = fb[j] * c[j] + fa[j] * sn;
  }
  a = f_to_bf8(oa);
  b = f_to_bf8(ob);
}
// Neighbouring head rows, mostly of one token, that a group takes in turn.  Forward, all loaded at once: two rows and 32 warps per SM
// 16.7 us at 4096 x 32 / 4 x 128, four rows and 16 warps 18.9.
constexpr int QK_FWD_RUN = 2, QK_RUN = 4;

template <int LPR, bool ROPE>
__global__ void __launch_bounds__(128, 8)
qk_norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wq,
                   const __nv_bfloat16* __restrict__ wk, __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out,
                   long rows, int hq, int hkv, int d, long ldx, long ldy, float eps, Rope rp) {
  PB_GRID_WAIT();
  const int lane = threadIdx.x % LPR;
  const long row0 = (blockIdx.x * (long)(128 / LPR) + threadIdx.x / LPR) * QK_FWD_RUN;
  const HeadLane l = HeadLane::make<ROPE>(lane, d, rp.rot_dim);
  const HeadRow first(row0, hq + 2 * hkv);
  Bf8 va[QK_FWD_RUN], vb[QK_FWD_RUN];
  HeadRow at = first;
  float c[8], s[8];
  if (ROPE && row0 < rows && l.turns) rope_entries(rp, at.t, lane, c, s);
#pragma unroll
  for (int r = 0; r < QK_FWD_RUN; ++r, at.next()) {
    const Bf8* src = reinterpret_cast<const Bf8*>(x + at.t * ldx + (long)at.h * d);
    if (row0 + r < rows && l.ina) va[r] = src[l.a];
    if (row0 + r < rows && l.inb) vb[r] = src[l.b];
  }
  at = first;
#pragma unroll
  for (int r = 0; r < QK_FWD_RUN; ++r, at.next()) {
    const bool live = row0 + r < rows, norm = at.h < hq + hkv;
    if (ROPE && live && l.turns && r > 0 && at.h == 0) rope_entries(rp, at.t, lane, c, s);
    float f[8], g[8], sa = 0.f, sb = 0.f;
    if (live && l.ina) {
      bf8_to_f(va[r], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sa += f[j] * f[j];
    }
    if (live && l.inb) {
      bf8_to_f(vb[r], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sb += f[j] * f[j];
    }
    const float rstd = rsqrtf(group_sum<LPR>(sa + sb, nullptr) / d + eps);
    if (!live) continue;
    if (norm) {
      const Bf8* w = reinterpret_cast<const Bf8*>(at.h < hq ? wq : wk);
      if (l.ina) {
        bf8_to_f(va[r], f);
        bf8_to_f(w[l.a], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        va[r] = f_to_bf8(f);
      }
      if (l.inb) {
        bf8_to_f(vb[r], f);
        bf8_to_f(w[l.b], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        vb[r] = f_to_bf8(f);
      }
      if (ROPE && l.turns) rope_pair(va[r], vb[r], c, s, 1.f);
      if (lane == 0) rstd_out[at.t * (hq + hkv) + at.h] = rstd;
    }
    Bf8* dst = reinterpret_cast<Bf8*>(y + at.t * ldy + (long)at.h * d);
    if (l.ina) dst[l.a] = va[r];
    if (l.inb) dst[l.b] = vb[r];
  }
}

// (two fp32 values per instruction: channel j of the lane's two vectors, so that each vector's sums keep their order)
struct Pairs {
  uint64_t v[8];
};
__device__ __forceinline__ Pairs unpack_pairs(const Bf8& a, const Bf8& b) {
  Pairs p;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t wa = *reinterpret_cast<const uint32_t*>(&a.v[i]), wb = *reinterpret_cast<const uint32_t*>(&b.v[i]);
    p.v[2 * i] = pb::pack_f32x2(__uint_as_float(wa << 16), __uint_as_float(wb << 16));
    p.v[2 * i + 1] = pb::pack_f32x2(__uint_as_float(wa & 0xffff0000u), __uint_as_float(wb & 0xffff0000u));
  }
  return p;
}
__device__ __forceinline__ void pack_pairs(const Pairs& p, Bf8& a, Bf8& b) {
  float fa[8], fb[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) pb::unpack_f32x2(p.v[j], fa[j], fb[j]);
  a = f_to_bf8(fa);
  b = f_to_bf8(fb);
}
// the gains of the lane's channels for q or k heads
struct HeadGains {
  Bf8 a, b;
  bool of_q;
  __device__ __forceinline__ void load(const __nv_bfloat16* wq, const __nv_bfloat16* wk, bool q, const HeadLane& l) {
    const Bf8* w = reinterpret_cast<const Bf8*>(q ? wq : wk);
    of_q = q;
    if (l.ina) a = w[l.a];
    if (l.inb) b = w[l.b];
  }
};

// Backward: dx of the q and k heads (ROPE: of gradients that are rotated back first), the v gradient copied; gain sums per CTA
// in partial [gridDim.x, 2 d] (q, then k).  A lane's copies of its vectors run QK_STAGES rows ahead, through slots of its own in
// shared memory (registers for as many rows left two CTAs of 256 threads per SM waiting for memory most of the time), and the
// arithmetic runs on pairs of values, which its issue is bound by.
constexpr int QK_STAGES = 4;
template <int LPR, bool ROPE>
__global__ void __launch_bounds__(256, 2)
qk_norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk,
                   const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, long rows,
                   int hq, int hkv, int d, long ldx, long lddy, long lddx, Rope rp) {
  PB_GRID_WAIT();
  constexpr int GROUPS = 256 / LPR;
  extern __shared__ __align__(16) uint8_t ring_raw[];
  Bf8* slots = reinterpret_cast<Bf8*>(ring_raw) + threadIdx.x;     // [stage][dy a, dy b, x a, x b][thread]
  const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR;
  const HeadLane l = HeadLane::make<ROPE>(lane, d, rp.rot_dim);
  const int heads = hq + 2 * hkv;
  const long runs = (rows + QK_RUN - 1) / QK_RUN, step = (long)gridDim.x * GROUPS;
  Pairs dw[2] = {};                      // gain sums of the lane's channels: q heads, k heads

  // the row after the last one fetched: run `frun`, `fr` rows into it
  long frun = (long)blockIdx.x * GROUPS + grp;
  int fr = 0;
  HeadRow fat(frun * QK_RUN, heads);
  auto fetch = [&](int st) {
    if (frun < runs && frun * QK_RUN + fr < rows) {
      Bf8* sl = slots + st * 4 * 256;
      const Bf8* g = reinterpret_cast<const Bf8*>(dy + fat.t * lddy + (long)fat.h * d);
      if (l.ina) pb::cp_async_16(sl, g + l.a);
      if (l.inb) pb::cp_async_16(sl + 256, g + l.b);
      if (fat.h < hq + hkv) {
        const Bf8* v = reinterpret_cast<const Bf8*>(x + fat.t * ldx + (long)fat.h * d);
        if (l.ina) pb::cp_async_16(sl + 512, v + l.a);
        if (l.inb) pb::cp_async_16(sl + 768, v + l.b);
      }
    }
    pb::cp_async_commit();               // also when empty: the wait below counts groups
    fat.next();
    if (++fr == QK_RUN) {
      fr = 0;
      frun += step;
      fat = HeadRow(frun * QK_RUN, heads);
    }
  };
#pragma unroll
  for (int st = 0; st < QK_STAGES; ++st) fetch(st);
  HeadGains w{};
  w.load(wq, wk, true, l);
  // the loop bound is the CTA's first run: all lanes of a warp make the same number of turns (shuffles inside)
  for (long base = (long)blockIdx.x * GROUPS; base < runs; base += step) {
    const long row0 = (base + grp) * QK_RUN;
    HeadRow at(row0, heads);
    float c[8], s[8], rs_run[QK_RUN];
    if (ROPE && row0 < rows && l.turns) rope_entries(rp, at.t, lane, c, s);
#pragma unroll
    for (int r = 0; r < QK_RUN; ++r) {
      const int h = at.h + r < heads ? at.h + r : at.h + r - heads;          // (a run of more than two tokens: below)
      const long t = at.h + r < heads ? at.t : at.t + 1;
      rs_run[r] = heads >= QK_RUN && row0 + r < rows && h < hq + hkv ? rstd[t * (hq + hkv) + h] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < QK_RUN; ++r, at.next()) {
      static_assert(QK_RUN == QK_STAGES, "row r of a run is in slot r");
      const int h = at.h;
      const bool live = row0 + r < rows, norm = live && h < hq + hkv;
      float rs = rs_run[r];
      if (heads < QK_RUN) rs = norm ? rstd[at.t * (hq + hkv) + h] : 0.f;
      if (ROPE && live && l.turns && r > 0 && h == 0) rope_entries(rp, at.t, lane, c, s);
      if (norm && (h < hq) != w.of_q) w.load(wq, wk, h < hq, l);
      pb::cp_async_wait<QK_STAGES - 1>();
      const Bf8* sl = slots + r * 4 * 256;
      Bf8 ga{}, gb{}, xa{}, xb{};
      if (live && l.ina) ga = sl[0];
      if (live && l.inb) gb = sl[256];
      if (norm && l.ina) xa = sl[512];
      if (norm && l.inb) xb = sl[768];
      if (ROPE && norm && l.turns) rope_pair(ga, gb, c, s, -1.f);
      const Pairs fx = unpack_pairs(xa, xb);
      Pairs fg = unpack_pairs(ga, gb);
      uint64_t dots = 0;
      if (norm) {
        const Pairs fw = unpack_pairs(w.a, w.b);
        const uint64_t rr = pb::pack_f32x2(rs, rs);
        auto products = [&](Pairs& sum) {
#pragma unroll
          for (int j = 0; j < 8; ++j) sum.v[j] = pb::fma_f32x2(pb::mul_f32x2(fg.v[j], fx.v[j]), rr, sum.v[j]);
        };
        if (h < hq) products(dw[0]);
        else products(dw[1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          fg.v[j] = pb::mul_f32x2(fg.v[j], fw.v[j]);
          dots = pb::fma_f32x2(fg.v[j], fx.v[j], dots);
        }
      }
      float da, db;
      pb::unpack_f32x2(dots, da, db);
      const float dot = group_sum<LPR>(da + db, nullptr);
      if (norm) {
        const float k = dot * rs * rs * rs / d;
        const uint64_t rr = pb::pack_f32x2(rs, rs), nk = pb::pack_f32x2(-k, -k);
#pragma unroll
        for (int j = 0; j < 8; ++j) fg.v[j] = pb::fma_f32x2(fg.v[j], rr, pb::mul_f32x2(fx.v[j], nk));
        pack_pairs(fg, ga, gb);
      }
      if (live) {
        Bf8* dst = reinterpret_cast<Bf8*>(dx + at.t * lddx + (long)h * d);
        if (l.ina) dst[l.a] = ga;
        if (l.inb) dst[l.b] = gb;
      }
      fetch(r);                          // (the slot's values are in registers: the lane's own, used above)
    }
  }
  pb::cp_async_wait<0>();
  // sums of the CTA's groups, through the ring's memory: GROUPS x d floats fit into it
  float* sums = reinterpret_cast<float*>(ring_raw);
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float a, b;
      pb::unpack_f32x2(dw[w].v[j], a, b);
      if (l.ina) sums[grp * d + l.a * 8 + j] = a;
      if (l.inb) sums[grp * d + l.b * 8 + j] = b;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < d; i += 256) {
      float t = sums[i];
      for (int g = 1; g < GROUPS; ++g) t += sums[g * d + i];
      partial[(long)blockIdx.x * 2 * d + w * d + i] = t;
    }
  }
}

// dw[h] (+)= sum_p partial[p, h].  A CTA owns 32 columns; its 16 thread rows each add every 16th partial (coalesced
// 128-byte reads, eight in flight) and a fixed-order tree in shared memory folds them, so the result does not depend on
// scheduling.
constexpr int DWR_COLS = 32, DWR_ROWS = 16;
constexpr int DW_STORE_BF16 = 2;     // of `accumulate`: dw is a bf16 vector, and stored
__global__ void __launch_bounds__(DWR_COLS * DWR_ROWS)
rmsnorm_dw_reduce_kernel(const float* __restrict__ partial, float* __restrict__ dw, int P, int H, long ld, int accumulate) {
  PB_GRID_WAIT();
  __shared__ float red[DWR_ROWS][DWR_COLS + 1];
  const int c = threadIdx.x % DWR_COLS, g = threadIdx.x / DWR_COLS;
  const int h = blockIdx.x * DWR_COLS + c;
  float s = 0.f;
  if (h < H) {
#pragma unroll 8
    for (int p = g; p < P; p += DWR_ROWS) s += partial[p * ld + h];
  }
  red[g][c] = s;
  __syncthreads();
#pragma unroll
  for (int step = DWR_ROWS / 2; step > 0; step >>= 1) {
    if (g < step) red[g][c] += red[g + step][c];
    __syncthreads();
  }
  if (g == 0 && h < H) {
    if (accumulate == DW_STORE_BF16) reinterpret_cast<__nv_bfloat16*>(dw)[h] = __float2bfloat16(red[0][c]);
    else dw[h] = accumulate ? dw[h] + red[0][c] : red[0][c];
  }
}

int rmsnorm_bwd(int P, const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, void* dx2,
                void* y, float* dw, float* scratch, long rows, int H, long ldx, long lddy, int dw_accumulate, cudaStream_t s) {
  if (rows == 0) {                                   // nothing to add; a stored sum of no rows is zero
    if (H == 0 || dw_accumulate == 1) return 0;
    P = 0;
  } else {
    // every one of the partial rows is fully written by its CTA before the reduction reads it
    P = bwd_ctas(P, rows, H);
    const int rc = launch_rmsnorm_bwd(P, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,
                                      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, (__nv_bfloat16*)dx2, (__nv_bfloat16*)y,
                                      scratch, rows, H, ldx, lddy);
    if (rc) return rc;
  }
  pbh::launch_dependent(rmsnorm_dw_reduce_kernel, (H + DWR_COLS - 1) / DWR_COLS, DWR_COLS * DWR_ROWS, 0, s, scratch, dw, P, H, H,
      dw_accumulate);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

int pb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* xsum, float* rstd,
                   long rows, int H, long ldx, long ldy, float eps, cudaStream_t s) {
  if (H % 8 || ldx % 8 || ldy % 8 || H > 16384) return -2;
  if (rows == 0) return 0;
  if (fwd_ring(rows, H, res)) {
#define PB_NORM_FWD_RING(VPT, THREADS, CTAS)                                                                     \
  (res ? launch_rmsnorm_fwd_ring<VPT, THREADS, CTAS, true> : launch_rmsnorm_fwd_ring<VPT, THREADS, CTAS, false>) \
  (s, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, (__nv_bfloat16*)y,            \
   (__nv_bfloat16*)xsum, rstd, rows, H, ldx, ldy, eps)
    const int rc = H <= 2048   ? launch_rmsnorm_fwd_ring<4, 64, 8, false>(s, (const __nv_bfloat16*)x, nullptr, (const __nv_bfloat16*)w,
                                                                         (__nv_bfloat16*)y, nullptr, rstd, rows, H, ldx, ldy, eps)
                   : H <= 4096 ? PB_NORM_FWD_RING(4, 128, 4)
                   : H <= 8192 ? PB_NORM_FWD_RING(4, 256, 4) : PB_NORM_FWD_RING(8, 256, 4);
#undef PB_NORM_FWD_RING
    return rc ? rc : (int)cudaGetLastError();
  }
  launch_rmsnorm_fwd(rows, H, s, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
                     (__nv_bfloat16*)y, (__nv_bfloat16*)xsum, rstd, rows, H, ldx, ldy, eps);
  return (int)cudaGetLastError();
}

// Number of CTAs (= rows of the [P, H] fp32 scratch) the backward uses for a given row count.
int pb_rmsnorm_bwd_num_partials(long rows) { return (int)(rows < BWD_MAX_PARTIALS ? (rows < 1 ? 1 : rows) : BWD_MAX_PARTIALS); }

// scratch: fp32 [pb_rmsnorm_bwd_num_partials(rows), H]. dw_accumulate: 1 -> dw += result; 2 -> dw is a bf16 vector, stored.
int pb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                   void* dx, float* dw, float* scratch, long rows, int H, long ldx, long lddy,
                   int dw_accumulate, cudaStream_t s) {
  if (H % 8 || ldx % 8 || lddy % 8 || H > 16384 || rows < 0 || rows > 2147483647L) return -2;
  return rmsnorm_bwd(pb_rmsnorm_bwd_num_partials(rows), dy, x, w, rstd, dres, dx, nullptr, nullptr, dw, scratch, rows, H, ldx, lddy,
                     dw_accumulate, s);
}

// dx is written twice, to dx and to dx2 (with dres only).
int pb_rmsnorm_bwd_two(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, void* dx2,
                       float* dw, float* scratch, long rows, int H, long ldx, long lddy, int dw_accumulate, cudaStream_t s) {
  if (H % 8 || ldx % 8 || lddy % 8 || H > 16384 || rows < 0 || rows > 2147483647L || (rows && !dres)) return -2;
  return rmsnorm_bwd(pb_rmsnorm_bwd_num_partials(rows), dy, x, w, rstd, dres, dx, dx2, nullptr, dw, scratch, rows, H, ldx,
                     lddy, dw_accumulate, s);
}

// The same with y, the normalised rows x * rstd * w that the forward pass gave (pitch ldx; rows of more than 64 channels); dx2 may
// be null.
int pb_rmsnorm_bwd_y(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, void* dx2, void* y,
                     float* dw, float* scratch, long rows, int H, long ldx, long lddy, int dw_accumulate, cudaStream_t s) {
  if (H <= 64 || H % 8 || ldx % 8 || lddy % 8 || H > 16384 || rows < 0 || rows > 2147483647L || (rows && dx2 && !dres)) return -2;
  return rmsnorm_bwd(pb_rmsnorm_bwd_num_partials(rows), dy, x, w, rstd, dres, dx, dx2, y, dw, scratch, rows, H, ldx, lddy,
                     dw_accumulate, s);
}

// y = qkv with RMSNorm over every q head (gain wq) and k head (gain wk); rstd: fp32 [T, hq + hkv].  cos_t (or null): the normalised
// heads are rotated in their first rot_dim channels by the tables' entries [positions, rot_dim / 2] of pos[t] (null: t).
int pb_qk_norm_rope_fwd(const void* x, const void* wq, const void* wk, void* y, float* rstd, long T, int hq, int hkv, int d,
                        long ldx, long ldy, float eps, const int* pos, const float* cos_t, const float* sin_t, int rot_dim,
                        cudaStream_t s) {
  if (d % 8 || d <= 0 || d > 256 || ldx % 8 || ldy % 8) return -2;
  if (cos_t && (rot_dim % 16 || rot_dim <= 0 || rot_dim > d)) return -2;
  const long rows = T * (hq + 2 * hkv);
  if (rows == 0) return 0;
#define PB_QK_FWD(LPR)                                                                                                  \
  {                                                                                                                     \
    auto kern = cos_t ? qk_norm_fwd_kernel<LPR, true> : qk_norm_fwd_kernel<LPR, false>;                                 \
    pbh::launch_dependent(kern, (unsigned)((rows + 128 / LPR * QK_FWD_RUN - 1) / (128 / LPR * QK_FWD_RUN)), 128, 0, s, \
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, (__nv_bfloat16*)y, rstd, rows, hq, \
        hkv, d, ldx, ldy, eps, Rope{pos, cos_t, sin_t, rot_dim});                                                       \
  }
  if (d <= 64) PB_QK_FWD(4)
  else if (d <= 128) PB_QK_FWD(8)
  else PB_QK_FWD(16)
#undef PB_QK_FWD
  return (int)cudaGetLastError();
}

// scratch: fp32 [pb_rmsnorm_bwd_num_partials(T), 2 d]; dwq / dwk: fp32 [d], dw_accumulate: += instead of =.  cos_t (or null), pos,
// sin_t, rot_dim: as the forward was called.
int pb_qk_norm_rope_bwd(const void* dy, const void* x, const void* wq, const void* wk, const float* rstd, void* dx, float* dwq,
                        float* dwk, float* scratch, long T, int hq, int hkv, int d, long ldx, long lddy, long lddx,
                        int dw_accumulate, const int* pos, const float* cos_t, const float* sin_t, int rot_dim, cudaStream_t s) {
  if (d % 8 || d <= 0 || d > 256 || ldx % 8 || lddy % 8 || lddx % 8) return -2;
  if (cos_t && (rot_dim % 16 || rot_dim <= 0 || rot_dim > d)) return -2;
  const long rows = T * (hq + 2 * hkv);
  if (rows == 0) return 0;
  const int P = pb_rmsnorm_bwd_num_partials(T);
  const int ring = QK_STAGES * 4 * 256 * (int)sizeof(Bf8);
#define PB_QK_BWD(LPR)                                                                                              \
  {                                                                                                                 \
    auto kern = cos_t ? qk_norm_bwd_kernel<LPR, true> : qk_norm_bwd_kernel<LPR, false>;                             \
    static std::atomic<bool> allowed[2][pbh::MAX_DEVICES];                                                          \
    const int rc = pbh::allow_shared_memory(kern, ring, allowed[cos_t != nullptr]);                                 \
    if (rc) return rc;                                                                                              \
    pbh::launch_dependent(kern, P, 256, ring, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)wq, \
                           (const __nv_bfloat16*)wk, rstd, (__nv_bfloat16*)dx, scratch, rows, hq, hkv, d, ldx, lddy, \
                           lddx, Rope{pos, cos_t, sin_t, rot_dim});                                                 \
  }
  if (d <= 64) PB_QK_BWD(4)
  else if (d <= 128) PB_QK_BWD(8)
  else PB_QK_BWD(16)
#undef PB_QK_BWD
  const int rc = (int)cudaGetLastError();
  if (rc) return rc;                                 // no gain sums from partial rows that nothing wrote
  const int blocks = (d + DWR_COLS - 1) / DWR_COLS, threads = DWR_COLS * DWR_ROWS;
  pbh::launch_dependent(rmsnorm_dw_reduce_kernel, blocks, threads, 0, s, scratch, dwq, P, d, 2 * d, dw_accumulate != 0);
  pbh::launch_dependent(rmsnorm_dw_reduce_kernel, blocks, threads, 0, s, scratch + d, dwk, P, d, 2 * d, dw_accumulate != 0);
  return (int)cudaGetLastError();
}
int pb_qk_norm_bwd(const void* dy, const void* x, const void* wq, const void* wk, const float* rstd, void* dx, float* dwq,
                   float* dwk, float* scratch, long T, int hq, int hkv, int d, long ldx, long lddy, long lddx,
                   int dw_accumulate, cudaStream_t s) {
  return pb_qk_norm_rope_bwd(dy, x, wq, wk, rstd, dx, dwq, dwk, scratch, T, hq, hkv, d, ldx, lddy, lddx, dw_accumulate, nullptr,
                             nullptr, nullptr, 0, s);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of pb_rmsnorm_bwd (declared in primus_b200_noalloc.h).
//
// For callers that cannot allocate at the call site (a host application that owns every cudaMalloc,
// a pre-planned memory arena, a latency-critical loop): the partial weight gradients go to a fixed
// array in this library's device image rather than to caller-provided scratch.  Host code must not
// pass the array's name to a kernel (on the host that name is only a stand-in for the symbol); its
// device address is looked up once per device with cudaGetSymbolAddress, with that device current.
#include "primus_b200_noalloc.h"

namespace {
static __device__ __align__(256) float g_noalloc_rmsnorm_partials[(long)PB_NOALLOC_MAX_PARTIALS * PB_NOALLOC_MAX_H];
constexpr int kMaxDevices = 64;
float* g_noalloc_scratch_ptr[kMaxDevices] = {nullptr};
}  // namespace

extern "C" int pb_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                      const void* dres, void* dx, float* dw, long rows, int H, long ldx,
                                      long lddy, int dw_accumulate, cudaStream_t s) {
  // more than INT_MAX rows are outside the interface, as they are for pb_rmsnorm_bwd
  if (H <= 0 || H % 8 || ldx % 8 || lddy % 8 || rows < 0 || rows > 2147483647L) return PB_NOALLOC_ERR_BAD_ARG;
  if (H > PB_NOALLOC_MAX_H) return PB_NOALLOC_ERR_TOO_LARGE;  // the built-in scratch holds rows of <= 8192 floats
  if (rows == 0 && dw_accumulate) return 0;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return PB_NOALLOC_ERR_BAD_ARG;
  if (!g_noalloc_scratch_ptr[dev]) {
    // once per device: device address of the scratch array of the image loaded on *this* device
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_rmsnorm_partials);
    if (e != cudaSuccess) return (int)e;
    g_noalloc_scratch_ptr[dev] = p;
  }
  const int P = (int)(rows < PB_NOALLOC_MAX_PARTIALS ? rows : PB_NOALLOC_MAX_PARTIALS);
  return rmsnorm_bwd(P, dy, x, w, rstd, dres, dx, nullptr, nullptr, dw, g_noalloc_scratch_ptr[dev], rows, H, ldx, lddy, dw_accumulate != 0, s);
}
