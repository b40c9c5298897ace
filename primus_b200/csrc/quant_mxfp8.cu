// MXFP8 quantisation: bf16 [R, C] -> E4M3 values with one UE8M0 (power-of-two) scale per 32 elements, in one
// pass for both directions a training GEMM needs:
//   row-wise : blocks of 32 along C (operand reduced over C: forward / data-gradient inputs)
//   col-wise : blocks of 32 along R (operand reduced over R: weight-gradient inputs, transposed use)
// Values keep the [R, C] layout in both cases.  Scales are written directly in the layout tcgen05 block-scaled
// MMAs consume from TMEM: the operand's non-reduced dimension MN and reduced dimension K are tiled in
// 128 x 128-element blocks of 512 bytes, block (mn / 128, k / 128) stored K-fastest, and inside a block
//   offset(mn, kb) = (mn % 32) * 16 + ((mn % 128) / 32) * 4 + kb            (kb = (k % 128) / 32)
// so a block is exactly what one `tcgen05.cp.32x128b.warpx4` moves from shared memory into 4 TMEM columns.
//
// Scale: e = ceil(log2(amax / 448)) (rounded up so that nothing saturates), stored biased by 127;
// value = RN-even E4M3 of x * 2^-e.
//
// Replaces the Turbo / Transformer-Engine MXFP8 cast kernels
// (primus/backends/megatron/core/extensions/primus_turbo.py: `pt.ops.quantize` users, float8 recipe mxfp8).
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include "vec.cuh"

namespace {

constexpr int TILE = 128;

__device__ __forceinline__ int e8m0_from_amax(float amax) {
  const float v = amax * (1.0f / 448.0f);
  const uint32_t b = __float_as_uint(v);
  int e = (int)((b >> 23) & 0xff);        // biased exponent of v
  if (b & 0x7fffff) e += 1;               // ceil for non powers of two
  if (e < 0) e = 0;
  if (e > 254) e = 254;
  return (amax == 0.f) ? 0 : e;           // biased UE8M0
}
__device__ __forceinline__ float inv_scale_from_e8m0(int biased) {
  int f = 254 - biased;                   // exponent field of 2^-(biased - 127)
  if (f < 1) f = 1;
  return __uint_as_float((uint32_t)f << 23);
}
__device__ __forceinline__ uint16_t cvt2(float a, float b) {
  return (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}

// MXFP4 numerics on the FP8 data path: the block exponent leaves the block maximum at or below 6 (the largest E2M1
// magnitude), values are rounded to E2M1 (RN-even, saturating) and stored as the E4M3 byte of the same number (every
// E2M1 value is exact in E4M3), so the block-scaled FP8 GEMM consumes them unchanged.
__device__ __forceinline__ uint16_t cvt2_fp4(float a, float b) {
  const uint32_t packed = (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(a, b), __NV_E2M1, cudaRoundNearest);
  // E2M1 code (sign, 3 magnitude bits: 0, 0.5, 1, 1.5, 2, 3, 4, 6) -> E4M3 byte of the same value
  constexpr unsigned long long lut = 0x4C4844403C383000ull;
  const uint32_t c0 = packed & 0xf, c1 = (packed >> 4) & 0xf;
  const uint32_t b0 = (uint32_t)((lut >> (8 * (c0 & 7))) & 0xff) | ((c0 & 8) << 4);
  const uint32_t b1 = (uint32_t)((lut >> (8 * (c1 & 7))) & 0xff) | ((c1 & 8) << 4);
  return (uint16_t)(b0 | (b1 << 8));
}
template <bool FP4>
__device__ __forceinline__ uint16_t cvt2_sel(float a, float b) {
  return FP4 ? cvt2_fp4(a, b) : cvt2(a, b);
}

__device__ __forceinline__ long sf_offset(int mn, int k_blk32, int k_groups) {
  // block (mn / 128, k_blk32 / 4), K-fastest
  return ((long)(mn >> 7) * k_groups + (k_blk32 >> 2)) * 512 + (mn & 31) * 16 + ((mn & 127) >> 5) * 4 + (k_blk32 & 3);
}

// ------------------------------------------------------------------ register quantiser
// A CTA of four warps quantises a 128 x 128 tile, one warp a strip of 32 rows, one 64-column half after the other.  Lane
// (cg = lane & 7, sub = lane >> 3) holds columns 8 cg .. 8 cg + 7 of rows 4 i + sub (i < 8) as packed bf16, so that a row's
// block maximum needs two shuffles inside four lanes, a column's block maximum two shuffles across the four subs, both on
// packed pairs, and loads, row results and column results are all whole 32-byte sectors.  The elements never pass through
// shared memory and the warps do not wait for one another (an earlier version staged the tile in shared memory and
// alternated load / barrier / two compute phases at 0.56 of copy bandwidth); only the 2 x 512 bytes of scales are gathered
// there, because the operand layout interleaves the bytes of 4 row blocks and 32 rows.
//
// MODE selects where a block of 32 takes its scale exponent from:
//   SCALE_BLOCK32 its own maximum (MXFP8);
//   SCALE_FIXED   `fixed_e` for every block (one power-of-two scale for the tensor, or for this 128 x 128 tile);
//   SCALE_VEC128  `e_rowv[r]` for the blocks of tile row r (row direction) and `e_colv[c]` for those of tile column c
//                 (column direction): one scale per 1 x 128 / 128 x 1 vector, written into its four 32-blocks.
enum { SCALE_BLOCK32 = 0, SCALE_FIXED = 1, SCALE_VEC128 = 2 };
constexpr int QT = 128;                 // threads of a quantising CTA

struct TileScales {
  uint4 row[32], col[32];               // the tile's two 512-byte scale blocks
};

__device__ __forceinline__ __nv_bfloat162 as_bf2(uint32_t w) { return *reinterpret_cast<__nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ uint32_t max_pair(uint32_t a, uint32_t b) { return as_u32(__hmax2(as_bf2(a), as_bf2(b))); }
__device__ __forceinline__ uint32_t abs_pair(uint32_t a) { return a & 0x7fff7fffu; }
// the larger magnitudes of two pairs, with the operands' signs multiplied: a chain of them needs abs_pair at its end only
__device__ __forceinline__ uint32_t max_mag(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// strip of 32 rows of this warp (a CTA of more than four warps has several on every strip, which share its parts)
__device__ __forceinline__ int strip() { return (threadIdx.x >> 5) & 3; }

// Scales of two blocks from the bf16 bits of their maxima (not NaN), both in 16-bit halves: `e` as e8m0_from_amax gives it, and
// `inv`, 2^-(e - 127) as bf16.  In these bits 448 (fp4: 6) is an exponent field 8 (2) above that of 1 and a fraction of 0x60
// (0x40), so that the quotient's exponent, rounded up, is the field less 8 after adding what carries a larger fraction into it.
// With both halves at once a scale costs 4 instructions instead of 12 (8192 x 4096 in both directions 24.7 -> 23.5 us).
struct PairScale {
  uint32_t e, inv;
};
template <bool FP4>
__device__ __forceinline__ PairScale pair_scale(uint32_t m) {
  constexpr uint32_t OFF = FP4 ? 2 : 8, CARRY = FP4 ? 0x3f : 0x1f, TWO = 0x10001u;
  const uint32_t t = __vmaxu2((m + CARRY * TWO) & 0x7f807f80u, ((OFF + 1) << 7) * TWO);   // (a subnormal quotient has e = 1)
  PairScale r;
  r.e = __vminu2((t >> 7) - OFF * TWO, m);       // zero for a block of zeros
  r.inv = ((254 + OFF) << 7) * TWO - t;
  const uint32_t inf = (m + 0x00800080u) & 0x80008000u;
  if (inf) {                                     // an infinite maximum: e = 254, inv = 2^-126
    const uint32_t mask = (inf >> 15) * 0xffffu;
    r.e = (r.e & ~mask) | (0x00fe00feu & mask);
    r.inv = (r.inv & ~mask) | (0x00800080u & mask);
  }
  return r;
}

// eight bf16 values times powers of two -> eight bytes; s[u]: the factors of the u-th pair
template <bool FP4>
__device__ __forceinline__ uint2 scale_cvt8(const uint64_t (&f)[4], uint64_t s0, uint64_t s1, uint64_t s2, uint64_t s3) {
  float a, b;
  uint32_t w[4];
  pb::unpack_f32x2(pb::mul_f32x2(f[0], s0), a, b);
  w[0] = cvt2_sel<FP4>(a, b);
  pb::unpack_f32x2(pb::mul_f32x2(f[1], s1), a, b);
  w[1] = cvt2_sel<FP4>(a, b);
  pb::unpack_f32x2(pb::mul_f32x2(f[2], s2), a, b);
  w[2] = cvt2_sel<FP4>(a, b);
  pb::unpack_f32x2(pb::mul_f32x2(f[3], s3), a, b);
  w[3] = cvt2_sel<FP4>(a, b);
  return make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
}

// Quantises half `h` of this warp's strip -- 64 columns, held in d[8] -- into q_row / q_col (either may be null).  p: offset of
// the lane's first element in the [R, C] tensor.  BOTH: neither is null, and each value is converted to fp32 once for the two,
// at the price of registers (the plain quantiser, five CTAs per SM, spills with it: 27.6 against 23.5 us at 8192 x 4096).
template <int MODE = SCALE_BLOCK32, bool FP4 = false, bool BOTH = false>
__device__ __forceinline__ void quantize_half(const uint4 (&d)[8], int h, long p, int C, uint8_t* __restrict__ q_row,
                                              uint8_t* __restrict__ q_col, TileScales* scales, int warp = strip(),
                                              int fixed_e = 0, const uint8_t* e_rowv = nullptr,
                                              const uint8_t* e_colv = nullptr) {
  const int lane = threadIdx.x & 31;
  const int cg = lane & 7, sub = lane >> 3;
  uint32_t row_inv[4];             // of the lane's rows 2 j, 2 j + 1
  if (BOTH || q_row) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t e;
      if (MODE == SCALE_BLOCK32) {
        uint32_t a[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint4& v = d[2 * j + u];
          a[u] = max_mag(max_mag(v.x, v.y), max_mag(v.z, v.w));
        }
        uint32_t m = max_mag(__byte_perm(a[0], a[1], 0x5410), __byte_perm(a[0], a[1], 0x7632));
        m = max_mag(m, __shfl_xor_sync(0xffffffffu, m, 1));
        // (a block of nothing but NaN counts as zero, as in the column direction: the maximum ignores a NaN operand)
        m = abs_pair(max_mag(0u, max_mag(m, __shfl_xor_sync(0xffffffffu, m, 2))));
        const PairScale ps = pair_scale<FP4>(m);
        e = ps.e;
        row_inv[j] = ps.inv;
      } else {
        const int r = 8 * j + sub;
        const int e0 = MODE == SCALE_FIXED ? fixed_e : (int)e_rowv[warp * 32 + r];
        const int e1 = MODE == SCALE_FIXED ? fixed_e : (int)e_rowv[warp * 32 + r + 4];
        e = (uint32_t)e0 | ((uint32_t)e1 << 16);
        row_inv[j] = (__float_as_uint(inv_scale_from_e8m0(e0)) >> 16) | __float_as_uint(inv_scale_from_e8m0(e1));
      }
      if ((cg & 3) == 0) {
        uint8_t* sf = reinterpret_cast<uint8_t*>(scales->row) + (8 * j + sub) * 16 + warp * 4 + h * 2 + (cg >> 2);
        sf[0] = (uint8_t)e;
        sf[64] = (uint8_t)(e >> 16);
      }
    }
  }
  auto unpack8 = [&](int i, uint64_t (&f)[4]) {
    f[0] = pb::pack_f32x2(lo_f(d[i].x), hi_f(d[i].x));
    f[1] = pb::pack_f32x2(lo_f(d[i].y), hi_f(d[i].y));
    f[2] = pb::pack_f32x2(lo_f(d[i].z), hi_f(d[i].z));
    f[3] = pb::pack_f32x2(lo_f(d[i].w), hi_f(d[i].w));
  };
  if (!BOTH && q_row) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint64_t f[4];
      unpack8(i, f);
      const float inv = (i & 1) ? hi_f(row_inv[i >> 1]) : lo_f(row_inv[i >> 1]);
      const uint64_t s = pb::pack_f32x2(inv, inv);
      *reinterpret_cast<uint2*>(q_row + p + (long)(4 * i) * C) = scale_cvt8<FP4>(f, s, s, s, s);
    }
  }
  if (BOTH || q_col) {
    uint64_t col_inv[4];                // of the column pairs 2 u, 2 u + 1
    uint32_t m[4] = {0, 0, 0, 0}, inv[4];
    const int c0 = h * 64 + cg * 8; // first of the lane's columns in the tile
    if (MODE == SCALE_BLOCK32) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        m[0] = max_mag(m[0], d[i].x);
        m[1] = max_mag(m[1], d[i].y);
        m[2] = max_mag(m[2], d[i].z);
        m[3] = max_mag(m[3], d[i].w);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) m[u] = max_mag(m[u], __shfl_xor_sync(0xffffffffu, m[u], o));
        const PairScale ps = pair_scale<FP4>(abs_pair(m[u]));
        m[u] = ps.e;
        inv[u] = ps.inv;
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e0 = MODE == SCALE_FIXED ? fixed_e : (int)e_colv[c0 + 2 * u];
        const int e1 = MODE == SCALE_FIXED ? fixed_e : (int)e_colv[c0 + 2 * u + 1];
        m[u] = (uint32_t)e0 | ((uint32_t)e1 << 16);
        inv[u] = (__float_as_uint(inv_scale_from_e8m0(e0)) >> 16) | __float_as_uint(inv_scale_from_e8m0(e1));
      }
    }
    // every sub holds the 8 exponents; sub u writes those of its two columns
    const uint32_t e = sub < 2 ? (sub == 0 ? m[0] : m[1]) : (sub == 2 ? m[2] : m[3]);
    const int c = c0 + 2 * sub;
    uint8_t* sf = reinterpret_cast<uint8_t*>(scales->col) + (c & 31) * 16 + (c >> 5) * 4 + warp;
    sf[0] = (uint8_t)e;
    sf[16] = (uint8_t)(e >> 16);
#pragma unroll
    for (int u = 0; u < 4; ++u) col_inv[u] = pb::pack_f32x2(lo_f(inv[u]), hi_f(inv[u]));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint64_t f[4];
      unpack8(i, f);
      if (BOTH) {
        const float inv = (i & 1) ? hi_f(row_inv[i >> 1]) : lo_f(row_inv[i >> 1]);
        const uint64_t s = pb::pack_f32x2(inv, inv);
        *reinterpret_cast<uint2*>(q_row + p + (long)(4 * i) * C) = scale_cvt8<FP4>(f, s, s, s, s);
      }
      *reinterpret_cast<uint2*>(q_col + p + (long)(4 * i) * C) = scale_cvt8<FP4>(f, col_inv[0], col_inv[1], col_inv[2], col_inv[3]);
    }
  }
}

// Writes the gathered scale blocks of the tile at (row0, col0) of an [R, C] tensor (all threads of the CTA).
__device__ __forceinline__ void store_scales(const TileScales* scales, int R, int C, int row0, int col0,
                                             uint8_t* __restrict__ sf_row, uint8_t* __restrict__ sf_col) {
  __syncthreads();
  const int t = threadIdx.x;
  if (t < 32) {
    if (sf_row) reinterpret_cast<uint4*>(sf_row + ((long)(row0 >> 7) * (C >> 7) + (col0 >> 7)) * 512)[t] = scales->row[t];
  } else if (t < 64) {
    if (sf_col) reinterpret_cast<uint4*>(sf_col + ((long)(col0 >> 7) * (R >> 7) + (row0 >> 7)) * 512)[t - 32] = scales->col[t - 32];
  }
}

// element offset of a lane: row `sub` of its warp's strip, first of its 8 columns of part 0
__device__ __forceinline__ long lane_offset(int row0, int col0, long ld, int strip_ = strip()) {
  const int lane = threadIdx.x & 31;
  return (long)(row0 + strip_ * 32 + (lane >> 3)) * ld + col0 + (lane & 7) * 8;
}

__device__ __forceinline__ void load_tile(const __nv_bfloat16* __restrict__ x, long p, int C, uint4 (&d)[2][8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 8; ++i) d[h][i] = *reinterpret_cast<const uint4*>(x + p + h * 64 + (long)(4 * i) * C);
}

template <bool FP4>
__global__ void __launch_bounds__(QT, 5)
quant_mxfp8_kernel(const __nv_bfloat16* __restrict__ x, int R, int C, uint8_t* __restrict__ q_row,
                   uint8_t* __restrict__ sf_row, uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col) {
  pb::grid_release();
  PB_GRID_WAIT();
  __shared__ TileScales scales;
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE;
  const long p = lane_offset(row0, col0, C);
  uint4 d[2][8];
  load_tile(x, p, C, d);
#pragma unroll
  for (int h = 0; h < 2; ++h) quantize_half<SCALE_BLOCK32, FP4>(d[h], h, p + h * 64, C, q_row, q_col, &scales);
  store_scales(&scales, R, C, row0, col0, sf_row, sf_col);
}

// Tensor-wise FP8 ("current scaling" with a power-of-two scale): one scale 2^e for the whole tensor,
// e = ceil(log2(amax / 448)) from the tensor maximum `tensor_amax` (device, written by amax_bf16_kernel).  The output has
// the MXFP8 layout with that exponent in every block, so the block-scaled GEMM consumes it unchanged.  The behaviour
// of the reference's tensor-wise quantiser (primus_turbo_cpp_extension::quantize_fp8_tensorwise, called from
// primus/backends/megatron/core/extensions/primus_turbo_float8_local.py:66-70).
__global__ void __launch_bounds__(QT, 5)
quant_tensorwise_kernel(const __nv_bfloat16* __restrict__ x, int R, int C, const float* __restrict__ tensor_amax,
                        const float* __restrict__ fallback_amax, uint8_t* __restrict__ q_row,
                        uint8_t* __restrict__ sf_row, uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col) {
  PB_GRID_WAIT();
  __shared__ TileScales scales;
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE;
  const long p = lane_offset(row0, col0, C);
  uint4 d[2][8];
  load_tile(x, p, C, d);
  // delayed scaling passes the maximum its history predicts as `tensor_amax` and this step's measured maximum as
  // `fallback_amax`, which is used while the history is still empty (0)
  float a = *tensor_amax;
  if (a == 0.f && fallback_amax != nullptr) a = *fallback_amax;
  const int fixed_e = e8m0_from_amax(a);
#pragma unroll
  for (int h = 0; h < 2; ++h) quantize_half<SCALE_FIXED>(d[h], h, p + h * 64, C, q_row, q_col, &scales, strip(), fixed_e);
  store_scales(&scales, R, C, row0, col0, sf_row, sf_col);
}

// Block-wise FP8 (blocks of 128): activations and gradients take one power-of-two scale per 1 x 128 vector along the
// reduced dimension (row direction: 128 consecutive columns of a row; column direction: 128 consecutive rows of a
// column), weights (TILEWISE) one per 128 x 128 tile.  Stored in the MXFP8 layout with the exponent repeated in the
// four 32-blocks it covers, so the block-scaled GEMM consumes it unchanged.  Granularity of the reference's
// "blockwise" recipe (primus/backends/megatron/core/extensions/primus_turbo.py: Float8QuantConfig with
// ScalingGranularity.BLOCKWISE, block_size 128), with scales restricted to powers of two.
template <bool TILEWISE>
__global__ void __launch_bounds__(QT, 4)
quant_blockwise_kernel(const __nv_bfloat16* __restrict__ x, int R, int C, uint8_t* __restrict__ q_row,
                       uint8_t* __restrict__ sf_row, uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col) {
  PB_GRID_WAIT();
  __shared__ TileScales scales;
  __shared__ uint8_t e_rowv[TILE], e_colv[TILE];
  __shared__ uint32_t col_max[4][TILE / 2];      // per warp strip: maxima of column pairs
  __shared__ uint32_t strip_max[4];
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cg = lane & 7, sub = lane >> 3;
  const long p = lane_offset(row0, col0, C);
  uint4 d[2][8];
  load_tile(x, p, C, d);
  uint32_t rm[4];                                // rows (8 j + sub, 8 j + 4 + sub): maximum over the tile's 128 columns
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t a[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      a[u] = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4& v = d[h][2 * j + u];
        a[u] = max_pair(a[u], max_pair(max_pair(abs_pair(v.x), abs_pair(v.y)), max_pair(abs_pair(v.z), abs_pair(v.w))));
      }
    }
    rm[j] = max_pair(__byte_perm(a[0], a[1], 0x5410), __byte_perm(a[0], a[1], 0x7632));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) rm[j] = max_pair(rm[j], __shfl_xor_sync(0xffffffffu, rm[j], o));
  }
  if (TILEWISE) {
    uint32_t m = max_pair(max_pair(rm[0], rm[1]), max_pair(rm[2], rm[3]));
    m = max_pair(m, __shfl_xor_sync(0xffffffffu, m, 8));
    m = max_pair(m, __shfl_xor_sync(0xffffffffu, m, 16));
    if (lane == 0) strip_max[warp] = m;
    __syncthreads();
    m = max_pair(max_pair(strip_max[0], strip_max[1]), max_pair(strip_max[2], strip_max[3]));
    const int fixed_e = e8m0_from_amax(fmaxf(lo_f(m), hi_f(m)));
#pragma unroll
    for (int h = 0; h < 2; ++h) quantize_half<SCALE_FIXED>(d[h], h, p + h * 64, C, q_row, q_col, &scales, strip(), fixed_e);
  } else {
    if (cg == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        e_rowv[warp * 32 + 8 * j + sub] = (uint8_t)e8m0_from_amax(lo_f(rm[j]));
        e_rowv[warp * 32 + 8 * j + 4 + sub] = (uint8_t)e8m0_from_amax(hi_f(rm[j]));
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t m[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        m[0] = max_pair(m[0], abs_pair(d[h][i].x));
        m[1] = max_pair(m[1], abs_pair(d[h][i].y));
        m[2] = max_pair(m[2], abs_pair(d[h][i].z));
        m[3] = max_pair(m[3], abs_pair(d[h][i].w));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        m[u] = max_pair(m[u], __shfl_xor_sync(0xffffffffu, m[u], 8));
        m[u] = max_pair(m[u], __shfl_xor_sync(0xffffffffu, m[u], 16));
        if (sub == u) col_max[warp][h * 32 + cg * 4 + u] = m[u];
      }
    }
    __syncthreads();
    if (threadIdx.x < TILE / 2) {
      const int t = threadIdx.x;
      const uint32_t m = max_pair(max_pair(col_max[0][t], col_max[1][t]), max_pair(col_max[2][t], col_max[3][t]));
      e_colv[2 * t] = (uint8_t)e8m0_from_amax(lo_f(m));
      e_colv[2 * t + 1] = (uint8_t)e8m0_from_amax(hi_f(m));
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      quantize_half<SCALE_VEC128>(d[h], h, p + h * 64, C, q_row, q_col, &scales, strip(), 0, e_rowv, e_colv);
  }
  store_scales(&scales, R, C, row0, col0, sf_row, sf_col);
}

// max |x| over n bf16 values (n a multiple of 8) into *out, which the caller zeroes first (non-negative floats order
// like their bit patterns, so the cross-CTA step is an integer atomicMax)
__global__ void __launch_bounds__(256)
amax_bf16_kernel(const __nv_bfloat16* __restrict__ x, long n8, float* __restrict__ out) {
  __nv_bfloat162 m = __floats2bfloat162_rn(0.f, 0.f);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
    const uint4 d = reinterpret_cast<const uint4*>(x)[i];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&d);
#pragma unroll
    for (int u = 0; u < 4; ++u) m = __hmax2(m, __habs2(h[u]));
  }
  const float2 f = __bfloat1622float2(m);
  float v = fmaxf(f.x, f.y);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __shared__ float s[8];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) v = fmaxf(v, s[i]);
    if (v != v) v = __uint_as_float(0x7f800000u);   // NaN in the input: report +inf
    atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(v));
  }
}

__device__ __forceinline__ void bf8_unpack(const uint4& d, float* f) {
  f[0] = lo_f(d.x); f[1] = hi_f(d.x); f[2] = lo_f(d.y); f[3] = hi_f(d.y);
  f[4] = lo_f(d.z); f[5] = hi_f(d.z); f[6] = lo_f(d.w); f[7] = hi_f(d.w);
}
__device__ __forceinline__ uint4 bf8_pack(const float* f) {
  uint4 o;
  o.x = pb::pack_bf16x2(f[0], f[1]);
  o.y = pb::pack_bf16x2(f[2], f[3]);
  o.z = pb::pack_bf16x2(f[4], f[5]);
  o.w = pb::pack_bf16x2(f[6], f[7]);
  return o;
}

// SwiGLU forward fused with the quantisation of its output: h1 [T, 2I] = [gate | up] -> MXFP8 of
// act[T, I] = silu(gate) * up (rounded to bf16 first, so the values equal quantising the un-fused kernel's output).
// Four rows' loads in flight per lane and round keep it at 80 registers: six CTAs (24 warps) per SM hide the two special-
// function operations per element (8192 x 14336, row direction: 97 us, 6.1 TB/s; 106 with scales computed one by one and 127 with
// the tile staged in shared memory; two fp32 operations per instruction, as in the backward, need more registers here: 115).
// WIDE: as many warps per strip as it has parts, for tensors of at most a tile per SM, where a warp's parts one after the other
// are the time (1024 x 1408: 5.4 -> 4.9 us); with several CTAs per SM the parts' registers are better spent on more CTAs.
template <bool WIDE, bool CLAMP>
__global__ void __launch_bounds__(WIDE ? 2 * QT : QT, WIDE ? 2 : 6)
swiglu_quant_mxfp8_kernel(const __nv_bfloat16* __restrict__ h1, int T, int I, float clamp, uint8_t* __restrict__ q_row,
                          uint8_t* __restrict__ sf_row, uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col) {
  PB_GRID_WAIT();
  __shared__ TileScales scales;
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE;
  const long pin = lane_offset(row0, col0, 2L * I), p = lane_offset(row0, col0, I);
#pragma unroll 1
  for (int h = WIDE ? threadIdx.x / QT : 0; h < 2; h += WIDE ? 2 : 1) {
    uint4 d[8];
#pragma unroll
    for (int i0 = 0; i0 < 8; i0 += 4) {
      uint4 up[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat16* g = h1 + pin + h * 64 + (long)(4 * (i0 + i)) * 2 * I;
        d[i0 + i] = *reinterpret_cast<const uint4*>(g);
        up[i] = *reinterpret_cast<const uint4*>(g + I);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float fg[8], fu[8], o[8];
        bf8_unpack(d[i0 + i], fg);
        bf8_unpack(up[i], fu);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float gg = fg[j], uu = fu[j];
          if (CLAMP) {
            gg = fminf(gg, clamp);
            uu = fminf(fmaxf(uu, -clamp), clamp);
          }
          o[j] = gg * pb::fast_sigmoid(gg) * uu;
        }
        d[i0 + i] = bf8_pack(o);
      }
    }
    quantize_half(d, h, p + h * 64, I, q_row, q_col, &scales);
  }
  store_scales(&scales, T, I, row0, col0, sf_row, sf_col);
}

constexpr int BWD_WARP_BYTES = 3 * 8 * 32 * 16;   // shared memory of a warp of the SwiGLU backward

// Two elements of the SwiGLU backward: dgate, dup and the activation from gate, up and dact (bf16 pairs), in the order and with the
// roundings of swiglu_bwd_kernel and swiglu_fwd_kernel (two fp32 operations an instruction).
template <bool CLAMP>
__device__ __forceinline__ void swiglu_bwd_pair(uint32_t gate, uint32_t up, uint32_t dact, float clamp, uint32_t& dgate, uint32_t& dup,
                                                uint32_t& act) {
  float g0 = lo_f(gate), g1 = hi_f(gate), u0 = lo_f(up), u1 = hi_f(up);
  uint64_t gmask = 0, umask = 0;
  if (CLAMP) {
    gmask = pb::pack_f32x2(g0 > clamp ? 0.f : 1.f, g1 > clamp ? 0.f : 1.f);
    umask = pb::pack_f32x2(u0 > clamp || u0 < -clamp ? 0.f : 1.f, u1 > clamp || u1 < -clamp ? 0.f : 1.f);
    if (g0 > clamp) g0 = clamp;
    if (g1 > clamp) g1 = clamp;
    if (u0 > clamp) u0 = clamp;
    if (u0 < -clamp) u0 = -clamp;
    if (u1 > clamp) u1 = clamp;
    if (u1 < -clamp) u1 = -clamp;
  }
  const uint64_t g = pb::pack_f32x2(g0, g1), u = pb::pack_f32x2(u0, u1), d = pb::pack_f32x2(lo_f(dact), hi_f(dact));
  const uint64_t one = pb::pack_f32x2(1.f, 1.f), minus = pb::pack_f32x2(-1.f, -1.f);
  const uint64_t sig = pb::fast_sigmoid2(g);
  const uint64_t sl = pb::mul_f32x2(g, sig);
  const uint64_t dsl = pb::mul_f32x2(sig, pb::fma_f32x2(g, pb::fma_f32x2(sig, minus, one), one));
  uint64_t og = pb::mul_f32x2(pb::mul_f32x2(d, u), dsl), ou = pb::mul_f32x2(d, sl);
  if (CLAMP) {
    og = pb::mul_f32x2(og, gmask);
    ou = pb::mul_f32x2(ou, umask);
  }
  float a, b;
  pb::unpack_f32x2(og, a, b);
  dgate = pb::pack_bf16x2(a, b);
  pb::unpack_f32x2(ou, a, b);
  dup = pb::pack_bf16x2(a, b);
  pb::unpack_f32x2(pb::mul_f32x2(sl, u), a, b);
  act = pb::pack_bf16x2(a, b);
}

// SwiGLU backward fused with the quantisation of its output: (h1 [T, 2I], dact [T, I]) -> MXFP8 (both directions) of
// dh1 [T, 2I] = [dgate | dup], and (optional) of the activation itself along T, the operand of the weight gradient, which
// another pass over h1 would otherwise recompute.  One CTA per 128 x 128 tile of the activation; a warp takes 32 rows of a
// 64-column half, with its neighbour the other half of the same rows, so that whole 128-byte lines of the results are written
// at about the same time (quarters one after the other left half-written lines for DRAM: with more CTAs in flight twice the time).
// gate, up and dact go to the lane's own slots of shared memory and the three results take their places there: a
// lane holds one result at a time in registers, and 16 warps share an SM.  8192 x 14336: 238 us, and another 107 for the
// activation, before; 194 and, with the activation, 221 now (5.8 TB/s).  What is left beside the memory is the issue of about
// 35 instructions an element.  WIDE: as above, eight warps, one round.
template <bool WIDE, bool CLAMP>
__global__ void __launch_bounds__(WIDE ? 2 * QT : QT, WIDE ? 2 : 4)
swiglu_bwd_quant_mxfp8_kernel(const __nv_bfloat16* __restrict__ h1, const __nv_bfloat16* __restrict__ dact, int T, int I,
                              float clamp, uint8_t* __restrict__ q_row, uint8_t* __restrict__ sf_row,
                              uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col, uint8_t* __restrict__ act_col,
                              uint8_t* __restrict__ act_sf) {
  PB_GRID_WAIT();
  extern __shared__ __align__(16) uint4 slots_raw[];   // [warp][gate, up, dact][row of the lane][lane]
  __shared__ TileScales scales[3];               // of the dgate, the dup and the activation tile
  constexpr int WARPS = WIDE ? 8 : 4, STRIPS = WARPS / 2;
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE, warp = threadIdx.x >> 5, h = warp & 1;
  uint4 *sg = slots_raw + warp * (BWD_WARP_BYTES / 16) + (threadIdx.x & 31), *su = sg + 256, *sd = su + 256;
#pragma unroll 1
  for (int st = warp >> 1; st < 4; st += STRIPS) {
    const long o2 = lane_offset(row0, col0, 2L * I, st) + h * 64, o1 = lane_offset(row0, col0, I, st) + h * 64;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat16* g = h1 + o2 + (long)(4 * i) * 2 * I;
      pb::cp_async_16(sg + i * 32, g);
      pb::cp_async_16(su + i * 32, g + I);
      pb::cp_async_16(sd + i * 32, dact + o1 + (long)(4 * i) * I);
    }
    pb::cp_async_commit();
    pb::cp_async_wait<0>();
#pragma unroll 2
    for (int i = 0; i < 8; ++i) {
      const uint4 vg = sg[i * 32], vu = su[i * 32], vd = sd[i * 32];
      uint32_t og[4], ou[4], oa[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        swiglu_bwd_pair<CLAMP>(reinterpret_cast<const uint32_t*>(&vg)[j], reinterpret_cast<const uint32_t*>(&vu)[j],
                               reinterpret_cast<const uint32_t*>(&vd)[j], clamp, og[j], ou[j], oa[j]);
      sg[i * 32] = make_uint4(og[0], og[1], og[2], og[3]);
      su[i * 32] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
      sd[i * 32] = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    }
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = sg[i * 32];
    quantize_half<SCALE_BLOCK32, false, true>(v, h, o2, 2 * I, q_row, q_col, &scales[0], st);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = su[i * 32];
    quantize_half<SCALE_BLOCK32, false, true>(v, h, o2 + I, 2 * I, q_row, q_col, &scales[1], st);
    if (act_col) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = sd[i * 32];
      quantize_half(v, h, o1, I, nullptr, act_col, &scales[2], st);
    }
  }
  store_scales(&scales[0], T, 2 * I, row0, col0, sf_row, sf_col);
  store_scales(&scales[1], T, 2 * I, row0, I + col0, sf_row, sf_col);
  store_scales(&scales[2], T, I, row0, col0, nullptr, act_sf);
}

// value [R, C] fp8 + scales (operand layout with MN = R or C) -> fp32 [R, C]; test / debugging helper
__global__ void dequant_mxfp8_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ sf, int R, int C,
                                     int colwise, float* __restrict__ out) {
  const long n = (long)R * C;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i / C), c = (int)(i - (long)r * C);
    const int e = colwise ? sf[sf_offset(c, r >> 5, R >> 7)] : sf[sf_offset(r, c >> 5, C >> 7)];
    const __nv_fp8_e4m3 v = *reinterpret_cast<const __nv_fp8_e4m3*>(q + i);
    out[i] = float(v) * exp2f((float)(e - 127));
  }
}

}  // namespace

extern "C" {

// Any of the two outputs may be null.  R and C must be multiples of 128.
// sf_row: R * C / 32 bytes, sf_col: R * C / 32 bytes.
int pb_quant_mxfp8(const void* x, int R, int C, void* q_row, void* sf_row, void* q_col, void* sf_col, cudaStream_t s) {
  if (R % TILE || C % TILE || R <= 0 || C <= 0) return -2;
  dim3 grid(C / TILE, R / TILE);
  pbh::launch_dependent(quant_mxfp8_kernel<false>, grid, QT, 0, s, reinterpret_cast<const __nv_bfloat16*>(x), R, C,
      reinterpret_cast<uint8_t*>(q_row), reinterpret_cast<uint8_t*>(sf_row), reinterpret_cast<uint8_t*>(q_col),
      reinterpret_cast<uint8_t*>(sf_col));
  return (int)cudaGetLastError();
}

// MXFP4 numerics in FP8 storage: E2M1 values (as E4M3 bytes) with one UE8M0 scale per 32 elements; outputs and
// constraints as pb_quant_mxfp8.
int pb_quant_mxfp4_as_fp8(const void* x, int R, int C, void* q_row, void* sf_row, void* q_col, void* sf_col,
                          cudaStream_t s) {
  if (R % TILE || C % TILE || R <= 0 || C <= 0) return -2;
  pbh::launch_dependent(quant_mxfp8_kernel<true>, dim3(C / TILE, R / TILE), QT, 0, s, reinterpret_cast<const __nv_bfloat16*>(x), R,
      C, reinterpret_cast<uint8_t*>(q_row), reinterpret_cast<uint8_t*>(sf_row), reinterpret_cast<uint8_t*>(q_col),
      reinterpret_cast<uint8_t*>(sf_col));
  return (int)cudaGetLastError();
}

// Tensor-wise FP8 of x [R, C] (multiples of 128): amax[0] receives max |x|; outputs as pb_quant_mxfp8.
int pb_quant_fp8_tensorwise(const void* x, int R, int C, float* amax, void* q_row, void* sf_row, void* q_col, void* sf_col,
                            cudaStream_t s) {
  if (R % TILE || C % TILE || R <= 0 || C <= 0) return -2;
  cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(float), s);
  if (e != cudaSuccess) return (int)e;
  const long n8 = (long)R * C / 8;
  const int blocks = (int)((n8 + 2047) / 2048 < 1184 ? (n8 + 2047) / 2048 : 1184);
  amax_bf16_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), n8, amax);
  pbh::launch_dependent(quant_tensorwise_kernel, dim3(C / TILE, R / TILE), QT, 0, s, reinterpret_cast<const __nv_bfloat16*>(x), R,
      C, amax, nullptr, reinterpret_cast<uint8_t*>(q_row), reinterpret_cast<uint8_t*>(sf_row), reinterpret_cast<uint8_t*>(q_col),
      reinterpret_cast<uint8_t*>(sf_col));
  return (int)cudaGetLastError();
}

// Delayed-scaling FP8 of x [R, C]: the scale comes from scale_amax[0] (the maximum predicted from the history of
// earlier steps; 0 = no history yet, then this call's own maximum is used), and max |x| is folded into amax_now[0]
// with an atomic maximum -- the caller zeroes amax_now when it rolls the history, so several calls between two rolls
// (micro-batches) record their overall maximum.  Values above the predicted range saturate at +-448.
int pb_quant_fp8_delayed(const void* x, int R, int C, float* amax_now, const float* scale_amax, void* q_row,
                         void* sf_row, void* q_col, void* sf_col, cudaStream_t s) {
  if (R % TILE || C % TILE || R <= 0 || C <= 0) return -2;
  const long n8 = (long)R * C / 8;
  const int blocks = (int)((n8 + 2047) / 2048 < 1184 ? (n8 + 2047) / 2048 : 1184);
  amax_bf16_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), n8, amax_now);
  pbh::launch_dependent(quant_tensorwise_kernel, dim3(C / TILE, R / TILE), QT, 0, s, reinterpret_cast<const __nv_bfloat16*>(x), R,
      C, scale_amax, amax_now, reinterpret_cast<uint8_t*>(q_row), reinterpret_cast<uint8_t*>(sf_row),
      reinterpret_cast<uint8_t*>(q_col), reinterpret_cast<uint8_t*>(sf_col));
  return (int)cudaGetLastError();
}

// Block-wise FP8 of x [R, C] (multiples of 128): one power-of-two scale per 1 x 128 vector (tilewise = 0:
// activations, gradients) or per 128 x 128 tile (tilewise = 1: weights); outputs as pb_quant_mxfp8.
int pb_quant_fp8_blockwise(const void* x, int R, int C, int tilewise, void* q_row, void* sf_row, void* q_col,
                           void* sf_col, cudaStream_t s) {
  if (R % TILE || C % TILE || R <= 0 || C <= 0) return -2;
  const dim3 grid(C / TILE, R / TILE);
  const __nv_bfloat16* xp = reinterpret_cast<const __nv_bfloat16*>(x);
  uint8_t *qr = reinterpret_cast<uint8_t*>(q_row), *sr = reinterpret_cast<uint8_t*>(sf_row);
  uint8_t *qc = reinterpret_cast<uint8_t*>(q_col), *sc = reinterpret_cast<uint8_t*>(sf_col);
  if (tilewise) pbh::launch_dependent(quant_blockwise_kernel<true>, grid, QT, 0, s, xp, R, C, qr, sr, qc, sc);
  else pbh::launch_dependent(quant_blockwise_kernel<false>, grid, QT, 0, s, xp, R, C, qr, sr, qc, sc);
  return (int)cudaGetLastError();
}

// act = silu(gate) * up of h1 [T, 2I] (T, I multiples of 128) quantised to MXFP8; either output pair may be null.
int pb_swiglu_quant_mxfp8(const void* h1, int T, int I, float clamp, void* q_row, void* sf_row, void* q_col,
                          void* sf_col, cudaStream_t s) {
  if (T % TILE || I % TILE || T <= 0 || I <= 0) return -2;
  const dim3 grid(I / TILE, T / TILE);
  const bool wide = (long)grid.x * grid.y <= 148;
  auto kern = clamp > 0.f ? (wide ? swiglu_quant_mxfp8_kernel<true, true> : swiglu_quant_mxfp8_kernel<false, true>)
                          : (wide ? swiglu_quant_mxfp8_kernel<true, false> : swiglu_quant_mxfp8_kernel<false, false>);
  pbh::launch_dependent(kern, grid, wide ? 2 * QT : QT, 0, s, reinterpret_cast<const __nv_bfloat16*>(h1), T, I, clamp,
      reinterpret_cast<uint8_t*>(q_row), reinterpret_cast<uint8_t*>(sf_row), reinterpret_cast<uint8_t*>(q_col),
      reinterpret_cast<uint8_t*>(sf_col));
  return (int)cudaGetLastError();
}

// dh1 [T, 2I] = swiglu backward of (h1, dact) quantised to MXFP8 (outputs sized for [T, 2I]).  act_col / act_sf (null or both):
// also the activation itself [T, I], quantised along T, as pb_swiglu_quant_mxfp8 gives it.
int pb_swiglu_bwd_quant_mxfp8(const void* h1, const void* dact, int T, int I, float clamp, void* q_row, void* sf_row,
                              void* q_col, void* sf_col, void* act_col, void* act_sf, cudaStream_t s) {
  if (T % TILE || I % TILE || T <= 0 || I <= 0 || !act_col != !act_sf) return -2;
  const dim3 grid(I / TILE, T / TILE);
  const bool wide = (long)grid.x * grid.y <= 148;
  auto kern = clamp > 0.f ? (wide ? swiglu_bwd_quant_mxfp8_kernel<true, true> : swiglu_bwd_quant_mxfp8_kernel<false, true>)
                          : (wide ? swiglu_bwd_quant_mxfp8_kernel<true, false> : swiglu_bwd_quant_mxfp8_kernel<false, false>);
  const int smem = (wide ? 8 : 4) * BWD_WARP_BYTES;
  static std::atomic<bool> allowed[4][pbh::MAX_DEVICES];
  const int rc = pbh::allow_shared_memory(kern, smem, allowed[wide + 2 * (clamp > 0.f)]);
  if (rc) return rc;
  pbh::launch_dependent(kern, grid, wide ? 2 * QT : QT, smem, s, reinterpret_cast<const __nv_bfloat16*>(h1),
      reinterpret_cast<const __nv_bfloat16*>(dact), T, I, clamp, reinterpret_cast<uint8_t*>(q_row),
      reinterpret_cast<uint8_t*>(sf_row), reinterpret_cast<uint8_t*>(q_col), reinterpret_cast<uint8_t*>(sf_col),
      reinterpret_cast<uint8_t*>(act_col), reinterpret_cast<uint8_t*>(act_sf));
  return (int)cudaGetLastError();
}

int pb_dequant_mxfp8(const void* q, const void* sf, int R, int C, int colwise, float* out, cudaStream_t s) {
  if (R % TILE || C % TILE) return -2;
  dequant_mxfp8_kernel<<<1184, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(q), reinterpret_cast<const uint8_t*>(sf), R,
                                           C, colwise, out);
  return (int)cudaGetLastError();
}

}  // extern "C"
