// Permutation maps of the padded expert-major layout (device-side, no host synchronisation).
//
// Copy i (arrival order) of expert e goes to row row_start[e] + (number of earlier copies of e); rows between an expert's
// count and its padded count, and rows past the last expert, are padding.  One CTA per expert walks the expert ids of all
// copies (they come from L2 after the first CTA) and hands out consecutive rows with a block-wide scan, so the result is
// the stable counting sort and does not depend on scheduling.  A sort-based map costs a dozen launches for the same
// tables; with the ids of 32768 copies the walk is 8 steps.
#include "common.cuh"

namespace {

constexpr int MAP_THREADS = 1024;
constexpr int MAP_ITEMS = 4;      // consecutive copies per thread and step

__global__ void __launch_bounds__(MAP_THREADS)
moe_permutation_maps_kernel(const long* __restrict__ expert, int R, int topk, int E, const int* __restrict__ row_start,
                            const int* __restrict__ padded, int rows_cap, int* __restrict__ src,
                            int* __restrict__ src_token, int* __restrict__ pos) {
  __shared__ int warp_sums[2][MAP_THREADS / 32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int start = row_start[e];
  int next = start;                 // first free row of the expert
  auto load = [&](int base, long* v) {
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) v[j] = base + j < R ? expert[base + j] : -1;
  };
  long cur[MAP_ITEMS];
  load(threadIdx.x * MAP_ITEMS, cur);
  int flip = 0;
  for (int base0 = 0; base0 < R; base0 += MAP_THREADS * MAP_ITEMS, flip ^= 1) {
    const int base = base0 + threadIdx.x * MAP_ITEMS;
    long nxt[MAP_ITEMS];
    load(base + MAP_THREADS * MAP_ITEMS, nxt);      // in flight during the scan
    int mine = 0;
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) mine += cur[j] == e;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[flip][warp] = incl;
    __syncthreads();                // the other buffer's readers are past the previous barrier
    const int ws = warp_sums[flip][lane];
    int before = lane < warp ? ws : 0, total = ws;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      total += __shfl_xor_sync(0xffffffffu, total, o);
    }
    int row = next + before + incl - mine;
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) {
      if (cur[j] == e) {
        if (row < rows_cap) {
          src[row] = base + j;
          if (src_token) src_token[row] = (base + j) / topk;
        }
        pos[base + j] = row++;
      }
      cur[j] = nxt[j];
    }
    next += total;
  }
  // padding: this expert's own, and (last expert) the rows past the layout
  const int end = e == E - 1 ? rows_cap : min(start + padded[e], rows_cap);
  for (int r = next + threadIdx.x; r < end; r += MAP_THREADS) {
    src[r] = -1;
    if (src_token) src_token[r] = -1;
  }
}

// out[i] = idx[i] >= 0 ? x[idx[i]] : 0
__global__ void gather_f32_kernel(const float* __restrict__ x, const int* __restrict__ idx, float* __restrict__ out, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int j = idx[i];
    out[i] = j >= 0 ? x[j] : 0.f;
  }
}

}  // namespace

extern "C" {

// expert: int64 [R] expert of every copy (arrival order, `topk` copies per token); src / src_token: int32 [rows_cap] copy /
// token feeding each row (-1: padding; src_token may be null); pos: int32 [R] row of every copy.
int pb_moe_permutation_maps(const long* expert, long R, int topk, int E, const int* row_start, const int* padded,
                            int rows_cap, int* src, int* src_token, int* pos, cudaStream_t s) {
  if (E <= 0 || topk <= 0 || R < 0 || R > 2147483647L - 2 * MAP_THREADS * MAP_ITEMS) return -2;
  moe_permutation_maps_kernel<<<E, MAP_THREADS, 0, s>>>(expert, (int)R, topk, E, row_start, padded, rows_cap, src, src_token,
                                                       pos);
  return (int)cudaGetLastError();
}

int pb_gather_f32(const float* x, const int* idx, float* out, long n, cudaStream_t s) {
  if (n == 0) return 0;
  const long blocks = (n + 255) / 256;
  gather_f32_kernel<<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, s>>>(x, idx, out, n);
  return (int)cudaGetLastError();
}

}  // extern "C"
