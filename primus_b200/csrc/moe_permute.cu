// Permutation maps of the padded expert-major layout (device-side, no host synchronisation).
//
// Copy i (arrival order) of expert e goes to row row_start[e] + (number of earlier copies of e); rows between an expert's
// count and its padded count, and rows past the last expert, are padding.  One CTA per expert walks the expert ids of all
// copies (they come from L2 after the first CTA) and hands out consecutive rows, so the result is the stable counting sort and
// does not depend on scheduling.  A sort-based map costs a dozen launches for the same tables; with the ids of 32768 copies the
// walk is 2 steps, in which a warp ranks 16 times 32 neighbouring ids by ballots (64 experts 9 us; four ids a lane in 8 steps
// of shuffled sums 16, sixteen, whose loads are 128 bytes apart, 28).
// LocalPlan: the CTA also derives what the layout follows from (its first row from the counts of the experts before it) and gathers
// the routing probabilities of its rows; for one rank's own tokens that is the whole plan in one launch.
#include "common.cuh"

namespace {

constexpr int MAP_THREADS = 1024;
constexpr int MAP_ITEMS = 16;     // 32 neighbouring copies each: a warp's share of a step

struct LocalPlan {
  const int* counts;
  const float* probs;                   // of the copies
  int *padded, *row_start, *mblock_expert, *total;
  float* probs_perm;                    // of the rows: 0 for padding
  int max_mblocks;
};

template <bool LOCAL>
__global__ void __launch_bounds__(MAP_THREADS)
moe_permutation_maps_kernel(const long* __restrict__ expert, int R, int topk, int E, const int* __restrict__ row_start,
                            const int* __restrict__ padded, int rows_cap, int* src,
                            int* __restrict__ src_token, int* __restrict__ pos, LocalPlan plan) {
  PB_GRID_WAIT();
  __shared__ int warp_sums[2][MAP_THREADS / 32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int start, pad;
  if (LOCAL) {
    auto padded_of = [&](int i) { return (plan.counts[i] + 127) / 128 * 128; };
    int before = 0;
    for (int i = threadIdx.x; i < e; i += MAP_THREADS) before += padded_of(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) warp_sums[0][warp] = before;
    __syncthreads();
    start = warp_sums[0][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) start += __shfl_xor_sync(0xffffffffu, start, o);
    __syncthreads();
    pad = padded_of(e);
    if (threadIdx.x == 0) {
      plan.padded[e] = pad;
      plan.row_start[e] = start;
      if (e == E - 1) plan.total[0] = start + pad;
    }
    const int m0 = start / 128, m1 = m0 + pad / 128, end = e == E - 1 ? plan.max_mblocks : min(m1, plan.max_mblocks);
    for (int m = m0 + threadIdx.x; m < end; m += MAP_THREADS) plan.mblock_expert[m] = m < m1 ? e : -1;
  } else {
    start = row_start[e];
    pad = padded[e];
  }
  int next = start;                 // first free row of the expert
  auto load = [&](long base0, int* v) {
    const long base = base0 + warp * (32 * MAP_ITEMS) + lane;
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) v[j] = base + 32 * j < R ? (int)expert[base + 32 * j] : -1;
  };
  int cur[MAP_ITEMS];
  load(0, cur);
  int flip = 0;
  for (long base0 = 0; base0 < R; base0 += MAP_THREADS * MAP_ITEMS, flip ^= 1) {
    int nxt[MAP_ITEMS];
    load(base0 + MAP_THREADS * MAP_ITEMS, nxt);     // in flight while the rows are handed out
    unsigned mine[MAP_ITEMS];
    int count = 0;
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) {
      mine[j] = __ballot_sync(0xffffffffu, cur[j] == e);
      count += __popc(mine[j]);
    }
    if (lane == 0) warp_sums[flip][warp] = count;
    __syncthreads();                // the other buffer's readers are past the previous barrier
    const int ws = warp_sums[flip][lane];
    int before = lane < warp ? ws : 0, total = ws;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      total += __shfl_xor_sync(0xffffffffu, total, o);
    }
    int row0 = next + before;
#pragma unroll
    for (int j = 0; j < MAP_ITEMS; ++j) {
      if (cur[j] == e) {
        const int i = (int)base0 + warp * (32 * MAP_ITEMS) + j * 32 + lane;
        const int row = row0 + __popc(mine[j] & ((1u << lane) - 1));
        if (row < rows_cap) src[row] = i;
        pos[i] = row;
      }
      row0 += __popc(mine[j]);
      cur[j] = nxt[j];
    }
    next += total;
  }
  __syncthreads();
  // what follows from a row's copy, for all rows at once (in the branch above its loads and division would come one after the other);
  // padding: this expert's own, and (last expert) the rows past the layout
  const int end = e == E - 1 ? rows_cap : min(start + pad, rows_cap);
  for (int r = start + threadIdx.x; r < end; r += MAP_THREADS) {
    const int i = r < next ? src[r] : -1;
    if (i < 0) src[r] = -1;
    if (src_token) src_token[r] = i < 0 ? -1 : i / topk;
    if (LOCAL) plan.probs_perm[r] = i < 0 ? 0.f : plan.probs[i];
  }
}

// out[i] = idx[i] >= 0 ? x[idx[i]] : 0
__global__ void gather_f32_kernel(const float* __restrict__ x, const int* __restrict__ idx, float* __restrict__ out, long n) {
  PB_GRID_WAIT();
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
  pbh::launch_dependent(moe_permutation_maps_kernel<false>, E, MAP_THREADS, 0, s, expert, (int)R, topk, E, row_start, padded,
      rows_cap, src, src_token, pos, LocalPlan{});
  return (int)cudaGetLastError();
}

// The padded layout and the maps of one rank's own R copies from their experts' counts (pb_moe_build_schedule and
// pb_moe_permutation_maps), and probs_perm: fp32 [rows_cap], the probability of each row's copy (0 for padding).
int pb_moe_local_plan(const long* expert, const int* counts, const float* probs, long R, int topk, int E, int rows_cap, int max_mblocks,
                      int* padded, int* row_start, int* mblock_expert, int* total, int* src, int* src_token, int* pos, float* probs_perm,
                      cudaStream_t s) {
  if (E <= 0 || E > 1024 || topk <= 0 || R < 0 || R > 2147483647L - 2 * MAP_THREADS * MAP_ITEMS) return -2;
  pbh::launch_dependent(moe_permutation_maps_kernel<true>, E, MAP_THREADS, 0, s, expert, (int)R, topk, E, nullptr, nullptr,
      rows_cap, src, src_token, pos, LocalPlan{counts, probs, padded, row_start, mblock_expert, total, probs_perm, max_mblocks});
  return (int)cudaGetLastError();
}

int pb_gather_f32(const float* x, const int* idx, float* out, long n, cudaStream_t s) {
  if (n == 0) return 0;
  const long blocks = (n + 255) / 256;
  pbh::launch_dependent(gather_f32_kernel, (unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, s, x, idx, out, n);
  return (int)cudaGetLastError();
}

}  // extern "C"
