// Weight gradients of the experts, added to what is there (fp32 main gradients), on CTA pairs (`cta_group::2`):
//   D[e][N, K] += dy_e^T . x_e,  dy [rows, N], x [rows, K], reduction over the expert's rows (schedule of csrc/grouped_gemm.cu).
//
// A tile moves its fp32 values in and out of memory for a reduction of a few hundred rows at most, and that traffic bounds it.
// Adding in L2 (TMA reduce, the one-CTA kernel) runs at 2.4 TB/s each way; here every epilogue warp fetches the old values of its
// 32 x 32 chunks two ahead, adds in registers and stores.  256 x 256 tiles on pairs, because operand traffic is next: a CTA
// fetches 32 KB per 512 clocks of MMA instead of 48 KB, and that leaves shared memory for the chunks.
// Both GEMMs of 64 experts of 2048 x 768 (302 M values, 370 us of copy bandwidth), one CTA -> pairs: 2 rows per expert 475 -> 372
// us, 128 rows 476 -> 414, 512 rows 508 -> 460 (with 470 MB of operands 441 us of copy bandwidth).  The same pairs for the other
// expert GEMMs (tiles of two row blocks of an expert) gained 5 % alone and nothing in a training loop under the power cap.
//
// Warps: 0 TMA producer, 1 MMA issuer (even CTA), 2..9 epilogue (32 rows x 128 columns of the CTA's 128 x 256 each).
#include "common.cuh"

namespace {

constexpr int BM = 128;            // rows per CTA (256 per pair)
constexpr int BN = 256;            // columns per pair; each CTA stages BN / 2 of B
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 32 * (2 + EPI_WARPS);
constexpr int BUF_BYTES = 4096;
constexpr int A_BYTES = BM * BK * 2;
constexpr int B_BYTES = (BN / 2) * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;      // 32 KiB
constexpr int TMEM_COLS = 2 * BN;
constexpr int STAGES = 4;
constexpr int BUFS = 3;                  // chunks of [32 rows, 32 fp32] per epilogue warp
constexpr int TILE_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * BUFS * BUF_BYTES;
constexpr int SMEM_BYTES = TILE_BYTES + 512;
static_assert(SMEM_BYTES <= 232448, "shared memory");

struct Barriers {
  uint64_t full[STAGES];         // used in the even CTA: 1 arrival, transaction bytes of both CTAs
  uint64_t empty[STAGES];        // both CTAs (multicast commit)
  uint64_t tmem_full[2];     // both CTAs (multicast commit)
  uint64_t tmem_empty[2];    // used in the even CTA: 2 x EPI_WARPS arrivals
  uint64_t old_full[EPI_WARPS][BUFS];   // old values of a chunk
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(Barriers) <= 512, "barriers");

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (pb::mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!pb::mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > PB_WAIT_CYCLES) return false;
  }
  return true;
}

// Warp-collective wait: lane 0 polls, the other lanes park at the shuffle.
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int lane) {
  int got = 1;
  if (lane == 0) got = wait_or_abort(bar, parity, abort_flag);
  return __shfl_sync(0xffffffffu, got, 0) != 0;
}

struct Tile {
  int expert;
  int m0, n0;      // first row of this CTA's half and first column of the pair's tile, in D[e]
  int k_begin;     // first reduction block (units of BK)
  int k_blocks;    // 0: an expert without tokens has nothing to add
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_wgrad_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmD, int N, int K, int E, const int* __restrict__ row_start,
                          const int* __restrict__ padded, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_pair[];
  uint8_t* smem_ab = smem_pair;
  uint8_t* smem_epi = smem_ab + STAGES * STAGE_BYTES;
  Barriers* bars = reinterpret_cast<Barriers*>(smem_pair + TILE_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = pb::cluster_ctarank();      // 0: even CTA (issues the MMAs), 1: odd CTA
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  volatile int* abort_flag = &bars->abort_flag;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      pb::mbar_init(&bars->full[i], 1);
      pb::mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      pb::mbar_init(&bars->tmem_full[i], 1);
      pb::mbar_init(&bars->tmem_empty[i], 2 * EPI_WARPS);
    }
    for (int w = 0; w < EPI_WARPS; ++w)
      for (int i = 0; i < BUFS; ++i) pb::mbar_init(&bars->old_full[w][i], 1);
    bars->abort_flag = 0;
    pb::fence_barrier_init();
    pb::prefetch_tmap(&tmA);
    pb::prefetch_tmap(&tmB);
    pb::prefetch_tmap(&tmD);
  }
  if (warp == 1) {
    pb::tmem_alloc<2>(&bars->tmem_base, TMEM_COLS);
    pb::tmem_relinquish<2>();
  }
  pb::tc_fence_before();
  __syncthreads();
  pb::cluster_sync();          // barriers of both CTAs are initialised before any remote arrive / multicast commit
  pb::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  const int num_m = (N + 2 * BM - 1) / (2 * BM), num_n = (K + BN - 1) / BN;
  const int per_e = num_m * num_n, num_tiles = per_e * E;
  auto tile_at = [&](int tile) {
    Tile t;
    const int e = tile / per_e, r = tile - e * per_e;
    t.expert = e;
    t.m0 = (r % num_m * 2 + (int)cta) * BM;
    t.n0 = r / num_m * BN;
    t.k_begin = row_start[e] / BK;
    t.k_blocks = padded[e] / BK;
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (pb::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const Tile t = tile_at(tile);
        const int n0 = t.n0 + (int)cta * (BN / 2);                  // this CTA's half of the B tile
        for (int kb = t.k_begin; kb < t.k_begin + t.k_blocks; ++kb) {
          if (!wait_or_abort(&bars->empty[stage], phase ^ 1, abort_flag)) {
            atomicCAS(status, 0, PB_ERR_TIMEOUT_TMA);
            bars->abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem_ab + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          if (cta == 0) pb::mbar_expect_tx(&bars->full[stage], 2 * STAGE_BYTES);
          const uint32_t fb = pb::mapa_shared(&bars->full[stage], 0);   // the even CTA's barrier
#pragma unroll
          for (int i = 0; i < BM / 64; ++i) pb::tma_load_2d_pair(sa + i * (BK * 128), &tmA, fb, t.m0 + i * 64, kb * BK);
#pragma unroll
          for (int i = 0; i < BN / 128; ++i) pb::tma_load_2d_pair(sb + i * (BK * 128), &tmB, fb, n0 + i * 64, kb * BK);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (cta == 0 && pb::elect_one()) {
      // ---------------------------------------------------------- MMA issuer (even CTA)
      constexpr uint32_t idesc = pb::make_idesc_bf16(2 * BM, BN, 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const Tile t = tile_at(tile);
        if (t.k_blocks == 0) continue;
        if (!wait_or_abort(&bars->tmem_empty[acc], acc_phase ^ 1, abort_flag)) {
          atomicCAS(status, 0, PB_ERR_TIMEOUT_MMA);
          bars->abort_flag = 1;
          break;
        }
        pb::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!wait_or_abort(&bars->full[stage], phase, abort_flag)) {
            atomicCAS(status, 0, PB_ERR_TIMEOUT_MMA);
            bars->abort_flag = 1;
            ok = false;
            break;
          }
          pb::tc_fence_after();
          const uint32_t sa = pb::smem_u32(smem_ab + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t da = pb::make_smem_desc(sa + k * (UMMA_K * 128), BK * 128, 1024, 2);
            const uint64_t db = pb::make_smem_desc(sb + k * (UMMA_K * 128), BK * 128, 1024, 2);
            pb::umma_f16_ss_2cta(d_tmem, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          pb::umma_commit_2cta(&bars->empty[stage], 3);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        pb::umma_commit_2cta(&bars->tmem_full[acc], 3);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs, 128 rows each)
    const int ew = warp - 2;                    // 0..7
    const int lane_grp = warp & 3;              // TMEM lane quarter this warp may access
    const int half = ew >> 2;                   // column half of the tile
    constexpr int HC = BN / 2;                  // columns per warp
    constexpr int CHUNKS = HC / 32;
    uint8_t* ebuf = smem_epi + ew * BUFS * BUF_BYTES;
    // old values: the chunk to fetch next (tile, chunk of the tile, number)
    int ftile = first, fchunk = 0;
    uint32_t fn = 0;
    auto fetch = [&]() {                        // lane 0 only
      while (ftile < num_tiles) {
        const Tile t = tile_at(ftile);
        const int m = t.m0 + lane_grp * 32, n = t.n0 + half * HC + fchunk * 32;
        const bool skip = t.k_blocks == 0, there = !skip && m < N && n < K;
        if (there) {
          const uint32_t b = fn % BUFS;
          pb::mbar_expect_tx(&bars->old_full[ew][b], BUF_BYTES);
          pb::tma_load_3d(ebuf + b * BUF_BYTES, &tmD, &bars->old_full[ew][b], n, m, t.expert);
          ++fn;
        }
        if (skip || ++fchunk == CHUNKS) {
          fchunk = 0;
          ftile += step;
        }
        if (there) return;
      }
    };
    if (lane == 0) {
      fetch();
      fetch();
    }
    uint32_t num = 0;                           // chunks so far
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = first; tile < num_tiles && ok; tile += step) {
      const Tile t = tile_at(tile);
      if (t.k_blocks == 0) continue;
      const int m0 = t.m0 + lane_grp * 32, n0 = t.n0 + half * HC;
      if (!warp_wait_or_abort(&bars->tmem_full[acc], acc_phase, abort_flag, lane)) {
        atomicCAS(status, 0, PB_ERR_TIMEOUT_EPILOGUE);
        bars->abort_flag = 1;
        break;
      }
      pb::tc_fence_after();
      const uint32_t t_row = tmem_base + (uint32_t(lane_grp * 32) << 16) + acc * BN + half * HC;
#pragma unroll 1
      for (int c = 0; c < CHUNKS; ++c) {
        uint32_t r[32];
        pb::tmem_ld_32x32b_x32(t_row + c * 32, r);
        pb::tmem_wait_ld();
        if (c == CHUNKS - 1) {                  // the accumulator is in registers or stored: hand its buffer back
          pb::tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (cta == 0) pb::mbar_arrive(&bars->tmem_empty[acc]);
            else pb::mbar_arrive_remote(pb::mapa_shared(&bars->tmem_empty[acc], 0));
          }
        }
        const int n = n0 + c * 32;
        if (m0 >= N || n >= K) continue;
        uint8_t* buf = ebuf + num % BUFS * BUF_BYTES;
        if (!warp_wait_or_abort(&bars->old_full[ew][num % BUFS], (num / BUFS) & 1, abort_flag, lane)) {
          atomicCAS(status, 0, PB_ERR_TIMEOUT_EPILOGUE);
          bars->abort_flag = 1;
          ok = false;
          break;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4* p = reinterpret_cast<float4*>(buf + lane * 128 + ((j ^ (lane & 7)) << 4));
          const float4 v = *p;
          *p = make_float4(v.x + __uint_as_float(r[4 * j]), v.y + __uint_as_float(r[4 * j + 1]),
                           v.z + __uint_as_float(r[4 * j + 2]), v.w + __uint_as_float(r[4 * j + 3]));
        }
        pb::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // the chunk before has left its buffer, which takes the chunk after the next
          pb::tma_store_wait_read<0>();
          fetch();
          pb::tma_store_3d(&tmD, buf, n, m0, t.expert);
          pb::tma_store_commit();
        }
        __syncwarp();
        ++num;
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (lane == 0) pb::tma_store_wait_all<0>();   // all stores of this warp are complete before the CTA exits
  }

  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  pb::tc_fence_before();
  __syncthreads();
  pb::cluster_sync();          // the peer may still multicast into / read from this CTA until here
  if (warp == 1) {
    pb::tc_fence_after();
    pb::tmem_dealloc<2>(tmem_base, TMEM_COLS);
  }
}

}  // namespace

// Arguments as pb_grouped_gemm, mode 2 with accumulate.
int pb_grouped_wgrad_pair(const void* dy, const void* x, void* D, int rows_cap, int N, int K, int E, const int* row_start,
                          const int* padded, int* status, cudaStream_t s) {
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  CUtensorMap tA, tB, tD;
  int rc;
  if ((rc = pbh::make_tmap_2d(&tA, dy, bf, 2, rows_cap, N, N, BK, 64, sw))) return rc;
  if ((rc = pbh::make_tmap_2d(&tB, x, bf, 2, rows_cap, K, K, BK, 64, sw))) return rc;
  if ((rc = pbh::make_tmap_3d(&tD, D, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, E, N, K, K, (long)N * K, 1, 32, 32, sw))) return rc;
  static std::atomic<bool> done[pbh::MAX_DEVICES];
  if ((rc = pbh::allow_shared_memory(grouped_wgrad_pair_kernel, SMEM_BYTES, done))) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const long tiles = (long)E * ((N + 2 * BM - 1) / (2 * BM)) * ((K + BN - 1) / BN), pairs = pbh::sm_count() / 2;
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)), 1, 1);
  cfg.stream = s;
  return (int)cudaLaunchKernelEx(&cfg, grouped_wgrad_pair_kernel, tA, tB, tD, N, K, E, row_start, padded, status);
}
