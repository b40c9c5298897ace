// bf16 GEMM on CTA pairs (`cta_group::2`): one 256 x 256 output tile per 2-CTA cluster, persistent over tiles.
//
// Each CTA of the pair stages its own 128 rows of A and only *half* of B (128 of the 256 N columns); one thread of the
// even CTA issues `tcgen05.mma.cta_group::2.kind::f16` with M = 256, which reads both CTAs' shared memory and writes 128
// accumulator rows into each CTA's tensor memory.  Per CTA and 16-wide K step the MMA reads 4 KB of A + 4 KB of B for
// 128 clk of tensor-pipe time, where the one-CTA 128 x 256 tile (csrc/gemm_bf16.cu) reads 4 + 8 KB: the operand reads and
// the loads that feed them fall by a third, so six stages instead of four fit and the tensor pipe stops waiting for
// shared memory.  No TMA load is multicast: each CTA fetches exactly the bytes it keeps.
//
// Warp roles in both CTAs: warp 0 TMA producer, warp 1 MMA issuer (even CTA only), warps 2..9 epilogue (each CTA drains
// its 128 rows through one 4 KB swizzled staging box per warp and TMA stores / reduce-adds).  The accumulator is double
// buffered in tensor memory, so the epilogue of a tile overlaps the main loop of the next one.
//
// Synchronisation inside the pair (all waits bounded, errors through the status word):
//   full[stage]     lives in the even CTA: its producer arrives once expecting the bytes of BOTH CTAs; the odd CTA's
//                   TMA loads (`cta_group::2` form) count their bytes on that same barrier;
//   empty[stage]    in both CTAs, multicast `tcgen05.commit` of the MMA thread;
//   tmem_full[acc]  in both CTAs, multicast commit after the last K step of a tile;
//   tmem_empty[acc] in the even CTA: one arrival per epilogue warp of both CTAs, as soon as the warp has read its part.
// A cluster barrier closes the kernel so that neither CTA exits while its peer may still touch its memory.
//
// Split K: where the output has too few tiles for the SMs and K is long (the data gradient of an output head over few
// tokens: K is the vocabulary), the K range is cut into `splits` parts whose fp32 partial tiles go to a workspace
// [splits, M rounded up to 256, N]; a second kernel adds the parts in order, so the result does not depend on scheduling.
//
// Operand layouts and output modes as in csrc/gemm_bf16.cu.
#include "common.cuh"

namespace {

constexpr int BM = 128;            // rows per CTA (256 per pair)
constexpr int BN = 256;            // columns per pair; each CTA stages BN / 2 of B
constexpr int BK = 64;             // 128 bytes: one swizzle row
constexpr int UMMA_K = 16;
constexpr int STAGES = 6;
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 32 * (2 + EPI_WARPS);
constexpr int EPI_BUF_BYTES = 4096;      // per epilogue warp: 32 rows x 128 bytes
constexpr int GROUP_M = 8;               // in units of 256-row pair tiles
constexpr int A_BYTES = BM * BK * 2;
constexpr int B_BYTES = (BN / 2) * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;      // 32 KiB
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * EPI_BUF_BYTES + 1024 + 256;
constexpr int TMEM_COLS = 2 * BN;
static_assert(SMEM_BYTES <= 232448, "shared memory");
enum OutMode { OUT_BF16 = 0, OUT_F32 = 1, OUT_F32_ADD = 2 };

struct Barriers {
  uint64_t full[STAGES];     // used in the even CTA: 1 arrival, transaction bytes of both CTAs
  uint64_t empty[STAGES];    // both CTAs (multicast commit)
  uint64_t tmem_full[2];     // both CTAs (multicast commit)
  uint64_t tmem_empty[2];    // used in the even CTA: 2 x EPI_WARPS arrivals
  uint32_t tmem_base;
  int abort_flag;
};

// D(tmem, both CTAs) (+)= A . B over a CTA pair: M = 256 (128 rows per CTA), operands at the same shared-memory offsets
__device__ __forceinline__ void umma_f16_ss_2cta(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (pb::mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!pb::mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > PB_WAIT_CYCLES) return false;
  }
  return true;
}

// Warp-collective wait: lane 0 polls, the other lanes park at the shuffle (no issue slots, no shared-memory traffic).
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int lane) {
  int got = 1;
  if (lane == 0 && !pb::mbar_try_wait(bar, parity)) {
    const long long t0 = clock64();
    while (!pb::mbar_try_wait(bar, parity)) {
      __nanosleep(64);
      if (*abort_flag || clock64() - t0 > PB_WAIT_CYCLES) {
        got = 0;
        break;
      }
    }
  }
  return __shfl_sync(0xffffffffu, got, 0) != 0;
}

__device__ __forceinline__ void tile_coords(int tile, int num_m, int num_n, int& mb, int& nb) {
  const int per_group = GROUP_M * num_n;
  const int g = tile / per_group;
  const int first_m = g * GROUP_M;
  const int gm = min(GROUP_M, num_m - first_m);
  const int r = tile - g * per_group;
  mb = first_m + r % gm;
  nb = r / gm;
}

template <int A_MN, int B_MN, int OUT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmD, int M, int N, int K, int splits, int kb_per_split,
                      int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_ab = smem;
  uint8_t* smem_epi = smem + STAGES * STAGE_BYTES;
  Barriers* bars = reinterpret_cast<Barriers*>(smem_epi + EPI_WARPS * EPI_BUF_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = pb::cluster_ctarank();      // 0: even CTA (issues the MMAs), 1: odd CTA
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int num_m = (M + 2 * BM - 1) / (2 * BM);
  const int num_n = (N + BN - 1) / BN;
  const int tiles_per_split = num_m * num_n;
  const int num_tiles = tiles_per_split * splits;
  const int num_kb = (K + BK - 1) / BK;
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
  PB_GRID_WAIT();
  pb::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (pb::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        int mb, nb;
        const int split = tile / tiles_per_split;
        tile_coords(tile - split * tiles_per_split, num_m, num_n, mb, nb);
        const int m0 = (mb * 2 + (int)cta) * BM;         // 128-row block of this CTA
        const int n0 = nb * BN + (int)cta * (BN / 2);    // this CTA's half of the B tile
        const int kb_end = min(num_kb, (split + 1) * kb_per_split);
        for (int kb = split * kb_per_split; kb < kb_end; ++kb) {
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
          if (A_MN == 0) {
            pb::tma_load_2d_pair(sa, &tmA, fb, kb * BK, m0);
          } else {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i) pb::tma_load_2d_pair(sa + i * (BK * 128), &tmA, fb, m0 + i * 64, kb * BK);
          }
          if (B_MN == 0) {
            pb::tma_load_2d_pair(sb, &tmB, fb, kb * BK, n0);
          } else {
#pragma unroll
            for (int i = 0; i < BN / 128; ++i) pb::tma_load_2d_pair(sb + i * (BK * 128), &tmB, fb, n0 + i * 64, kb * BK);
          }
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
      constexpr uint32_t idesc = pb::make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        if (!wait_or_abort(&bars->tmem_empty[acc], acc_phase ^ 1, abort_flag)) {
          atomicCAS(status, 0, PB_ERR_TIMEOUT_MMA);
          bars->abort_flag = 1;
          break;
        }
        pb::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        const int kb0 = tile / tiles_per_split * kb_per_split, kb_end = min(num_kb, kb0 + kb_per_split);
        for (int kb = kb0; kb < kb_end; ++kb) {
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
            const uint64_t da = A_MN ? pb::make_smem_desc(sa + k * (UMMA_K * 128), BK * 128, 1024, 2)
                                     : pb::make_smem_desc(sa + k * (UMMA_K * 2), 0, 1024, 2);
            const uint64_t db = B_MN ? pb::make_smem_desc(sb + k * (UMMA_K * 128), BK * 128, 1024, 2)
                                     : pb::make_smem_desc(sb + k * (UMMA_K * 2), 0, 1024, 2);
            umma_f16_ss_2cta(d_tmem, da, db, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
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
    const int half = ew >> 2;                   // column half of the tile (ew and ew + 4 share a lane quarter)
    constexpr int HC = BN / 2;                  // columns per thread
    uint8_t* ebuf = smem_epi + ew * EPI_BUF_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int mb, nb;
      const int split = tile / tiles_per_split;
      tile_coords(tile - split * tiles_per_split, num_m, num_n, mb, nb);
      const int m0 = (mb * 2 + (int)cta) * BM + lane_grp * 32, n0 = nb * BN + half * HC;
      const int row0 = split * num_m * 2 * BM + m0;     // in the output, or in the workspace of the parts
      if (!warp_wait_or_abort(&bars->tmem_full[acc], acc_phase, abort_flag, lane)) {
        atomicCAS(status, 0, PB_ERR_TIMEOUT_EPILOGUE);
        bars->abort_flag = 1;
        break;
      }
      pb::tc_fence_after();
      const uint32_t t_row = tmem_base + (uint32_t(lane_grp * 32) << 16) + acc * BN + half * HC;
      auto stage_and_store = [&](const uint4* chunks, int n) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(ebuf + lane * 128 + ((c ^ (lane & 7)) << 4)) = chunks[c];
        pb::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && m0 < M && n < N) {
          if (OUT == OUT_F32_ADD) pb::tma_reduce_add_2d(&tmD, ebuf, n, row0);
          else pb::tma_store_2d(&tmD, ebuf, n, row0);
          pb::tma_store_commit();
          pb::tma_store_wait_read<0>();    // the staging buffer may be overwritten by the next round
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int c = 0; c < HC / 64; ++c) {
        uint32_t r[64];
        pb::tmem_ld_32x32b_x32(t_row + c * 64, r);
        pb::tmem_ld_32x32b_x32(t_row + c * 64 + 32, r + 32);
        pb::tmem_wait_ld();
        if (c == HC / 64 - 1) {            // the accumulator is in registers or stored: hand its buffer back
          pb::tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (cta == 0) pb::mbar_arrive(&bars->tmem_empty[acc]);
            else pb::mbar_arrive_remote(pb::mapa_shared(&bars->tmem_empty[acc], 0));
          }
        }
        uint4 ch[8];
        if (OUT == OUT_BF16) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            ch[j] = make_uint4(pb::pack_bf16x2(__uint_as_float(r[8 * j]), __uint_as_float(r[8 * j + 1])),
                               pb::pack_bf16x2(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])),
                               pb::pack_bf16x2(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])),
                               pb::pack_bf16x2(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])));
          stage_and_store(ch, n0 + c * 64);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              ch[j] = make_uint4(r[h * 32 + 4 * j], r[h * 32 + 4 * j + 1], r[h * 32 + 4 * j + 2], r[h * 32 + 4 * j + 3]);
            stage_and_store(ch, n0 + c * 64 + h * 32);
          }
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (lane == 0) pb::tma_store_wait_all<0>();   // all stores of this warp are complete before the CTA exits
  }

  // ---------------------------------------------------------------- teardown
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

template <int A_MN, int B_MN, int OUT>
int launch(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tD, int M, int N, int K, int* status,
           int max_ctas, cudaStream_t stream, int splits = 1) {
  auto kern = gemm_bf16_2cta_kernel<A_MN, B_MN, OUT>;
  static std::atomic<bool> allowed[pbh::MAX_DEVICES];
  const int rc = pbh::allow_shared_memory(kern, SMEM_BYTES, allowed);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // a persistent grid must not exceed the number of CTA pairs the device can keep resident at once (SMs pair up
  // inside a GPC, so this can be fewer than SMs / 2)
  static int max_pairs = 0;
  if (max_pairs == 0) {
    cfg.gridDim = dim3(pbh::sm_count() / 2 * 2, 1, 1);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = pbh::sm_count() / 2;
    }
    max_pairs = n;
  }
  const int num_kb = (K + BK - 1) / BK;
  const int kb_per_split = (num_kb + splits - 1) / splits;
  const int tiles = ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN) * splits;
  int pairs = max_pairs;
  if (max_ctas > 0 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  if (tiles < pairs) pairs = tiles;
  if (pairs < 1) pairs = 1;
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.stream = stream;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // (pb::grid_wait)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  return (int)cudaLaunchKernelEx(&cfg, kern, tA, tB, tD, M, N, K, splits, kb_per_split, status);
}

// out[m, n] (=|+=) sum over the parts of ws[s, m, n]; four columns per thread, parts in order
template <int OUT>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ ws, void* __restrict__ out, int M, int N, long ldd, int splits, long part) {
  PB_GRID_WAIT();
  const int nv = N / 4;
  const long i = blockIdx.x * 256L + threadIdx.x;
  const long m = i / nv;
  if (m >= M) return;
  const int n = (int)(i - m * nv) * 4;
  const float4* p = reinterpret_cast<const float4*>(ws + m * N + n);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float4 v = p[s * (part / 4)];
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  if (OUT == OUT_BF16) {
    uint2 h = make_uint2(pb::pack_bf16x2(a.x, a.y), pb::pack_bf16x2(a.z, a.w));
    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + m * ldd + n) = h;
  } else {
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + m * ldd + n);
    if (OUT == OUT_F32_ADD) {
      const float4 v = *o;
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    *o = a;
  }
}

int check_operands(const void* A, const void* B, const void* D, long lda, long ldb, long ldd, int out_mode) {
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16) ||
      (reinterpret_cast<uintptr_t>(D) % 16))
    return -2;
  return (out_mode == 0 ? (ldd % 8) : (ldd % 4)) ? -2 : 0;
}

int operand_maps(CUtensorMap& tA, CUtensorMap& tB, const void* A, const void* B, int M, int N, int K, long lda, long ldb,
                 int a_mn, int b_mn) {
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  int rc;
  if (!a_mn) rc = pbh::make_tmap_2d(&tA, A, bf, 2, M, K, lda, BM, BK, sw);
  else rc = pbh::make_tmap_2d(&tA, A, bf, 2, K, M, lda, BK, 64, sw);
  if (rc) return rc;
  if (!b_mn) return pbh::make_tmap_2d(&tB, B, bf, 2, N, K, ldb, BN / 2, BK, sw);
  return pbh::make_tmap_2d(&tB, B, bf, 2, K, N, ldb, BK, 64, sw);
}

}  // namespace

// Same contract as pb_gemm_bf16 (csrc/gemm_bf16.cu); output tile 256 x 256 per CTA pair.
extern "C" int pb_gemm_bf16_2cta(const void* A, const void* B, void* D, int M, int N, int K, long lda, long ldb, long ldd,
                                 int a_mn, int b_mn, int out_mode, int max_ctas, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  int rc = check_operands(A, B, D, lda, ldb, ldd, out_mode);
  if (rc) return rc;
  CUtensorMap tA, tB, tD;
  if ((rc = operand_maps(tA, tB, A, B, M, N, K, lda, ldb, a_mn, b_mn))) return rc;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  // output boxes: 32 rows x 128 bytes (64 bf16 / 32 fp32 columns); rows and columns past M, N are clipped by TMA
  if (out_mode == 0) rc = pbh::make_tmap_2d(&tD, D, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, N, ldd, 32, 64, sw);
  else rc = pbh::make_tmap_2d(&tD, D, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, M, N, ldd, 32, 32, sw);
  if (rc) return rc;

#define PB_DISPATCH_OUT(AM, BMN)                                                                         \
  switch (out_mode) {                                                                                    \
    case 0: return launch<AM, BMN, OUT_BF16>(tA, tB, tD, M, N, K, status, max_ctas, stream);             \
    case 1: return launch<AM, BMN, OUT_F32>(tA, tB, tD, M, N, K, status, max_ctas, stream);              \
    case 2: return launch<AM, BMN, OUT_F32_ADD>(tA, tB, tD, M, N, K, status, max_ctas, stream);          \
    default: return -3;                                                                                  \
  }
  if (!a_mn && !b_mn) { PB_DISPATCH_OUT(0, 0) }
  else if (!a_mn && b_mn) { PB_DISPATCH_OUT(0, 1) }
  else if (a_mn && b_mn) { PB_DISPATCH_OUT(1, 1) }
  else { PB_DISPATCH_OUT(1, 0) }
  return -3;
}

// The same with K cut into `splits` parts.  ws: fp32 [splits, M rounded up to 256, N] (not initialised); N % 4 == 0 and
// splits <= ceil(K / 64).  A split count that would leave a part without a K step is lowered.
extern "C" int pb_gemm_bf16_splitk(const void* A, const void* B, void* D, float* ws, int M, int N, int K, long lda, long ldb,
                                   long ldd, int a_mn, int b_mn, int out_mode, int splits, int* status,
                                   cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  int rc = check_operands(A, B, D, lda, ldb, ldd, out_mode);
  if (rc) return rc;
  const int num_kb = (K + BK - 1) / BK;
  if (N % 4 || splits < 1 || splits > num_kb || out_mode < 0 || out_mode > 2 || (reinterpret_cast<uintptr_t>(ws) % 16)) return -2;
  const int per = (num_kb + splits - 1) / splits;
  splits = (num_kb + per - 1) / per;
  CUtensorMap tA, tB, tD;
  if ((rc = operand_maps(tA, tB, A, B, M, N, K, lda, ldb, a_mn, b_mn))) return rc;
  const long rows = (M + 2 * BM - 1) / (2 * BM) * (2 * BM);
  if ((rc = pbh::make_tmap_2d(&tD, ws, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, rows * splits, N, N, 32, 32,
                              CU_TENSOR_MAP_SWIZZLE_128B)))
    return rc;
  if (!a_mn && !b_mn) rc = launch<0, 0, OUT_F32>(tA, tB, tD, M, N, K, status, 0, stream, splits);
  else if (!a_mn && b_mn) rc = launch<0, 1, OUT_F32>(tA, tB, tD, M, N, K, status, 0, stream, splits);
  else if (a_mn && b_mn) rc = launch<1, 1, OUT_F32>(tA, tB, tD, M, N, K, status, 0, stream, splits);
  else rc = launch<1, 0, OUT_F32>(tA, tB, tD, M, N, K, status, 0, stream, splits);
  if (rc) return rc;
  const unsigned blocks = (unsigned)(((long)M * (N / 4) + 255) / 256);
  if (out_mode == OUT_BF16) pbh::launch_dependent(splitk_reduce_kernel<OUT_BF16>, blocks, 256, 0, stream, ws, D, M, N, ldd, splits,
      rows * N);
  else if (out_mode == OUT_F32) pbh::launch_dependent(splitk_reduce_kernel<OUT_F32>, blocks, 256, 0, stream, ws, D, M, N, ldd,
      splits, rows * N);
  else pbh::launch_dependent(splitk_reduce_kernel<OUT_F32_ADD>, blocks, 256, 0, stream, ws, D, M, N, ldd, splits, rows * N);
  return (int)cudaGetLastError();
}
