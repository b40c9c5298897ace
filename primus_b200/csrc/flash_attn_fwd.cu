// Flash-attention forward for sm_100a (causal or full, GQA / MQA / MLA head shapes).
//
// Persistent: one CTA per SM takes a pair of 128-row query tiles of one head after the other (the next one from the hardware
// scheduler, by clusterlaunchcontrol.try_cancel, so that the longest pairs of the grid still start first) and walks their KV
// sequence in blocks of 128:
//   warp 0       : scheduler and TMA producer (Q tiles, K / V blocks through mbarrier rings that run on across pairs)
//   warps 1, 2   : tcgen05 issuers of  S_t = Q_t K^T  and of  O_t += P_t V  for both tiles t.  An issuing thread stays only a
//                  few MMAs ahead of the tensor pipe, so that its waits leave gaps; two threads fill each other's
//   warps 4..7   : softmax warpgroup of tile 0        warps 8..11 : softmax warpgroup of tile 1
// One thread owns one query row: it takes the whole S row from tensor memory into registers, which frees S for the other
// tile's next block, keeps the running max / sum, and writes P = exp2(.) as packed bf16 to the tile's own columns of tensor
// memory; the P.V MMA takes its A operand straight from there, so P never touches shared memory.
// Tensor memory: one S buffer for both tiles (128 columns), P_0 and P_1 (64 each), O_0 and O_1 (128 each).  With S in P's place,
// as two buffers, S of a tile's next block had to wait for its P.V and with it for the exponentials: 3485 clocks per pair of
// 128 x 128 blocks, of which the GEMMs take 2048; now 2800, with the special-function unit busy for 2048.  A pair's start and
// end (Q, tensor memory, output: 8000 clocks of 20250 for a window of 128) pass under its neighbours' blocks.
// Before and now, us (median of the kernel in a short run): 8192 x 32/8 x 128 483 -> 412 (1.33 PFLOP/s, under the power cap), 2048
// x 32/8 x 128 43 -> 35, 4096 x 16 x 192/128 83 -> 74, window of 128 at 2 x 2048 x 64/8 x 64 79 -> 51.  Tensor pipe busy 65 % of
// the time at 4096 x 32/8 x 128, 62 % with 192/128.
// O is rescaled in tensor memory only when the running max grew by more than 2^8.
// V is consumed straight from its [kv, d] row-major tile through an MN-major descriptor, so no
// transposes are needed.  All waits are bounded.
//
// Replaces `flash_attn_func` call sites of the reference
// (primus/backends/megatron/core/extensions/primus_turbo.py:812-823, 888-990); MLA shape
// d_qk = 192 / d_v = 128 as in primus/configs/models/megatron/deepseek_v2_lite.yaml:10-33.
#include "common.cuh"

namespace {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int ATOM_BYTES = 128 * 128;  // 128 rows x 64 bf16
constexpr int FA_THREADS = 384;
constexpr int MAX_GRID_Y = 65535;
// Registers move from the producer / issuer warpgroup to the softmax warpgroups, which hold a row of S: 4 * 120 + 8 * 192 =
// 12 * 168 per lane, the allocation of the launch.
constexpr int FA_REGS_AUX = 120, FA_REGS_SOFTMAX = 192;

template <int DQK, int DV>
struct FaCfg {
  static constexpr int KS = 2;                      // K stages
  static constexpr int VS = (DQK > 128) ? 1 : 2;    // V stages
  static constexpr bool STAGE = DQK <= 128;         // room for a staging tile per softmax warpgroup; else O leaves through Q's
  static constexpr int Q_BYTES = BQ * DQK * 2;      // one tile
  static constexpr int K_BYTES = BKV * DQK * 2;
  static constexpr int V_BYTES = BKV * DV * 2;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + KS * K_BYTES + VS * V_BYTES + (STAGE ? 2 * ATOM_BYTES : 0) + 512;
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};

struct FaBars {
  uint4 next[2];        // answers of try_cancel, by item parity
  uint64_t next_full[2], next_empty[2];
  uint64_t q_full[2], q_empty[2];   // per tile
  uint64_t k_full[2], k_empty[2];
  uint64_t v_full[2], v_empty[2];
  uint64_t s_full[2];   // per tile
  uint64_t s_read;      // the S buffer is in registers
  uint64_t p_full[2];   // per tile
  uint64_t pv_done[2];  // per tile
  uint64_t o_free[2];   // per tile: O of the finished pair has been read
  uint32_t tmem_base;
  int abort_flag;
};

// What a pair of query tiles needs; step j stands for key block j_lo + j.
struct FaItem {
  int head, batch, kv_head, qt0;
  int j_lo, n;          // first key block and number of steps of the pair
  int lo[2], nb[2];     // steps of each tile: [lo, nb)
  __device__ __forceinline__ bool has(int t, int j) const { return j >= lo[t] && j < nb[t]; }
};

__device__ __forceinline__ bool fa_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (pb::mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!pb::mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > PB_WAIT_CYCLES) return false;
  }
  return true;
}

// in a role's lambda: a wait that runs out ends the role
#define FA_WAIT(bar, parity, code)                 \
  if (!fa_wait((bar), (parity), abort_flag)) {     \
    atomicCAS(status, 0, (code));                  \
    bars->abort_flag = 1;                          \
    return false;                                  \
  }

template <int DQK, int DV, bool WIN>
__global__ void __launch_bounds__(FA_THREADS, 1)
flash_attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                      float* __restrict__ lse, int seq, int seq_k, int q_off_blocks, int hq, int hkv,
                      float scale_log2, int causal, int window_arg, const float* __restrict__ sinks_arg, float softcap_arg,
                      int* status) {
  // WIN = false: the plain instantiation carries no code for windows or sinks
  const int window = WIN ? window_arg : 0;
  const float* sinks = WIN ? sinks_arg : nullptr;
  // softcap > 0: scores become softcap * tanh(scale * s / softcap) before the softmax
  const float softcap = WIN ? softcap_arg : 0.f;
  // seq: query rows per sequence; seq_k: key rows per sequence; query row i sits at key position
  // q_off_blocks * 128 + i (causal masking is relative to that position).  window > 0 (causal only): a query attends
  // to its last `window` keys, itself included.  sinks: optional per-query-head logit (natural-log units) that only
  // adds exp(sink) to the softmax denominator.
  using C = FaCfg<DQK, DV>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_smem = smem;  // two tiles
  uint8_t* k_smem = q_smem + 2 * C::Q_BYTES;
  uint8_t* v_smem = k_smem + C::KS * C::K_BYTES;
  uint8_t* o_smem = v_smem + C::VS * C::V_BYTES;
  FaBars* bars = reinterpret_cast<FaBars*>(o_smem + (C::STAGE ? 2 * ATOM_BYTES : 0));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_q128 = seq / BQ;
  const int num_pairs = (num_q128 + 1) / 2;
  const int n_kv = seq_k / BKV;
  volatile int* abort_flag = &bars->abort_flag;
  // grid (heads, batch, pairs): x-fastest issue order starts all heads of the heaviest (longest KV range) pair first
  auto item_of = [&](int3 b) {
    FaItem w;
    w.qt0 = 2 * (num_pairs - 1 - b.z);
    w.head = b.x;
    w.batch = b.y;
    w.kv_head = w.head / (hq / hkv);
    const int qk0 = w.qt0 + q_off_blocks;      // key block of the first tile's diagonal
    // first key block that any row of a tile can see
    w.j_lo = window > 0 ? max(0, qk0 * BQ - window + 1) / BKV : 0;
    w.lo[0] = 0;
    w.lo[1] = (window > 0 ? max(0, (qk0 + 1) * BQ - window + 1) / BKV : 0) - w.j_lo;
    w.nb[0] = (causal ? min(n_kv, qk0 + 1) : n_kv) - w.j_lo;
    w.nb[1] = w.qt0 + 1 < num_q128 ? (causal ? min(n_kv, qk0 + 2) : n_kv) - w.j_lo : 0;
    w.n = max(w.nb[0], w.nb[1]);
    return w;
  };

  // the pair after pair `item` of this CTA: waits for the scheduler's answer; false: there is none
  auto next_item = [&](uint32_t item, int3& b) -> bool {
    const uint32_t nx = item & 1;
    FA_WAIT(&bars->next_full[nx], (item >> 1) & 1, PB_ERR_TIMEOUT_MMA);
    const bool more = pb::clc_taken(&bars->next[nx], b);
    pb::fence_proxy_async_smem();
    pb::mbar_arrive(&bars->next_empty[nx]);
    return more;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      pb::mbar_init(&bars->next_full[i], 1);
      pb::mbar_init(&bars->next_empty[i], 2 + FA_THREADS - 128);   // the issuers and the softmax threads
      pb::mbar_init(&bars->q_full[i], 1);
      pb::mbar_init(&bars->q_empty[i], 1);
      pb::mbar_init(&bars->k_full[i], 1);
      pb::mbar_init(&bars->k_empty[i], 1);
      pb::mbar_init(&bars->v_full[i], 1);
      pb::mbar_init(&bars->v_empty[i], 1);
      pb::mbar_init(&bars->s_full[i], 1);
      pb::mbar_init(&bars->p_full[i], 4);   // one arrival per softmax warp of the tile
      pb::mbar_init(&bars->pv_done[i], 1);
      pb::mbar_init(&bars->o_free[i], 4);
    }
    pb::mbar_init(&bars->s_read, 4);
    bars->abort_flag = 0;
    pb::fence_barrier_init();
    pb::prefetch_tmap(&tmQ);
    pb::prefetch_tmap(&tmK);
    pb::prefetch_tmap(&tmV);
    pb::prefetch_tmap(&tmO);
  }
  if (warp == 1) {
    pb::tmem_alloc<1>(&bars->tmem_base, 512);
    pb::tmem_relinquish<1>();
  }
  pb::tc_fence_before();
  __syncthreads();
  PB_GRID_WAIT();
  pb::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  constexpr uint32_t P_COL = 128, O_COL = 256;      // S [0, 128)  P_t [128 + 64 t, +64)  O_t [256 + 128 t, +DV)

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FA_REGS_AUX));
    if (warp == 0 && pb::elect_one()) {
      // ------------------------------------------------------------------ scheduler and producer
      [&]() -> bool {
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        uint32_t kc = 0, vc = 0, qc[2] = {0, 0};       // K / V blocks and Q tiles loaded so far
        for (uint32_t item = 0;; ++item) {
          const FaItem w = item_of(b);
          const int tok0 = w.batch * seq, tokk0 = w.batch * seq_k;
          const uint32_t nx = item & 1;
          // K of a step before V of the step before: that is the order in which the issuer needs them
          for (int j = 0; j <= w.n; ++j) {
            if (j == w.n) {
              // Ask for the next pair as late as its operands allow: a pair taken over early is not there for a CTA that
              // runs out of work first (2048 x 32/8 x 128: 48 us asked for at the start of a pair, 35 us here).
              FA_WAIT(&bars->next_empty[nx], ((item >> 1) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
              pb::mbar_expect_tx(&bars->next_full[nx], 16);
              pb::clc_try_cancel(&bars->next[nx], &bars->next_full[nx]);
            } else {
              const uint32_t ks = kc % C::KS;
              FA_WAIT(&bars->k_empty[ks], ((kc / C::KS) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
              ++kc;
              pb::mbar_expect_tx(&bars->k_full[ks], C::K_BYTES);
#pragma unroll
              for (int a = 0; a < DQK / 64; ++a)
                pb::tma_load_3d(k_smem + ks * C::K_BYTES + a * ATOM_BYTES, &tmK, &bars->k_full[ks], a * 64, w.kv_head,
                                tokk0 + (j + w.j_lo) * BKV);
            }
            if (j == 0) {
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                if (w.nb[t] == 0) continue;
                FA_WAIT(&bars->q_empty[t], (qc[t] & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
                ++qc[t];
                pb::mbar_expect_tx(&bars->q_full[t], C::Q_BYTES);
#pragma unroll
                for (int a = 0; a < DQK / 64; ++a)
                  pb::tma_load_3d(q_smem + t * C::Q_BYTES + a * ATOM_BYTES, &tmQ, &bars->q_full[t], a * 64, w.head,
                                  tok0 + (w.qt0 + t) * BQ);
              }
            } else {
              const uint32_t vs = vc % C::VS;
              FA_WAIT(&bars->v_empty[vs], ((vc / C::VS) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
              ++vc;
              pb::mbar_expect_tx(&bars->v_full[vs], C::V_BYTES);
#pragma unroll
              for (int a = 0; a < DV / 64; ++a)
                pb::tma_load_3d(v_smem + vs * C::V_BYTES + a * ATOM_BYTES, &tmV, &bars->v_full[vs], a * 64, w.kv_head,
                                tokk0 + (j - 1 + w.j_lo) * BKV);
            }
          }
          FA_WAIT(&bars->next_full[nx], (item >> 1) & 1, PB_ERR_TIMEOUT_TMA);
          if (!pb::clc_taken(&bars->next[nx], b)) return true;
        }
      }();
    } else if (warp == 1 && pb::elect_one()) {
      // ------------------------------------------------------------------ issuer of S = Q K^T
      [&]() -> bool {
        constexpr uint32_t idesc = pb::make_idesc_bf16(BQ, BKV, 0, 0);
        uint32_t s_count = 0, kc = 0, qc[2] = {0, 0};  // S, K blocks and Q tiles so far
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        for (uint32_t item = 0;; ++item) {
          const FaItem w = item_of(b);
          for (int j = 0; j < w.n; ++j, ++kc) {
            const uint32_t ks = kc % C::KS;
            FA_WAIT(&bars->k_full[ks], (kc / C::KS) & 1, PB_ERR_TIMEOUT_MMA);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (!w.has(t, j)) continue;
              if (j == w.lo[t]) {
                FA_WAIT(&bars->q_full[t], qc[t] & 1, PB_ERR_TIMEOUT_MMA);
                ++qc[t];
              }
              FA_WAIT(&bars->s_read, (s_count & 1) ^ 1, PB_ERR_TIMEOUT_MMA);    // the S before this one
              ++s_count;
              pb::tc_fence_after();
              const uint32_t qa = pb::smem_u32(q_smem + t * C::Q_BYTES), ka = pb::smem_u32(k_smem + ks * C::K_BYTES);
#pragma unroll
              for (int k = 0; k < DQK / 16; ++k) {
                const uint32_t off = (k / 4) * ATOM_BYTES + (k % 4) * 32;
                pb::umma_f16_ss(tmem_base, pb::make_smem_desc(qa + off, 0, 1024, 2), pb::make_smem_desc(ka + off, 0, 1024, 2),
                                idesc, k > 0 ? 1u : 0u);
              }
              pb::umma_commit(&bars->s_full[t]);
              if (t == 1 || !w.has(1, j)) pb::umma_commit(&bars->k_empty[ks]);
              if (C::STAGE && j == w.nb[t] - 1) pb::umma_commit(&bars->q_empty[t]);
            }
          }
          if (!next_item(item, b)) return true;
        }
      }();
    } else if (warp == 2 && pb::elect_one()) {
      // ------------------------------------------------------------------ issuer of O += P V
      [&]() -> bool {
        constexpr uint32_t idesc = pb::make_idesc_bf16(BQ, DV, 0, 1);
        uint32_t vc = 0, pc[2] = {0, 0}, oc[2] = {0, 0};   // V blocks so far; per tile: products, finished outputs
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        for (uint32_t item = 0;; ++item) {
          const FaItem w = item_of(b);
          for (int j = 0; j < w.n; ++j, ++vc) {
            const uint32_t vs = vc % C::VS;
            FA_WAIT(&bars->v_full[vs], (vc / C::VS) & 1, PB_ERR_TIMEOUT_MMA);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (!w.has(t, j)) continue;
              if (j == w.lo[t]) {                      // overwrites the output of the pair before
                FA_WAIT(&bars->o_free[t], (oc[t] & 1) ^ 1, PB_ERR_TIMEOUT_MMA);
                ++oc[t];
              }
              FA_WAIT(&bars->p_full[t], pc[t] & 1, PB_ERR_TIMEOUT_MMA);
              ++pc[t];
              pb::tc_fence_after();
              const uint32_t va = pb::smem_u32(v_smem + vs * C::V_BYTES);
#pragma unroll
              for (int k = 0; k < BKV / 16; ++k)       // P_t: packed bf16, 8 columns per 16-wide k step
                pb::umma_f16_ts(tmem_base + O_COL + t * 128, tmem_base + P_COL + t * 64 + k * 8,
                                pb::make_smem_desc(va + k * 2048, ATOM_BYTES, 1024, 2), idesc, (j > w.lo[t] || k > 0) ? 1u : 0u);
              pb::umma_commit(&bars->pv_done[t]);
              if (t == 1 || !w.has(1, j)) pb::umma_commit(&bars->v_empty[vs]);
            }
          }
          if (!next_item(item, b)) return true;
        }
      }();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FA_REGS_SOFTMAX));
    // ------------------------------------------------------------------ softmax + epilogue
    [&]() -> bool {
      const int t = (warp - 4) >> 2;  // tile / warpgroup
      const int wq = warp & 3;
      const int row = wq * 32 + lane;
      const uint32_t lane_addr = uint32_t(wq * 32) << 16;
      const uint32_t t_s = tmem_base + lane_addr;
      const uint32_t t_p = tmem_base + lane_addr + P_COL + t * 64;
      const uint32_t t_o = tmem_base + lane_addr + O_COL + t * 128;
      const bool leader = (threadIdx.x & 127) == 0;
      const uint64_t scale2 = pb::pack_f32x2(scale_log2, scale_log2);
      int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
      uint32_t count = 0;                       // blocks of this tile so far
      for (uint32_t item = 0;; ++item) {
        const FaItem w = item_of(b);
        const int qk = w.qt0 + t + q_off_blocks;
        float m_ref = -1e30f;
        float l = 0.f;
        const int j0 = t == 0 ? w.lo[0] : w.lo[1], j1 = t == 0 ? w.nb[0] : w.nb[1];
        for (int j = j0; j < j1; ++j, ++count) {
          FA_WAIT(&bars->s_full[t], count & 1, PB_ERR_TIMEOUT_EPILOGUE);
          pb::tc_fence_after();
          const bool diag = causal && (j + w.j_lo == qk);
          // keys of this block older than the window of this row: columns [0, lim)
          const int lim = (window > 0) ? qk * BQ + row - window + 1 - (j + w.j_lo) * BKV : 0;
          const bool edge = __any_sync(0xffffffffu, lim > 0);
          // the whole S row (128 fp32) is read once and stays in registers for both passes
          uint32_t sr[128];
#pragma unroll
          for (int c = 0; c < 4; ++c) pb::tmem_ld_32x32b_x32(t_s + c * 32, sr + c * 32);
          pb::tmem_wait_ld();
          pb::tc_fence_before();
          __syncwarp();
          if (lane == 0) pb::mbar_arrive(&bars->s_read);
          if (WIN && softcap > 0.f) {
            // keep the later `s * scale_log2` form: store softcap * tanh(scale * s / softcap) / scale
            const float scale = scale_log2 * 0.6931471805599453f;
            const float a = scale / softcap, b = softcap / scale;
#pragma unroll
            for (int i = 0; i < 128; ++i) sr[i] = __float_as_uint(b * pb::fast_tanh(__uint_as_float(sr[i]) * a));
          }
          if (diag) {
#pragma unroll
            for (int i = 0; i < 128; ++i)
              if (i > row) sr[i] = 0xff800000u;  // -inf: masked out of max and exp
          }
          if (edge) {
#pragma unroll
            for (int i = 0; i < 128; ++i)
              if (i < lim) sr[i] = 0xff800000u;
          }
          // pass 1: row maximum (four independent chains)
          float mx4[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
          for (int i = 0; i < 128; i += 8) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
              mx4[u] = fmaxf(mx4[u], fmaxf(__uint_as_float(sr[i + u]), __uint_as_float(sr[i + 4 + u])));
          }
          const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
          const float m_new = fmaxf(m_ref, mx * scale_log2);
          const bool grow = m_new > m_ref + 8.f;
          const bool any = __any_sync(0xffffffffu, grow);
          if (any) {
            const float alpha = exp2f(m_ref - m_new);
            m_ref = m_new;
            l *= alpha;
            if (j > j0) {
              FA_WAIT(&bars->pv_done[t], (count - 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
              pb::tc_fence_after();
#pragma unroll 1
              for (int c = 0; c < DV / 32; ++c) {
                uint32_t r[32];
                pb::tmem_ld_32x32b_x32(t_o + c * 32, r);
                pb::tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                pb::tmem_st_32x32b_x32(t_o + c * 32, r);
              }
            }
          }
          // pass 2: P = exp2(S * scale - m) as packed bf16
          if (j > j0) {                          // P is free again
            FA_WAIT(&bars->pv_done[t], (count - 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
            pb::tc_fence_after();
          }
          const uint64_t neg_m = pb::pack_f32x2(-m_ref, -m_ref);
          // (row sums as scalars: packed additions are 1.5 % faster and, in another order, differ in the last bit)
          float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float e0, e1;
              pb::unpack_f32x2(pb::fma_f32x2(pb::pack_f32x2(__uint_as_float(sr[c * 32 + 2 * i]),
                                                            __uint_as_float(sr[c * 32 + 2 * i + 1])), scale2, neg_m), e0, e1);
              e0 = pb::fast_exp2(e0);
              e1 = pb::fast_exp2(e1);
              l4[i & 3] += e0 + e1;
              pk[i] = pb::pack_bf16x2(e0, e1);
            }
            pb::tmem_st_32x32b_x16(t_p + c * 16, pk);
          }
          l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
          pb::tmem_wait_st();
          pb::tc_fence_before();
          __syncwarp();
          if (lane == 0) pb::mbar_arrive(&bars->p_full[t]);   // 128 arrivals on one mbarrier would serialise
        }
        // epilogue: O / l -> bf16 -> shared -> TMA store; log-sum-exp
        if (j1 > 0) {
          float l_scale = 1.f;
          if (sinks != nullptr) {   // the sink joins the denominator only
            const float s2 = sinks[w.head] * 1.4426950408889634f;
            const float m_fin = fmaxf(m_ref, s2);
            const float a = exp2f(m_ref - m_fin);
            l = l * a + exp2f(s2 - m_fin);
            l_scale = a;
            m_ref = m_fin;
          }
          const float inv = l_scale / l;
          lse[((long)w.batch * hq + w.head) * seq + (w.qt0 + t) * BQ + row] = (m_ref + log2f(l)) * 0.6931471805599453f;
          FA_WAIT(&bars->pv_done[t], (count - 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
          pb::tc_fence_after();
          uint8_t* stage = C::STAGE ? o_smem + t * ATOM_BYTES : q_smem + t * C::Q_BYTES;
#pragma unroll
          for (int a = 0; a < DV / 64; ++a) {
            uint32_t r[64];
            pb::tmem_ld_32x32b_x32(t_o + a * 64, r);
            pb::tmem_ld_32x32b_x32(t_o + a * 64 + 32, r + 32);
            pb::tmem_wait_ld();
            if (a == DV / 64 - 1) {
              pb::tc_fence_before();
              __syncwarp();
              if (lane == 0) pb::mbar_arrive(&bars->o_free[t]);
            }
            if (C::STAGE) {                      // the tile before has left the staging buffer
              if (leader) pb::tma_store_wait_read<0>();
              pb::named_bar_sync(1 + t, 128);
            }
            uint8_t* atom = stage + (C::STAGE ? 0 : a * ATOM_BYTES);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              uint4 v;
              v.x = pb::pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
              v.y = pb::pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
              v.z = pb::pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
              v.w = pb::pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
              *reinterpret_cast<uint4*>(atom + row * 128 + ((i ^ (row & 7)) << 4)) = v;
            }
            pb::fence_proxy_async_smem();
            pb::named_bar_sync(1 + t, 128);
            if (leader) {
              pb::tma_store_3d(&tmO, atom, a * 64, w.head, w.batch * seq + (w.qt0 + t) * BQ);
              pb::tma_store_commit();
            }
          }
          if (!C::STAGE && leader) {             // the tile of Q is free for the next pair
            pb::tma_store_wait_read<0>();
            pb::mbar_arrive(&bars->q_empty[t]);
          }
        }
        if (!next_item(item, b)) break;
      }
      if (leader) pb::tma_store_wait_all<0>();
      return true;
    }();
  }

  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  pb::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    pb::tc_fence_after();
    pb::tmem_dealloc<1>(tmem_base, 512);
  }
}

template <int DQK, int DV>
int launch_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int batch, int seq, int seq_k,
               int q_off, int hq, int hkv, long q_row, long k_row, long v_row, long o_row, float scale, int causal,
               int window, const float* sinks, float softcap, int* status, cudaStream_t stream) {
  using C = FaCfg<DQK, DV>;
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  const long T = (long)batch * seq;
  const long TK = (long)batch * seq_k;
  CUtensorMap tq, tk, tv, to;
  int rc;
  if ((rc = pbh::make_tmap_3d(&tq, q, bf, 2, T, hq, DQK, DQK, q_row, BQ, 1, 64, sw))) return rc;
  if ((rc = pbh::make_tmap_3d(&tk, k, bf, 2, TK, hkv, DQK, DQK, k_row, BKV, 1, 64, sw))) return rc;
  if ((rc = pbh::make_tmap_3d(&tv, v, bf, 2, TK, hkv, DV, DV, v_row, BKV, 1, 64, sw))) return rc;
  if ((rc = pbh::make_tmap_3d(&to, o, bf, 2, T, hq, DV, DV, o_row, BQ, 1, 64, sw))) return rc;
  const bool win = window > 0 || sinks != nullptr || softcap > 0.f;
  auto kern = win ? flash_attn_fwd_kernel<DQK, DV, true> : flash_attn_fwd_kernel<DQK, DV, false>;
  static std::atomic<bool> allowed[2][pbh::MAX_DEVICES];
  if ((rc = pbh::allow_shared_memory(kern, C::SMEM_BYTES, allowed[win]))) return rc;
  dim3 grid(hq, batch, (seq / BQ + 1) / 2);
  pbh::launch_dependent(kern, grid, FA_THREADS, C::SMEM_BYTES, stream, tq, tk, tv, to, lse, seq, seq_k, q_off / BQ, hq, hkv,
      scale * 1.4426950408889634f, causal, window, sinks, softcap, status);
  return (int)cudaGetLastError();
}

}  // namespace

// q: [batch*seq, hq, d_qk] (row pitch q_row elements, heads contiguous), k: [batch*seq_k, hkv, d_qk],
// v: [batch*seq_k, hkv, d_v], o: [batch*seq, hq, d_v]; lse: [batch, hq, seq] fp32 (natural log).  seq, seq_k and q_off
// are multiples of 128.  Query row i of a sequence sits at key position q_off + i: with `causal` it attends to keys
// [0, q_off + i] (the last `window` of them when window > 0) and q_off + seq must equal seq_k (the layout of a
// sequence chunk attending to the gathered prefix).  sinks: null or one fp32 logit per query head.
extern "C" int pb_flash_attn_fwd_cap(const void* q, const void* k, const void* v, void* o, float* lse, int batch,
                                     int seq, int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row,
                                     long k_row, long v_row, long o_row, float scale, int causal, int window,
                                     const float* sinks, float softcap, int* status, cudaStream_t stream) {
  if (seq % 128 || seq_k % 128 || q_off % 128 || q_off < 0 || hq % hkv || (q_row % 8) || (k_row % 8) || (v_row % 8) ||
      (o_row % 8))
    return -2;
  if (causal ? (q_off + seq != seq_k) : (q_off != 0)) return -2;
  if (window < 0 || (window > 0 && (!causal || q_off != 0)) || softcap < 0.f) return -2;
  if (batch > MAX_GRID_Y) {                    // (sequences are the grid's second dimension)
    for (int b = 0; b < batch; b += MAX_GRID_Y) {
      const long tq = (long)b * seq, tk = (long)b * seq_k;
      auto at = [](const void* p, long rows, long pitch) { return static_cast<const __nv_bfloat16*>(p) + rows * pitch; };
      const int rc = pb_flash_attn_fwd_cap(at(q, tq, q_row), at(k, tk, k_row), at(v, tk, v_row),
                                           const_cast<__nv_bfloat16*>(at(o, tq, o_row)), lse + tq * hq,
                                           batch - b < MAX_GRID_Y ? batch - b : MAX_GRID_Y, seq, seq_k, q_off, hq, hkv, d_qk, d_v,
                                           q_row, k_row, v_row, o_row, scale, causal, window, sinks, softcap, status, stream);
      if (rc) return rc;
    }
    return 0;
  }
  if (d_qk == 128 && d_v == 128)
    return launch_fwd<128, 128>(q, k, v, o, lse, batch, seq, seq_k, q_off, hq, hkv, q_row, k_row, v_row, o_row, scale,
                                causal, window, sinks, softcap, status, stream);
  if (d_qk == 192 && d_v == 128)
    return launch_fwd<192, 128>(q, k, v, o, lse, batch, seq, seq_k, q_off, hq, hkv, q_row, k_row, v_row, o_row, scale,
                                causal, window, sinks, softcap, status, stream);
  if (d_qk == 64 && d_v == 64)
    return launch_fwd<64, 64>(q, k, v, o, lse, batch, seq, seq_k, q_off, hq, hkv, q_row, k_row, v_row, o_row, scale,
                              causal, window, sinks, softcap, status, stream);
  return -3;
}

// No logit soft-capping.
extern "C" int pb_flash_attn_fwd_win(const void* q, const void* k, const void* v, void* o, float* lse, int batch,
                                     int seq, int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row,
                                     long k_row, long v_row, long o_row, float scale, int causal, int window,
                                     const float* sinks, int* status, cudaStream_t stream) {
  return pb_flash_attn_fwd_cap(q, k, v, o, lse, batch, seq, seq_k, q_off, hq, hkv, d_qk, d_v, q_row, k_row, v_row, o_row,
                               scale, causal, window, sinks, 0.f, status, stream);
}

// No sliding window, no sinks.
extern "C" int pb_flash_attn_fwd_ex(const void* q, const void* k, const void* v, void* o, float* lse, int batch,
                                    int seq, int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row,
                                    long k_row, long v_row, long o_row, float scale, int causal, int* status,
                                    cudaStream_t stream) {
  return pb_flash_attn_fwd_win(q, k, v, o, lse, batch, seq, seq_k, q_off, hq, hkv, d_qk, d_v, q_row, k_row, v_row, o_row,
                               scale, causal, 0, nullptr, status, stream);
}

// Self-attention form: seq_k = seq, q_off = 0.
extern "C" int pb_flash_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int batch,
                                 int seq, int hq, int hkv, int d_qk, int d_v, long q_row, long k_row, long v_row,
                                 long o_row, float scale, int causal, int* status, cudaStream_t stream) {
  return pb_flash_attn_fwd_ex(q, k, v, o, lse, batch, seq, seq, 0, hq, hkv, d_qk, d_v, q_row, k_row, v_row, o_row,
                              scale, causal, status, stream);
}
