// Flash-attention backward for sm_100a: two passes that share all plumbing.
//   MODE_DKDV: a CTA owns 128 KV rows of one KV head (resident tiles X1 = K, X2 = V) and streams
//              tiles of Q / dO (Y1, Y2) of every query head of the group;
//              S^T = K Q^T, dP^T = V dO^T  ->  P^T, dS^T  ->  dV += P^T dO,  dK += dS^T Q.
//   MODE_DQ  : a CTA owns 128 query rows of one head (X1 = Q, X2 = dO) and streams tiles of
//              K / V;  S = Q K^T, dP = dO V^T  ->  dS  ->  dQ += dS K.
// Where the blocks are few or uneven, the CTAs of a cluster share a block's steps and add up their sums over distributed
// shared memory, in the order of their ranks (bwd_cluster_size).
// In both the accumulators live in tensor memory for the whole loop (no atomics, results are
// bit-reproducible), and the streamed tiles are used twice from one shared-memory copy (K-major operand for
// the first GEMM, MN-major operand for the second).  The softmax threads turn S / dP into bf16 P / dS *in tensor
// memory*, 8 packed columns per 16 values, and the second GEMM takes its A operand from there (`tcgen05.mma` with A in
// TMEM), one 16-wide K step per column group.  Nothing but mbarriers goes through shared memory between the two GEMMs of
// a step.
//   flash_attn_bwd_wide_kernel  128-row steps: both passes of the heads with d_qk == d_v, the dQ pass of the multi-latent
//                               head shape (d_qk 192, d_v 128).
//   flash_attn_bwd_kernel       64-row steps: the dK / dV pass of the multi-latent shape, whose accumulators leave too little
//                               tensor memory for wider ones.  Two teams of 256 softmax threads work on alternating
//                               steps while the MMA thread runs ahead.
//
// Replaces the backward of `flash_attn_func` (primus/backends/megatron/core/extensions/
// primus_turbo.py:812-823); deterministic by construction (cf. the `deterministic=` flag there, :805).
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BR = 128;  // resident rows
constexpr int BC = 64;   // streamed rows per step
constexpr int BW_THREADS = 576;   // warp0 TMA, warp1 MMA, warps 2..17: two softmax teams of 256 threads
constexpr int BW_COMPUTE = 512;
constexpr int BW_TEAMS = 2;       // team t handles steps i = t (mod 2): two threads per resident row, 32 columns each
constexpr int BW_HALF = BC / 2;   // streamed columns of a step per softmax thread
constexpr int XATOM = 128 * 128;  // bytes of a [128 rows x 64 bf16] atom
constexpr int YATOM = 64 * 128;   // bytes of a [64 rows x 64 bf16] atom
enum { MODE_DKDV = 0, MODE_DQ = 1 };

template <int DQK, int DV>
struct BwCfg {
  static constexpr int ACC_COLS = DQK + DV;
  // Next to the accumulators there is room for three 64-column buffers: two of S and one of dP.  P and dS are both packed
  // into the step's S columns (8 + 8 of every 16), so the dP buffer is free again as soon as the softmax threads have *read*
  // it, and the S / dP GEMMs of a step run under the softmax of the step before instead of after it.
  static constexpr int DP_COL = 2 * BC;                  // dP columns of the region behind the accumulators
  static_assert(ACC_COLS + 3 * BC <= 512, "tensor memory");
  static constexpr int X1_BYTES = BR * DQK * 2;
  static constexpr int X2_BYTES = BR * DV * 2;
  static constexpr int Y1_BYTES = BC * DQK * 2;
  static constexpr int Y2_BYTES = BC * DV * 2;
  static constexpr int STAT_BYTES = 512;  // 64 lse + 64 delta
  static constexpr int FIXED_BYTES = X1_BYTES + X2_BYTES + 1024 + 512;
  static constexpr int STAGE_BYTES = Y1_BYTES + Y2_BYTES + STAT_BYTES;
  static constexpr int NS_FIT = (232448 - FIXED_BYTES) / STAGE_BYTES;
  // streamed-tile ring depth: a stage is held from the first GEMM (S/dP) to the last (dK/dQ) of its
  // step, so at least three stages are needed to keep a load in flight behind the running step
  static constexpr int NS = NS_FIT >= 4 ? 4 : (NS_FIT >= 3 ? 3 : 2);
  static constexpr int SMEM_BYTES = FIXED_BYTES + NS * STAGE_BYTES;
  static_assert(ACC_COLS * 4 * BR <= FIXED_BYTES - 1536 + NS * (Y1_BYTES + Y2_BYTES), "sums of a shared block");
};

struct BwBars {
  uint64_t x_full;
  uint64_t y_full[4], y_empty[4];
  uint64_t s_full[2];  // per team
  uint64_t p_ready[2]; // per team: P / dS of its current step are in tensor memory (one arrival per warp)
  uint64_t acc_done;   // all MMAs of the CTA have completed
  uint64_t dp_free;    // the softmax threads hold the step's dP in registers (one arrival per warp of the team)
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ bool bw_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (pb::mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!pb::mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > PB_WAIT_CYCLES) return false;
  }
  return true;
}
#define BW_WAIT(bar, parity, code)             \
  if (!bw_wait((bar), (parity), abort_flag)) { \
    atomicCAS(status, 0, (code));              \
    bars->abort_flag = 1;                      \
    ok = false;                                \
    break;                                     \
  }

__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          pb::smem_u32(smem_dst)),
      "l"(gsrc), "r"(bytes), "r"(pb::smem_u32(bar))
      : "memory");
}

// What a launch adds for blocks whose steps are shared by the CTAs of a cluster: the outputs as plain pointers.
struct BwOut {
  __nv_bfloat16 *p1, *p2;
  long ld1, ld2;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// Accumulators of a block whose steps were shared by the CTAs of a cluster: every CTA has left its fp32 sums in its shared
// memory ([128 rows][C1 + C2], 16-byte chunks of a row XORed with row & 7); this CTA adds up a share of the rows, always in
// the order of the ranks, and stores them.
template <int C1, int C2>
__device__ __forceinline__ void cluster_sum_rows(const uint8_t* stage, int rank, int csize, int tid, int nthreads, long row0,
                                                 int head, const BwOut& out, float mul1) {
  constexpr int GROUPS = (C1 + C2) / 8;
  const int rows = BR / csize;
  for (int it = tid; it < rows * GROUPS; it += nthreads) {
    const int row = rank * rows + it / GROUPS, grp = it % GROUPS;
    const uint32_t off = row * (C1 + C2) * 4;
    const uint32_t o0 = off + (((2 * grp) ^ (row & 7)) << 4), o1 = off + (((2 * grp + 1) ^ (row & 7)) << 4);
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll 4
    for (int p = 0; p < csize; ++p) {
      const uint32_t base = pb::mapa_shared(stage, p);
      const float4 a = ld_cluster_f4(base + o0), b = ld_cluster_f4(base + o1);
      acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
      acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
    }
    const bool first = grp < C1 / 8;
    const float mul = first ? mul1 : 1.f;
    __nv_bfloat16* dst = first ? out.p1 + (row0 + row) * out.ld1 + (long)head * C1 + grp * 8
                               : out.p2 + (row0 + row) * out.ld2 + (long)head * C2 + (grp - C1 / 8) * 8;
    *reinterpret_cast<uint4*>(dst) =
        make_uint4(pb::pack_bf16x2(acc[0] * mul, acc[1] * mul), pb::pack_bf16x2(acc[2] * mul, acc[3] * mul),
                   pb::pack_bf16x2(acc[4] * mul, acc[5] * mul), pb::pack_bf16x2(acc[6] * mul, acc[7] * mul));
  }
}
// 32 columns of a row of the staging layout above
__device__ __forceinline__ void stage_row_chunk(uint8_t* stage, int row_bytes, int row, int c32, const uint32_t* r) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<uint4*>(stage + row * row_bytes + (((c32 * 8 + q) ^ (row & 7)) << 4)) =
        make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
}

template <int DQK, int DV, bool WIN>
__global__ void __launch_bounds__(BW_THREADS, 1)
flash_attn_bwd_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                      const __grid_constant__ CUtensorMap tmY1, const __grid_constant__ CUtensorMap tmY2,
                      const __grid_constant__ CUtensorMap tmO1, const __grid_constant__ CUtensorMap tmO2,
                      const float* __restrict__ lse, const float* __restrict__ delta, int seq, int seq_k, int q_off,
                      int hq, int hkv, float scale, int causal, int window_arg, float softcap_arg, const BwOut out, int* status) {
  const int window = WIN ? window_arg : 0;   // the instantiation without a window carries no code for it
  // softcap > 0: scores were softcap * tanh(scale * s / softcap) in the forward pass
  const float softcap = WIN ? softcap_arg : 0.f;
  const float cap_a = (WIN && softcap > 0.f) ? scale / softcap : 0.f;
  const float cap_b = (WIN && softcap > 0.f) ? softcap / scale : 0.f;
  // seq: query rows per sequence, seq_k: key rows per sequence, q_off: key position of query row 0 (multiple of 128);
  // window > 0 (causal self-attention only): a query sees its last `window` keys, itself included
  using C = BwCfg<DQK, DV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x1_smem = smem;
  uint8_t* x2_smem = x1_smem + C::X1_BYTES;
  uint8_t* y1_smem = x2_smem + C::X2_BYTES;           // NS stages
  uint8_t* y2_smem = y1_smem + C::NS * C::Y1_BYTES;   // NS stages
  float* stat_smem = reinterpret_cast<float*>(y2_smem + C::NS * C::Y2_BYTES);  // NS stages x (64 lse, 64 delta)
  BwBars* bars = reinterpret_cast<BwBars*>(reinterpret_cast<uint8_t*>(stat_smem) + C::NS * C::STAT_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = hq / hkv;
  const int num_c = seq / BC;
  const int qo = q_off / BC;                              // offset in streamed-tile units
  // grid (heads * batch, row blocks): blocks are issued x-fastest, so all heads of the longest row block start
  // first and the short ones fill the tail (work per block is proportional to the number of streamed tiles)
  const int rb = blockIdx.y;
  const int csize = pb::cluster_nctarank(), rank = pb::cluster_ctarank();   // CTAs that share the block's steps
  const int xhead = (blockIdx.x / csize) % hkv;
  const int batch = blockIdx.x / csize / hkv;
  const int tok0 = batch * seq_k;
  const int toky0 = batch * seq;
  // streamed-tile schedule: the query tiles at or after this key block (query row i sits at key position q_off + i)
  const int c_start = causal ? max(0, 2 * rb - qo) : 0;
  const int c_end = window > 0 ? min(num_c, (rb * BR + BR - 1 + window - 1 - q_off) / BC + 1) : num_c;
  const int n_per_head = max(0, c_end - c_start);
  const int i0 = g * n_per_head * rank / csize;           // first step of this CTA
  const int n_iter = g * n_per_head * (rank + 1) / csize - i0;
  volatile int* abort_flag = &bars->abort_flag;
  const float sl2 = scale * 1.4426950408889634f;

  if (threadIdx.x == 0) {
    pb::mbar_init(&bars->x_full, 1);
    for (int i = 0; i < 4; ++i) {
      pb::mbar_init(&bars->y_full[i], 1);
      pb::mbar_init(&bars->y_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) pb::mbar_init(&bars->s_full[i], 1);
    for (int i = 0; i < 2; ++i) pb::mbar_init(&bars->p_ready[i], BW_COMPUTE / BW_TEAMS / 32);
    pb::mbar_init(&bars->acc_done, 1);
    pb::mbar_init(&bars->dp_free, BW_COMPUTE / BW_TEAMS / 32);
    bars->abort_flag = 0;
    pb::fence_barrier_init();
  }
  if (warp == 1) {
    pb::tmem_alloc<1>(&bars->tmem_base, 512);
    pb::tmem_relinquish<1>();
  }
  pb::tc_fence_before();
  __syncthreads();
  PB_GRID_WAIT();
  pb::grid_release();           // the dQ pass behind (see flash_attn_bwd_wide_kernel)
  pb::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  const uint32_t tmem_sbuf = tmem_base + C::ACC_COLS;  // [S 64][S 64][dP 64]

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (pb::elect_one()) {
      bool ok = true;
      pb::mbar_expect_tx(&bars->x_full, C::X1_BYTES + C::X2_BYTES);
#pragma unroll
      for (int a = 0; a < DQK / 64; ++a)
        pb::tma_load_3d(x1_smem + a * XATOM, &tmX1, &bars->x_full, a * 64, xhead, tok0 + rb * BR);
#pragma unroll
      for (int a = 0; a < DV / 64; ++a)
        pb::tma_load_3d(x2_smem + a * XATOM, &tmX2, &bars->x_full, a * 64, xhead, tok0 + rb * BR);
      for (int i = 0; i < n_iter && ok; ++i) {
        const int st = i % C::NS;
        const int yhead = xhead * g + (i0 + i) / n_per_head;
        const int cs = c_start + (i0 + i) % n_per_head;
        BW_WAIT(&bars->y_empty[st], ((i / C::NS) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
        pb::mbar_expect_tx(&bars->y_full[st], C::STAGE_BYTES);
#pragma unroll
        for (int a = 0; a < DQK / 64; ++a)
          pb::tma_load_3d(y1_smem + st * C::Y1_BYTES + a * YATOM, &tmY1, &bars->y_full[st], a * 64, yhead,
                          toky0 + cs * BC);
#pragma unroll
        for (int a = 0; a < DV / 64; ++a)
          pb::tma_load_3d(y2_smem + st * C::Y2_BYTES + a * YATOM, &tmY2, &bars->y_full[st], a * 64, yhead,
                          toky0 + cs * BC);
        const long off = ((long)batch * hq + yhead) * seq + cs * BC;
        bulk_load_1d(stat_smem + st * 128, lse + off, 256, &bars->y_full[st]);
        bulk_load_1d(stat_smem + st * 128 + 64, delta + off, 256, &bars->y_full[st]);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (pb::elect_one()) {
      constexpr uint32_t idesc_s = pb::make_idesc_bf16(BR, BC, 0, 0);
      constexpr uint32_t idesc_a1 = pb::make_idesc_bf16(BR, DQK, 0, 1);  // acc(DQK) += dS . Y1
      constexpr uint32_t idesc_a2 = pb::make_idesc_bf16(BR, DV, 0, 1);   // acc(DV)  += P  . Y2
      const uint32_t x1a = pb::smem_u32(x1_smem), x2a = pb::smem_u32(x2_smem);
      bool ok = true;
      auto s_cols = [&](int i) { return tmem_sbuf + (i & 1) * BC; };
      auto issue_s = [&](int i) {
        const uint32_t y1a = pb::smem_u32(y1_smem + (i % C::NS) * C::Y1_BYTES);
#pragma unroll
        for (int k = 0; k < DQK / 16; ++k)
          pb::umma_f16_ss(s_cols(i), pb::make_smem_desc(x1a + (k / 4) * XATOM + (k % 4) * 32, 0, 1024, 2),
                          pb::make_smem_desc(y1a + (k / 4) * YATOM + (k % 4) * 32, 0, 1024, 2), idesc_s, k > 0 ? 1u : 0u);
      };
      auto issue_dp = [&](int i) {
        const uint32_t y2a = pb::smem_u32(y2_smem + (i % C::NS) * C::Y2_BYTES);
#pragma unroll
        for (int k = 0; k < DV / 16; ++k)
          pb::umma_f16_ss(tmem_sbuf + C::DP_COL, pb::make_smem_desc(x2a + (k / 4) * XATOM + (k % 4) * 32, 0, 1024, 2),
                          pb::make_smem_desc(y2a + (k / 4) * YATOM + (k % 4) * 32, 0, 1024, 2), idesc_s, k > 0 ? 1u : 0u);
      };
      // S runs two steps ahead of the second GEMMs, dP one.  S of step i + 2 reuses the columns of step i; it is issued
      // after the second GEMMs of step i (same thread: the tensor pipe keeps the order), which themselves wait for the
      // softmax threads to have replaced S of step i by P / dS.
      do {
        if (n_iter == 0) break;
        BW_WAIT(&bars->x_full, 0, PB_ERR_TIMEOUT_MMA);
        for (int j = 0; j < 2 && j < n_iter && ok; ++j) {
          BW_WAIT(&bars->y_full[j % C::NS], (j / C::NS) & 1, PB_ERR_TIMEOUT_MMA);
          pb::tc_fence_after();
          issue_s(j);
          if (j == 0) {
            issue_dp(0);
            pb::umma_commit(&bars->s_full[0]);
          }
        }
      } while (false);
      for (int i = 0; i < n_iter && ok; ++i) {
        const int st = i % C::NS;
        if (i + 1 < n_iter) {                 // S of step i + 1 is already on its way
          BW_WAIT(&bars->dp_free, i & 1, PB_ERR_TIMEOUT_MMA);
          pb::tc_fence_after();
          issue_dp(i + 1);
          pb::umma_commit(&bars->s_full[(i + 1) & 1]);
        }
        BW_WAIT(&bars->p_ready[i & 1], (i >> 1) & 1, PB_ERR_TIMEOUT_MMA);
        pb::tc_fence_after();
        const uint32_t y1a = pb::smem_u32(y1_smem + st * C::Y1_BYTES);
        const uint32_t y2a = pb::smem_u32(y2_smem + st * C::Y2_BYTES);
        const uint32_t ts = s_cols(i);
#pragma unroll
        for (int k = 0; k < BC / 16; ++k)     // acc(DV) += P . Y2, A = packed P of K step k (TMEM columns 16k .. 16k+7)
          pb::umma_f16_ts(tmem_base + DQK, ts + 16 * k, pb::make_smem_desc(y2a + k * 2048, YATOM, 1024, 2), idesc_a2,
                          (i > 0 || k > 0) ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < BC / 16; ++k)     // acc(DQK) += dS . Y1
          pb::umma_f16_ts(tmem_base, ts + 8 + 16 * k, pb::make_smem_desc(y1a + k * 2048, YATOM, 1024, 2), idesc_a1,
                          (i > 0 || k > 0) ? 1u : 0u);
        pb::umma_commit(&bars->y_empty[st]);
        const int in = i + 2;
        if (in < n_iter) {
          BW_WAIT(&bars->y_full[in % C::NS], (in / C::NS) & 1, PB_ERR_TIMEOUT_MMA);
          pb::tc_fence_after();
          issue_s(in);
        }
      }
      if (ok) pb::umma_commit(&bars->acc_done);
    }
  } else {
    // ------------------------------------------------------------------ softmax-gradient threads
    const int wq = warp & 3;              // TMEM lane quarter of this warp
    const int team = (warp - 2) >> 3;     // 0 / 1: even / odd steps
    const int half = ((warp - 2) >> 2) & 1;   // which 32 of a step's 64 columns
    const int row = wq * 32 + lane;
    const uint32_t lane_addr = uint32_t(wq * 32) << 16;
    const int row_g = rb * BR + row;
    bool ok = true;
    int cs = n_iter > team ? c_start + (i0 + team) % n_per_head : 0;    // tile of the step, advanced at the end of the loop
    for (int i = team; i < n_iter && ok; i += BW_TEAMS) {
      const int st = i % C::NS;
      BW_WAIT(&bars->s_full[i & 1], (i >> 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
      BW_WAIT(&bars->y_full[st], (i / C::NS) & 1, PB_ERR_TIMEOUT_EPILOGUE);  // lse / delta tile visible
      pb::tc_fence_after();
      const uint32_t ts = tmem_sbuf + lane_addr + (i & 1) * BC + half * BW_HALF;
      const uint32_t tdp = tmem_sbuf + lane_addr + C::DP_COL + half * BW_HALF;
      const int cs_rel = cs + qo;   // streamed tile index in the stationary block's frame
      // largest (query position - key position) inside this tile pair: beyond the window -> element-wise mask
      const int max_diff = cs_rel * BC + BC - 1 - rb * BR;
      const bool diag = (causal && (cs_rel >= 2 * rb) && (cs_rel <= 2 * rb + 1)) || (window > 0 && max_diff >= window);
      const float* st_lse = stat_smem + st * 128 + half * BW_HALF;
      const float* st_delta = st_lse + 64;
      uint32_t s[BW_HALF], dp[BW_HALF];
      pb::tmem_ld_32x32b_x32(ts, s);
      pb::tmem_ld_32x32b_x32(tdp, dp);
      pb::tmem_wait_ld();
      pb::tc_fence_before();
      __syncwarp();
      if (lane == 0) pb::mbar_arrive(&bars->dp_free);
      auto body = [&](auto diag_tag) {
        constexpr bool DIAG = decltype(diag_tag)::value;
#pragma unroll
        for (int kk = 0; kk < BW_HALF / 16; ++kk) {   // one 16-wide K step of the second GEMM at a time
          uint32_t pk[8], dsk[8];
#pragma unroll
          for (int e4 = 0; e4 < 16; e4 += 4) {
            const int c = kk * 16 + e4;
            const float4 l4 = *reinterpret_cast<const float4*>(st_lse + c);
            const float4 d4 = *reinterpret_cast<const float4*>(st_delta + c);
            const float l2[4] = {l4.x, l4.y, l4.z, l4.w}, dl[4] = {d4.x, d4.y, d4.z, d4.w};
            float pv[4], dv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float sv = __uint_as_float(s[c + u]);
              float dcap = 1.f;
              if (WIN && softcap > 0.f) {
                const float t = pb::fast_tanh(sv * cap_a);
                sv = t * cap_b;                  // = softcap * tanh(scale * s / softcap) / scale
                dcap = 1.f - t * t;              // derivative of the capped score with respect to scale * s
              }
              float p = pb::fast_exp2(fmaf(sv, sl2, l2[u]));   // (lse is stored negated)
              if (DIAG) {
                const int col_g = cs_rel * BC + half * BW_HALF + c + u;
                const int diff = col_g - row_g;   // query - key position
                if (diff < 0 || (window > 0 && diff >= window)) p = 0.f;
              }
              pv[u] = p;
              dv[u] = p * (__uint_as_float(dp[c + u]) - dl[u]) * scale * dcap;
            }
            pk[e4 / 2] = pb::pack_bf16x2(pv[0], pv[1]);
            pk[e4 / 2 + 1] = pb::pack_bf16x2(pv[2], pv[3]);
            dsk[e4 / 2] = pb::pack_bf16x2(dv[0], dv[1]);
            dsk[e4 / 2 + 1] = pb::pack_bf16x2(dv[2], dv[3]);
          }
          // P and dS (bf16 pairs) replace the 16 S columns of this K step
          pb::tmem_st_32x32b_x8(ts + 16 * kk, pk);
          pb::tmem_st_32x32b_x8(ts + 8 + 16 * kk, dsk);
        }
      };
      if (diag) body(std::true_type{}); else body(std::false_type{});
      pb::tmem_wait_st();
      pb::tc_fence_before();
      __syncwarp();
      if (lane == 0) pb::mbar_arrive(&bars->p_ready[i & 1]);   // one arrival per warp
      cs += BW_TEAMS;
      while (cs >= c_start + n_per_head) cs -= n_per_head;
    }
    // ---- epilogue: accumulators -> bf16 -> (dead) resident tiles -> TMA store
    do {
      if (!ok) break;
      BW_WAIT(&bars->acc_done, 0, PB_ERR_TIMEOUT_EPILOGUE);
      BW_WAIT(&bars->x_full, 0, PB_ERR_TIMEOUT_EPILOGUE);     // (long past, except for a CTA without a step)
      pb::tc_fence_after();
      auto drain = [&](uint32_t tcol, int ncols, uint8_t* dst) {
#pragma unroll 1
        for (int c = 2 * team + half; c < ncols / 32; c += 4) {
          uint32_t r[32];
          pb::tmem_ld_32x32b_x32(tmem_base + lane_addr + tcol + c * 32, r);
          pb::tmem_wait_ld();
          if (n_iter == 0) {                      // nothing was accumulated: the columns are undefined
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = 0u;
          }
          if (pb::cluster_nctarank() > 1) {
            stage_row_chunk(smem, (DQK + DV) * 4, row, tcol / 32 + c, r);
            continue;
          }
          uint8_t* atom = dst + (c >> 1) * XATOM + row * 128;
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 v;
            v.x = pb::pack_bf16x2(__uint_as_float(r[8 * q4 + 0]), __uint_as_float(r[8 * q4 + 1]));
            v.y = pb::pack_bf16x2(__uint_as_float(r[8 * q4 + 2]), __uint_as_float(r[8 * q4 + 3]));
            v.z = pb::pack_bf16x2(__uint_as_float(r[8 * q4 + 4]), __uint_as_float(r[8 * q4 + 5]));
            v.w = pb::pack_bf16x2(__uint_as_float(r[8 * q4 + 6]), __uint_as_float(r[8 * q4 + 7]));
            const int chunk = (c & 1) * 4 + q4;
            *reinterpret_cast<uint4*>(atom + ((chunk ^ (row & 7)) << 4)) = v;
          }
        }
      };
      drain(0, DQK, x1_smem);
      drain(DQK, DV, x2_smem);
      if (pb::cluster_nctarank() > 1) break;
      pb::fence_proxy_async_smem();
      pb::named_bar_sync(1, BW_COMPUTE);
      if (threadIdx.x == 64) {
#pragma unroll
        for (int a = 0; a < DQK / 64; ++a)
          pb::tma_store_3d(&tmO1, x1_smem + a * XATOM, a * 64, xhead, tok0 + rb * BR);
#pragma unroll
        for (int a = 0; a < DV / 64; ++a)
          pb::tma_store_3d(&tmO2, x2_smem + a * XATOM, a * 64, xhead, tok0 + rb * BR);
        pb::tma_store_commit();
        pb::tma_store_wait_all<0>();
      }
    } while (false);
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
  if (pb::cluster_nctarank() > 1) {
    pb::cluster_sync();
    cluster_sum_rows<DQK, DV>(smem, pb::cluster_ctarank(), pb::cluster_nctarank(), threadIdx.x, BW_THREADS, tok0 + (long)rb * BR, xhead, out, 1.f);
    pb::cluster_sync();       // this CTA's sums may be read until here
  }
}

// ------------------------------------------------------------------------------------------------
// 128-wide steps, for d_qk == d_v (64, 128) and the dQ pass of (192, 128).  A tcgen05.mma with N = 64 occupies the tensor pipe for
// three quarters of the time of one with N = 128 (48 and 64 clocks), so the 64-row steps above pay half as much again for S and
// dP; and there the two second GEMMs of a step run only after its whole softmax.  Here a step streams 128 rows, and its work is
// cut so that the tensor pipe always has some of it:
//   * the softmax threads take P = exp2(S) as soon as S is there, before dP;
//   * dS and the second GEMMs go by column halves A (64 columns) and B: the GEMMs of half A run while half B is computed;
//   * what frees a tensor-memory region is the *read* of it.  With two S buffers (64-wide heads) P and dS are packed into
//     the step's S columns (8 + 8 of every 16) and the next dP starts as soon as this one is in registers; with one S
//     buffer (128-wide) they are packed into the dP columns and the next S starts instead.
// The two streamed tiles of a step have rings of their own, NS1 and NS2 buffers of 128 rows: the tile of S is wanted a whole step
// before the tile of dP, and the dQ pass is done with V after dP.  In the dQ pass of 128-wide heads the resident tiles (Q, dO)
// move to tensor memory at the start of a block, as A operands of the first GEMMs; their shared memory then stages the outputs.
// A step of 128 x 128 x 128 holds four GEMMs of 512 clocks each in the dK / dV pass, three in the dQ pass; the passes take 2750
// and 1960 clocks per step (3600 and 2600 with one ring of two or three buffers for both tiles: S waited for its tile).  8192 x
// 32/8 x 128: dK / dV pass 924 -> 800 us; 4096 x 16 x 192/128: dQ pass 119 -> 103 us.  Tensor pipe busy 72 % of the time in the
// dK / dV pass at 4096 x 32/8 x 128, 68 % in the dQ pass (57 and 52 with one ring).
//
// The CTAs are persistent where the heads have d_qk == d_v: one takes the next block from the hardware scheduler
// (clusterlaunchcontrol.try_cancel, so that the longest blocks still start first) and loads its tiles, and issues its first
// GEMMs, while the sums of this block leave.  A CTA of a cluster that shares a block, and the multi-latent shape, whose resident
// tile fills the shared memory, have one block.  dQ pass, one block per CTA -> persistent, us: window of 128 at 2 x 2048 x
// 64/8 x 64 98 -> 59 (start and end were 8500 of 11600 clocks), 2048 x 32/8 x 128 54 -> 47, 8192 x 32/8 x 128 603 -> 590.
//   warp 0 scheduler and TMA producer; warp 1 issues the MMAs; warp 2 stores the outputs; warps 4..19 softmax and gradients
template <int DQK, int DV, int MODE>
struct BwWideCfg {
  static constexpr int BCW = 128;
  static constexpr bool PERSIST = DQK == DV;
  static constexpr int ACC_COLS = (MODE == MODE_DKDV) ? DQK + DV : DQK;
  static constexpr int NSB = DQK == 64 ? 2 : 1;                        // S buffers
  static constexpr bool XA1 = MODE == MODE_DQ && DQK == 128;           // X1 (Q) in tensor memory
  static constexpr bool XA2 = MODE == MODE_DQ && DV == 128;            // X2 (dO) in tensor memory
  static constexpr int S_COL = ACC_COLS;
  static constexpr int DP_COL = ACC_COLS + NSB * BCW;
  static constexpr int XA1_COL = DP_COL + BCW;
  static constexpr int XA2_COL = XA1_COL + (XA1 ? DQK / 2 : 0);
  static constexpr int T1_BYTES = BR * DQK * 2;                        // a [128, DQK] tile (X1, Y1)
  static constexpr int T2_BYTES = BR * DV * 2;                         // a [128, DV] tile (X2, Y2)
  static constexpr int STAT = MODE == MODE_DKDV ? 128 : 0;             // statistics of a tile: lse with Y1, delta with Y2
  static constexpr int NX = DQK == 64 ? 2 : 1;                         // buffers of the resident tiles
  // X2 of the multi-latent dQ pass goes to tensor memory by way of the V buffer
  static constexpr bool X2_IN_RING = !PERSIST && XA2;
  static constexpr int X_BYTES = T1_BYTES + (X2_IN_RING ? 0 : T2_BYTES);
  static constexpr int NS1 = DQK == 64 ? 4 : 3;
  static constexpr int NS2 = DQK == 64 ? 4 : DQK == 128 ? 2 : 1;
  static constexpr int TILE_BYTES = NX * X_BYTES + NS1 * T1_BYTES + NS2 * T2_BYTES;
  static constexpr int SMEM_BYTES = TILE_BYTES + (NS1 + NS2) * STAT * 4 + 512;
  static_assert(SMEM_BYTES <= 232448, "shared memory");
  static_assert(ACC_COLS * 4 * BR <= TILE_BYTES, "sums of a shared block");
  static_assert(XA2_COL + (XA2 ? DV / 2 : 0) <= 512, "tensor memory");
};
constexpr int BWW_WARPS = 16;                       // softmax warps: thread = one resident row x 16 columns of each half
constexpr int BWW_THREADS = 128 + 32 * BWW_WARPS;
// registers move from warps 0..3 to the softmax warps: 64 + 4 * 104 = 5 * 96 per lane of a scheduler
constexpr int BWW_REGS_AUX = 64, BWW_REGS_SOFTMAX = 104;

struct BwWideBars {
  uint4 next[2];           // answers of try_cancel, by block parity
  uint64_t next_full[2], next_empty[2];
  uint64_t x_full[2], x_empty[2];
  uint64_t y1_full[4], y2_full[4];
  uint64_t s_full[2];
  uint64_t dp_full[4], done[4];   // by step: dP is there; all products of the step are.  They release the streamed tiles too
  uint64_t freed;          // the softmax threads hold S (one S buffer) or dP (two) of the step in registers
  uint64_t pa[2], pb[2];   // P / dS of half A / B are in tensor memory; by step parity, because with two S buffers a warp can
                           // be a step ahead of another
  uint64_t acc_done;       // all products of the block are there
  uint64_t acc_free;       // and have been read
  uint64_t out_ready;      // the outputs are in shared memory
  uint64_t xa_ready;       // resident tiles copied into tensor memory
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(BwWideBars) <= 512, "barriers");

// one look at a barrier, without waiting
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(pb::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// in a role's lambda: a wait that runs out ends the role
#define BWW_WAIT(bar, parity, code)            \
  if (!bw_wait((bar), (parity), abort_flag)) { \
    atomicCAS(status, 0, (code));              \
    bars->abort_flag = 1;                      \
    return false;                              \
  }

// VAR: 0 plain, 1 sliding window, 2 soft-capped scores (with or without a window); a variant carries no code of a later one
template <int DQK, int DV, int MODE, int VAR>
__global__ void __launch_bounds__(BWW_THREADS, 1)
flash_attn_bwd_wide_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                           const __grid_constant__ CUtensorMap tmY1, const __grid_constant__ CUtensorMap tmY2,
                           const __grid_constant__ CUtensorMap tmO1, const __grid_constant__ CUtensorMap tmO2,
                           const float* __restrict__ lse, const float* __restrict__ delta, int seq, int seq_k, int q_off,
                           int hq, int hkv, float scale, int causal, int window_arg, float softcap_arg, const BwOut out,
                           int* status) {
  using C = BwWideCfg<DQK, DV, MODE>;
  constexpr int BCW = C::BCW;
  constexpr bool CAP = VAR == 2;
  const int window = VAR ? window_arg : 0;
  const float cap_a = CAP ? scale / softcap_arg : 0.f;
  const float cap_b = CAP ? softcap_arg / scale : 0.f;
  extern __shared__ __align__(1024) uint8_t smem_wide[];
  uint8_t* smem = smem_wide;
  uint8_t* y1_smem = smem + C::NX * C::X_BYTES;
  uint8_t* y2_smem = y1_smem + C::NS1 * C::T1_BYTES;
  auto x1_smem = [&](uint32_t slot) { return smem + slot * C::X_BYTES; };
  auto x2_smem = [&](uint32_t slot) { return C::X2_IN_RING ? y2_smem + (C::NS2 - 1) * C::T2_BYTES : smem + slot * C::X_BYTES + C::T1_BYTES; };
  float* lse_smem = reinterpret_cast<float*>(y2_smem + C::NS2 * C::T2_BYTES);
  float* delta_smem = lse_smem + C::NS1 * C::STAT;
  BwWideBars* bars = reinterpret_cast<BwWideBars*>(delta_smem + C::NS2 * C::STAT);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = hq / hkv;
  const int seq_x = (MODE == MODE_DKDV) ? seq_k : seq;
  const int seq_y = (MODE == MODE_DKDV) ? seq : seq_k;
  const int num_rb = seq_x / BR;
  const int num_c = seq_y / BCW;
  const int qo = q_off / BCW;
  const bool shared_block = pb::cluster_nctarank() > 1;    // the CTAs of the cluster share the steps of one block
  const bool one_block = !C::PERSIST || shared_block;
  struct Block {
    int rb, xhead, batch;
    int c_start, n_per_head;    // streamed tiles of a query head
    int i0, n;                  // first step of this CTA and its number of steps
  };
  // grid (heads * cluster, batch, row blocks): longest row blocks first, as in the kernel above, and no division to find one
  auto block_of = [&](int3 b) {
    Block w;
    const int csize = pb::cluster_nctarank(), rank = pb::cluster_ctarank();
    w.rb = (MODE == MODE_DKDV) ? b.z : (num_rb - 1 - b.z);
    w.xhead = b.x >> (__ffs(csize) - 1);                          // (csize is a power of two)
    w.batch = b.y;
    w.c_start = (MODE == MODE_DKDV) ? (causal ? max(0, w.rb - qo) : 0)
                                    : (window > 0 ? max(0, w.rb * BR + q_off - window + 1) / BCW : 0);
    const int c_end = (MODE == MODE_DKDV)
                          ? (window > 0 ? min(num_c, (w.rb * BR + BR - 1 + window - 1 - q_off) / BCW + 1) : num_c)
                          : (causal ? min(num_c, w.rb + 1 + qo) : num_c);
    w.n_per_head = max(0, c_end - w.c_start);
    const int n_all = (MODE == MODE_DKDV) ? g * w.n_per_head : w.n_per_head;
    w.i0 = (n_all * rank) >> (__ffs(csize) - 1);
    w.n = ((n_all * (rank + 1)) >> (__ffs(csize) - 1)) - w.i0;
    return w;
  };
  volatile int* abort_flag = &bars->abort_flag;
  const float sl2 = scale * 1.4426950408889634f;
  // the block after block `item` of this CTA: waits for the scheduler's answer; false: there is none
  auto next_block = [&](uint32_t item, int3& b) -> bool {
    if (one_block) return false;
    const uint32_t nx = item & 1;
    BWW_WAIT(&bars->next_full[nx], (item >> 1) & 1, PB_ERR_TIMEOUT_MMA);
    return pb::clc_taken(&bars->next[nx], b);
  };
  auto next_seen = [&](uint32_t item) {
    pb::fence_proxy_async_smem();
    pb::mbar_arrive(&bars->next_empty[item & 1]);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      pb::mbar_init(&bars->next_full[i], 1);
      pb::mbar_init(&bars->next_empty[i], 2 + BWW_WARPS);   // issuer, store and softmax warps
      pb::mbar_init(&bars->x_full[i], 1);
      pb::mbar_init(&bars->x_empty[i], 1);
      pb::mbar_init(&bars->s_full[i], 1);
      pb::mbar_init(&bars->pa[i], BWW_WARPS);
      pb::mbar_init(&bars->pb[i], BWW_WARPS);
    }
    for (int i = 0; i < 4; ++i) {
      pb::mbar_init(&bars->y1_full[i], 1);
      pb::mbar_init(&bars->y2_full[i], 1);
      pb::mbar_init(&bars->dp_full[i], 1);
      pb::mbar_init(&bars->done[i], 1);
    }
    pb::mbar_init(&bars->freed, BWW_WARPS);
    pb::mbar_init(&bars->acc_done, 1);
    pb::mbar_init(&bars->acc_free, BWW_WARPS);
    pb::mbar_init(&bars->out_ready, BWW_WARPS);
    pb::mbar_init(&bars->xa_ready, BWW_WARPS);
    bars->abort_flag = 0;
    pb::fence_barrier_init();
  }
  if (warp == 1) {
    pb::tmem_alloc<1>(&bars->tmem_base, 512);
    pb::tmem_relinquish<1>();
  }
  pb::tc_fence_before();
  __syncthreads();
  // The dQ pass needs nothing of the dK / dV pass in front of it, only what that one has waited for: its CTAs start where that one
  // has no blocks left, and wait before they end, so that their end stands for both.  us without and with: 2 x 2048 tokens, 64 / 8
  // heads of 64, window 128, 184 -> 175; 8192 x 32 / 8 x 128 2059 -> 2027; 4096 x 32 / 4 x 128 564 -> 556; 4096 x 16 x 192 / 128
  // 340 -> 336; 4 x 1024 of these 156 -> 148 (forward and backward).
  if (MODE == MODE_DKDV) {
    PB_GRID_WAIT();
    pb::grid_release();
  }
  pb::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(BWW_REGS_AUX));
    if (warp == 0 && pb::elect_one()) {
      // ------------------------------------------------------------------ scheduler and producer
      [&]() -> bool {
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        uint32_t u0 = 0;                               // steps of the blocks before
        for (uint32_t item = 0;; ++item) {
          const Block w = block_of(b);
          const int tok0 = w.batch * seq_x, toky0 = w.batch * seq_y;
          auto load_x = [&]() -> bool {
            const uint32_t slot = item % C::NX;
            if (C::XA1) {                              // free once copied, and the outputs of the block before have left it
              if (item == 1) BWW_WAIT(&bars->xa_ready, 0, PB_ERR_TIMEOUT_TMA);
              if (item >= 2) BWW_WAIT(&bars->x_empty[0], item & 1, PB_ERR_TIMEOUT_TMA);
            } else if (item >= C::NX) {                // free when the outputs of the block that had it have left it
              BWW_WAIT(&bars->x_empty[slot], ((item / C::NX) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
            }
            pb::mbar_expect_tx(&bars->x_full[slot], C::T1_BYTES + C::T2_BYTES);
#pragma unroll
            for (int a = 0; a < DQK / 64; ++a)
              pb::tma_load_3d(x1_smem(slot) + a * XATOM, &tmX1, &bars->x_full[slot], a * 64, w.xhead, tok0 + w.rb * BR);
#pragma unroll
            for (int a = 0; a < DV / 64; ++a)
              pb::tma_load_3d(x2_smem(slot) + a * XATOM, &tmX2, &bars->x_full[slot], a * 64, w.xhead, tok0 + w.rb * BR);
            return true;
          };
          auto load_y1 = [&](int i) -> bool {
            const uint32_t u = u0 + i, st = u % C::NS1, rel = u - C::NS1;     // rel: the step that had the buffer
            if (u >= C::NS1) BWW_WAIT(&bars->done[rel & 3], (rel >> 2) & 1, PB_ERR_TIMEOUT_TMA);
            pb::mbar_expect_tx(&bars->y1_full[st], C::T1_BYTES + C::STAT * 4);
            const int yhead = (MODE == MODE_DKDV) ? (w.xhead * g + (w.i0 + i) / w.n_per_head) : (w.xhead / g);
            const int row = (w.c_start + (w.i0 + i) % w.n_per_head) * BCW;
#pragma unroll
            for (int a = 0; a < DQK / 64; ++a)
              pb::tma_load_3d(y1_smem + st * C::T1_BYTES + a * XATOM, &tmY1, &bars->y1_full[st], a * 64, yhead, toky0 + row);
            if (MODE == MODE_DKDV)
              bulk_load_1d(lse_smem + st * C::STAT, lse + ((long)w.batch * hq + yhead) * seq + row, 512, &bars->y1_full[st]);
            return true;
          };
          auto load_y2 = [&](int i) -> bool {
            const uint32_t u = u0 + i, st = u % C::NS2, rel = u - C::NS2;
            if (C::X2_IN_RING && u == C::NS2 - 1) BWW_WAIT(&bars->xa_ready, 0, PB_ERR_TIMEOUT_TMA);
            // the dQ pass is done with V after dP
            if (u >= C::NS2)
              BWW_WAIT(MODE == MODE_DKDV ? &bars->done[rel & 3] : &bars->dp_full[rel & 3], (rel >> 2) & 1, PB_ERR_TIMEOUT_TMA);
            pb::mbar_expect_tx(&bars->y2_full[st], C::T2_BYTES + C::STAT * 4);
            const int yhead = (MODE == MODE_DKDV) ? (w.xhead * g + (w.i0 + i) / w.n_per_head) : (w.xhead / g);
            const int row = (w.c_start + (w.i0 + i) % w.n_per_head) * BCW;
#pragma unroll
            for (int a = 0; a < DV / 64; ++a)
              pb::tma_load_3d(y2_smem + st * C::T2_BYTES + a * XATOM, &tmY2, &bars->y2_full[st], a * 64, yhead, toky0 + row);
            if (MODE == MODE_DKDV)
              bulk_load_1d(delta_smem + st * C::STAT, delta + ((long)w.batch * hq + yhead) * seq + row, 512,
                           &bars->y2_full[st]);
            return true;
          };
          // a resident tile whose buffer waits for the outputs of the block before does not hold up the streamed ones
          constexpr bool X_LAST = C::PERSIST && C::NX == 1 && !C::XA1;
          if (!X_LAST && !load_x()) return false;
          if (w.n > 0 && !load_y1(0)) return false;
          if (X_LAST && w.n > 0 && !load_y2(0)) return false;
          if (X_LAST && !load_x()) return false;
          for (int i = 0; i < w.n; ++i) {      // in the order in which they are wanted and their buffers are free
            if (C::NS2 == 1 && i + 1 < w.n && !load_y1(i + 1)) return false;
            if (!(X_LAST && i == 0) && !load_y2(i)) return false;
            if (C::NS2 != 1 && i + 1 < w.n && !load_y1(i + 1)) return false;
          }
          if (one_block) return true;
          u0 += w.n;
          // ask for the next block as late as its loads allow: one taken over early is not there for a CTA that runs out first
          const uint32_t nx = item & 1;
          BWW_WAIT(&bars->next_empty[nx], ((item >> 1) & 1) ^ 1, PB_ERR_TIMEOUT_TMA);
          pb::mbar_expect_tx(&bars->next_full[nx], 16);
          pb::clc_try_cancel(&bars->next[nx], &bars->next_full[nx]);
          if (!next_block(item, b)) return true;
        }
      }();
    } else if (warp == 1 && pb::elect_one()) {
      // ------------------------------------------------------------------ MMA issuer
      [&]() -> bool {
        constexpr uint32_t idesc_s = pb::make_idesc_bf16(BR, BCW, 0, 0);
        constexpr uint32_t idesc_a1 = pb::make_idesc_bf16(BR, DQK, 0, 1);  // acc(DQK) += dS . Y1
        constexpr uint32_t idesc_a2 = pb::make_idesc_bf16(BR, DV, 0, 1);   // acc(DV)  += P  . Y2
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        uint32_t u = 0;                                // step, counted over all blocks
        for (uint32_t item = 0;; ++item) {
          const int n = block_of(b).n;
          const uint32_t slot = item % C::NX;
          const uint32_t x1a = pb::smem_u32(x1_smem(slot)), x2a = pb::smem_u32(x2_smem(slot));
          // X . Y^T -> 128 columns, X from shared or from tensor memory
          auto issue_first = [&](auto dim, auto from_tmem, uint32_t tcol, uint32_t xa, uint32_t xt, uint32_t ya) {
#pragma unroll
            for (int k = 0; k < decltype(dim)::value / 16; ++k) {
              const uint32_t off = (k / 4) * XATOM + (k % 4) * 32;
              const uint64_t db = pb::make_smem_desc(ya + off, 0, 1024, 2);
              if (decltype(from_tmem)::value)
                pb::umma_f16_ts(tmem_base + tcol, tmem_base + xt + 8 * k, db, idesc_s, k > 0 ? 1u : 0u);
              else
                pb::umma_f16_ss(tmem_base + tcol, pb::make_smem_desc(xa + off, 0, 1024, 2), db, idesc_s, k > 0 ? 1u : 0u);
            }
          };
          auto issue_s = [&](uint32_t v) {
            pb::tc_fence_after();
            issue_first(std::integral_constant<int, DQK>{}, std::bool_constant<C::XA1>{},
                        C::S_COL + (C::NSB == 2 ? (v & 1) * BCW : 0), x1a, C::XA1_COL,
                        pb::smem_u32(y1_smem + (v % C::NS1) * C::T1_BYTES));
            pb::umma_commit(&bars->s_full[C::NSB == 2 ? (v & 1) : 0]);
          };
          auto issue_dp = [&](uint32_t v) -> bool {
            BWW_WAIT(&bars->y2_full[v % C::NS2], (v / C::NS2) & 1, PB_ERR_TIMEOUT_MMA);
            pb::tc_fence_after();
            issue_first(std::integral_constant<int, DV>{}, std::bool_constant<C::XA2>{}, C::DP_COL, x2a, C::XA2_COL,
                        pb::smem_u32(y2_smem + (v % C::NS2) * C::T2_BYTES));
            pb::umma_commit(&bars->dp_full[v & 3]);
            return true;
          };
          auto issue_second = [&](int i, int half) {                       // accumulators += (P, dS of the half) . Y
            pb::tc_fence_after();
            const uint32_t y1a = pb::smem_u32(y1_smem + (u % C::NS1) * C::T1_BYTES);
            const uint32_t y2a = pb::smem_u32(y2_smem + (u % C::NS2) * C::T2_BYTES);
            const uint32_t tp = tmem_base + (C::NSB == 2 ? C::S_COL + (u & 1) * BCW : C::DP_COL);
            if (MODE == MODE_DKDV) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                const int k = half * 4 + kk;
                pb::umma_f16_ts(tmem_base + DQK, tp + 16 * k, pb::make_smem_desc(y2a + k * 2048, XATOM, 1024, 2), idesc_a2,
                                (i > 0 || k > 0) ? 1u : 0u);
              }
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const int k = half * 4 + kk;
              pb::umma_f16_ts(tmem_base, tp + 16 * k + 8, pb::make_smem_desc(y1a + k * 2048, XATOM, 1024, 2), idesc_a1,
                              (i > 0 || k > 0) ? 1u : 0u);
            }
          };
          auto y1_there = [&](uint32_t v) { return mbar_test(&bars->y1_full[v % C::NS1], (v / C::NS1) & 1); };
          // the first GEMMs of the block: the products of the block before have been issued, its last S and dP been read
          if (C::XA1 || C::XA2) BWW_WAIT(&bars->xa_ready, item & 1, PB_ERR_TIMEOUT_MMA);
          if (!C::XA1) BWW_WAIT(&bars->x_full[slot], (item / C::NX) & 1, PB_ERR_TIMEOUT_MMA);
          if (n > 0) {
            BWW_WAIT(&bars->y1_full[u % C::NS1], (u / C::NS1) & 1, PB_ERR_TIMEOUT_MMA);
            issue_s(u);
            if (!issue_dp(u)) return false;
            if (C::NSB == 2 && n > 1) {
              BWW_WAIT(&bars->y1_full[(u + 1) % C::NS1], ((u + 1) / C::NS1) & 1, PB_ERR_TIMEOUT_MMA);
              issue_s(u + 1);
            }
          }
          for (int i = 0; i < n; ++i, ++u) {
            // S of the next step (one S buffer) goes out at the first point at which its tile has arrived: the issuing thread
            // must not wait for a load while P / dS of this step are ready
            bool s_next = C::NSB == 2 || i + 1 >= n;
            auto try_s = [&]() {
              if (!s_next && y1_there(u + 1)) {
                issue_s(u + 1);
                s_next = true;
              }
            };
            BWW_WAIT(&bars->freed, u & 1, PB_ERR_TIMEOUT_MMA);
            if (i + 1 < n) {
              if (C::NSB == 2 && !issue_dp(u + 1)) return false;
              try_s();
            }
            if (i == 0 && item > 0) BWW_WAIT(&bars->acc_free, (item - 1) & 1, PB_ERR_TIMEOUT_MMA);
            BWW_WAIT(&bars->pa[u & 1], (u >> 1) & 1, PB_ERR_TIMEOUT_MMA);
            issue_second(i, 0);
            try_s();
            BWW_WAIT(&bars->pb[u & 1], (u >> 1) & 1, PB_ERR_TIMEOUT_MMA);
            issue_second(i, 1);
            pb::umma_commit(&bars->done[u & 3]);
            if (C::NSB == 1) {
              if (!s_next) {
                BWW_WAIT(&bars->y1_full[(u + 1) % C::NS1], ((u + 1) / C::NS1) & 1, PB_ERR_TIMEOUT_MMA);
                issue_s(u + 1);
              }
              if (i + 1 < n && !issue_dp(u + 1)) return false;
            } else if (i + 2 < n) {
              BWW_WAIT(&bars->y1_full[(u + 2) % C::NS1], ((u + 2) / C::NS1) & 1, PB_ERR_TIMEOUT_MMA);
              issue_s(u + 2);
            }
          }
          pb::umma_commit(&bars->acc_done);
          if (!next_block(item, b)) return true;
          next_seen(item);
        }
      }();
    } else if (warp == 2 && !shared_block && pb::elect_one()) {
      // ------------------------------------------------------------------ outputs: shared -> global
      [&]() -> bool {
        int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
        for (uint32_t item = 0;; ++item) {
          const Block w = block_of(b);
          const uint32_t slot = item % C::NX;
          const int row = w.batch * seq_x + w.rb * BR;
          BWW_WAIT(&bars->out_ready, item & 1, PB_ERR_TIMEOUT_EPILOGUE);
#pragma unroll
          for (int a = 0; a < DQK / 64; ++a) pb::tma_store_3d(&tmO1, x1_smem(slot) + a * XATOM, a * 64, w.xhead, row);
          if (MODE == MODE_DKDV) {
#pragma unroll
            for (int a = 0; a < DV / 64; ++a) pb::tma_store_3d(&tmO2, x2_smem(slot) + a * XATOM, a * 64, w.xhead, row);
          }
          pb::tma_store_commit();
          pb::tma_store_wait_read<0>();
          pb::mbar_arrive(&bars->x_empty[slot]);
          if (!next_block(item, b)) break;
          next_seen(item);
        }
        pb::tma_store_wait_all<0>();
        return true;
      }();
    }
    __syncwarp();
    if (shared_block) {      // (in both branches: what follows them may use no more registers than these warps have)
      pb::cluster_sync();
      pb::cluster_sync();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(BWW_REGS_SOFTMAX));
    // ------------------------------------------------------------------ softmax-gradient threads
    [&]() -> bool {
      const int wq = warp & 3;                      // TMEM lane quarter of this warp
      const int qd = (warp - 4) >> 2;               // 16-column group of each half
      const int row = wq * 32 + lane;
      const uint32_t lane_addr = uint32_t(wq * 32) << 16;
      const uint64_t sl2_2 = pb::pack_f32x2(sl2, sl2), minus_one = pb::pack_f32x2(-1.f, -1.f);
      // a thread copies 64 channels of its row of Q (groups 0, 1) or dO (groups 2, 3; 0, 1 when Q stays) from the
      // 128-byte-swizzled tile: word w of a row (elements 2w, 2w + 1) goes to column w, the layout of a TMEM A operand
      auto copy_x = [&](uint32_t item) -> bool {
        BWW_WAIT(&bars->x_full[0], item & 1, PB_ERR_TIMEOUT_EPILOGUE);
        const bool q_part = C::XA1 && qd < 2;
        if (C::XA1 || qd < 2) {
          const uint8_t* xs = (q_part ? x1_smem(0) : x2_smem(0)) + (qd & 1) * XATOM + row * 128;
          uint32_t wds[32];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(xs + ((c ^ (row & 7)) << 4));
            wds[4 * c] = v.x; wds[4 * c + 1] = v.y; wds[4 * c + 2] = v.z; wds[4 * c + 3] = v.w;
          }
          pb::tmem_st_32x32b_x32(tmem_base + lane_addr + (q_part ? C::XA1_COL : C::XA2_COL) + (qd & 1) * 32, wds);
          pb::tmem_wait_st();
        }
        pb::tc_fence_before();
        __syncwarp();
        if (lane == 0) pb::mbar_arrive(&bars->xa_ready);
        return true;
      };
      if ((C::XA1 || C::XA2) && !copy_x(0)) return false;
      int3 b = make_int3(blockIdx.x, blockIdx.y, blockIdx.z);
      uint32_t u = 0;
      float lse2_row = 0.f, delta_row = 0.f;        // of this thread's query row, for the dQ pass
      auto load_stats = [&]() {
        if (MODE == MODE_DQ) {
          const Block w = block_of(b);
          const long off = ((long)w.batch * hq + w.xhead) * seq + w.rb * BR + row;
          lse2_row = __ldcg(lse + off);  // negated, in log2 units; from L2, as this pass does not wait itself
          delta_row = __ldcg(delta + off);
        }
      };
      load_stats();
      for (uint32_t item = 0;; ++item) {
        const Block w = block_of(b);
        const int rb = w.rb, row_g = rb * BR + row, c_end = w.c_start + w.n_per_head;
        const uint64_t row_l2 = pb::pack_f32x2(lse2_row, lse2_row), row_delta = pb::pack_f32x2(delta_row, delta_row);
        int cs = w.c_start + (w.i0 > 0 && w.n > 0 ? w.i0 % w.n_per_head : 0);    // tile of the step, advanced at the end of the loop
        for (int i = 0; i < w.n; ++i, ++u) {
          if (MODE == MODE_DKDV) {
            BWW_WAIT(&bars->y1_full[u % C::NS1], (u / C::NS1) & 1, PB_ERR_TIMEOUT_EPILOGUE);  // the tile's lse is visible
          }
          const uint32_t ts = tmem_base + lane_addr + C::S_COL + (C::NSB == 2 ? (u & 1) * BCW : 0) + 16 * qd;
          const uint32_t td = tmem_base + lane_addr + C::DP_COL + 16 * qd;
          const uint32_t tout = C::NSB == 2 ? ts : td;
          const int cs_rel = (MODE == MODE_DKDV) ? cs + qo : cs - qo;   // streamed tile index in the stationary block's frame
          const int max_diff = (MODE == MODE_DKDV) ? (cs_rel * BCW + BCW - 1 - rb * BR) : (rb * BR + BR - 1 - cs_rel * BCW);
          const bool diag = (causal && cs_rel == rb) || (window > 0 && max_diff >= window);
          const float* lse_t = lse_smem + (u % C::NS1) * C::STAT + 16 * qd;
          const float* delta_t = delta_smem + (u % C::NS2) * C::STAT + 16 * qd;
          BWW_WAIT(&bars->s_full[C::NSB == 2 ? (u & 1) : 0], C::NSB == 2 ? ((u >> 1) & 1) : (u & 1), PB_ERR_TIMEOUT_EPILOGUE);
          pb::tc_fence_after();
          auto masked = [&](int e) {
            const int col_g = cs_rel * BCW + (e >> 4) * 64 + 16 * qd + (e & 15);
            const int diff = (MODE == MODE_DKDV) ? (col_g - row_g) : (row_g - col_g);   // query - key position
            return diff < 0 || (window > 0 && diff >= window);
          };
          float p[32];      // CAP: tanh(scale * s / softcap) until dP is there, so that no element needs two registers
          auto probabilities = [&](int e2, float s0, float s1) {      // p[e2], p[e2 + 1] of two scores
            uint64_t l2 = row_l2;
            if (MODE == MODE_DKDV) l2 = *reinterpret_cast<const uint64_t*>(lse_t + (e2 >> 4) * 64 + (e2 & 15));
            pb::unpack_f32x2(pb::fma_f32x2(pb::pack_f32x2(s0, s1), sl2_2, l2), p[e2], p[e2 + 1]);
            p[e2] = pb::fast_exp2(p[e2]);
            p[e2 + 1] = pb::fast_exp2(p[e2 + 1]);
          };
          {
            uint32_t sr[32];
            pb::tmem_ld_32x32b_x16(ts, sr);
            pb::tmem_ld_32x32b_x16(ts + 64, sr + 16);
            pb::tmem_wait_ld();
            if (C::NSB == 1) {
              pb::tc_fence_before();
              __syncwarp();
              if (lane == 0) pb::mbar_arrive(&bars->freed);
            }
#pragma unroll
            for (int e2 = 0; e2 < 32; e2 += 2) {
              const float s0 = __uint_as_float(sr[e2]), s1 = __uint_as_float(sr[e2 + 1]);
              if (CAP) {
                p[e2] = pb::fast_tanh(s0 * cap_a);
                p[e2 + 1] = pb::fast_tanh(s1 * cap_a);
              } else {
                probabilities(e2, s0, s1);
              }
            }
            if (!CAP && diag) {
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (masked(e)) p[e] = 0.f;
            }
          }
          BWW_WAIT(&bars->dp_full[u & 3], (u >> 2) & 1, PB_ERR_TIMEOUT_EPILOGUE);
          if (MODE == MODE_DKDV) {
            BWW_WAIT(&bars->y2_full[u % C::NS2], (u / C::NS2) & 1, PB_ERR_TIMEOUT_EPILOGUE);  // the tile's delta is visible
          }
          pb::tc_fence_after();
          uint32_t dp[32];
          pb::tmem_ld_32x32b_x16(td, dp);
          pb::tmem_ld_32x32b_x16(td + 64, dp + 16);
          pb::tmem_wait_ld();
          if (C::NSB == 2) {
            pb::tc_fence_before();
            __syncwarp();
            if (lane == 0) pb::mbar_arrive(&bars->freed);
          }
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t pk[16];                          // packed P (8), dS (8) of this thread's 16 columns
#pragma unroll
            for (int e2 = 0; e2 < 16; e2 += 2) {
              const int e = half * 16 + e2;
              float dc0 = 1.f, dc1 = 1.f;
              if (CAP) {
                // the score is softcap * tanh(scale * s / softcap) / scale; dc: its derivative with respect to scale * s
                const float t0 = p[e], t1 = p[e + 1];
                dc0 = fmaf(-t0, t0, 1.f);
                dc1 = fmaf(-t1, t1, 1.f);
                probabilities(e, t0 * cap_b, t1 * cap_b);
                if (diag) {
                  if (masked(e)) p[e] = 0.f;
                  if (masked(e + 1)) p[e + 1] = 0.f;
                }
              }
              uint64_t dl = row_delta;
              if (MODE == MODE_DKDV) dl = *reinterpret_cast<const uint64_t*>(delta_t + half * 64 + e2);
              const uint64_t pp = pb::pack_f32x2(p[e], p[e + 1]);
              // dS = P (dP - delta), times the score scale, which the epilogue applies
              uint64_t ds = pb::mul_f32x2(pp, pb::fma_f32x2(dl, minus_one, pb::pack_f32x2(__uint_as_float(dp[e]), __uint_as_float(dp[e + 1]))));
              if (CAP) ds = pb::mul_f32x2(ds, pb::pack_f32x2(dc0, dc1));
              float d0, d1;
              pb::unpack_f32x2(ds, d0, d1);
              pk[e2 / 2] = pb::pack_bf16x2(p[e], p[e + 1]);
              pk[8 + e2 / 2] = pb::pack_bf16x2(d0, d1);
            }
            if (MODE == MODE_DKDV) pb::tmem_st_32x32b_x16(tout + half * 64, pk);
            else pb::tmem_st_32x32b_x8(tout + half * 64 + 8, pk + 8);
            pb::tmem_wait_st();
            pb::tc_fence_before();
            __syncwarp();
            if (lane == 0) pb::mbar_arrive(half == 0 ? &bars->pa[u & 1] : &bars->pb[u & 1]);
          }
          if (++cs == c_end) cs = w.c_start;
        }
        // ---- the block's end: what the next one's first GEMMs wait for, then accumulators -> bf16 -> (dead) resident tiles
        const bool more = next_block(item, b);
        if (!one_block) {
          __syncwarp();
          if (lane == 0) next_seen(item);
        }
        if (more) load_stats();
        if (C::PERSIST && C::XA1 && more && !copy_x(item + 1)) return false;
        const uint32_t slot = item % C::NX;
        BWW_WAIT(&bars->acc_done, item & 1, PB_ERR_TIMEOUT_EPILOGUE);
        // the staging tiles: the resident ones have arrived (long past, except for a block without a step); with copies in
        // tensor memory, all warps have made those of the next block and the outputs of the block before have left
        if (!C::XA1) BWW_WAIT(&bars->x_full[slot], (item / C::NX) & 1, PB_ERR_TIMEOUT_EPILOGUE);
        if (C::XA1 && more) BWW_WAIT(&bars->xa_ready, (item + 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
        if (C::XA1 && item > 0) BWW_WAIT(&bars->x_empty[0], (item - 1) & 1, PB_ERR_TIMEOUT_EPILOGUE);
        pb::tc_fence_after();
        auto drain = [&](uint32_t tcol, int ncols, uint8_t* dst, float mul) {
#pragma unroll 1
          for (int c = qd; c < ncols / 32; c += 4) {
            uint32_t r[32];
            pb::tmem_ld_32x32b_x32(tmem_base + lane_addr + tcol + c * 32, r);
            pb::tmem_wait_ld();
            if (w.n == 0) {                         // nothing was accumulated: the columns are undefined
#pragma unroll
              for (int e = 0; e < 32; ++e) r[e] = 0u;
            }
            if (shared_block) {
              stage_row_chunk(smem, C::ACC_COLS * 4, row, tcol / 32 + c, r);
              continue;
            }
            uint8_t* atom = dst + (c >> 1) * XATOM + row * 128;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint32_t wd[4];
#pragma unroll
              for (int v = 0; v < 4; ++v)
                wd[v] = pb::pack_bf16x2(__uint_as_float(r[8 * q4 + 2 * v]) * mul, __uint_as_float(r[8 * q4 + 2 * v + 1]) * mul);
              const int chunk = (c & 1) * 4 + q4;
              *reinterpret_cast<uint4*>(atom + ((chunk ^ (row & 7)) << 4)) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
            }
          }
        };
        drain(0, DQK, x1_smem(slot), scale);
        if (MODE == MODE_DKDV) drain(DQK, DV, x2_smem(slot), 1.f);
        pb::tc_fence_before();
        pb::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          pb::mbar_arrive(&bars->acc_free);
          if (!shared_block) pb::mbar_arrive(&bars->out_ready);
        }
        if (!more) return true;
      }
    }();
    if (shared_block) {
      const Block w = block_of(make_int3(blockIdx.x, blockIdx.y, blockIdx.z));
      __syncwarp();
      pb::cluster_sync();
      cluster_sum_rows<DQK, MODE == MODE_DKDV ? DV : 0>(smem, pb::cluster_ctarank(), pb::cluster_nctarank(), threadIdx.x - 128,
                                                        32 * BWW_WARPS, (long)w.batch * seq_x + (long)w.rb * BR, w.xhead, out,
                                                        scale);
      __syncwarp();
      pb::cluster_sync();       // this CTA's sums may be read until here
    }
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
  if (MODE == MODE_DQ) pb::grid_wait();
}

// delta[b, h, s] = sum_d dO * O ;  neg_lse2 = -lse * log2(e) (the addend of the main kernels' exponent).
// A CTA takes 32 positions x 8 heads.  DV / 8 lanes share a (position, head) row, neighbouring rows of the same position
// are neighbours in memory, so a warp reads whole 128-byte lines; the 32 sums of a head then leave as one 128-byte line.
// What bounds it are the loads in flight: of U rows per thread, few where many CTAs share an SM (more of them fit by their registers),
// many where there are at most two CTAs per SM.  us, four rows before and now: 8192 x 32 x 128 31.5 -> 26.3, 4096 x 64 x 64 16.2 ->
// 11.8, both with two; 4096 x 16 x 128 12.2 -> 10.3, 1024 x 16 x 128 7.5 -> 6.4, with eight (with two 13.7 for the former).
constexpr int DL_POS = 32, DL_HEADS = 8, DL_THREADS = 256;
template <int DV, int U>
__global__ void __launch_bounds__(DL_THREADS)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                  const float* __restrict__ lse, float* __restrict__ delta, float* __restrict__ neg_lse2, int seq, int hq,
                  long o_row, long do_row) {
  pb::grid_release();
  PB_GRID_WAIT();
  constexpr int LANES = DV / 8;
  constexpr int GROUPS = DL_THREADS / LANES;
  constexpr int ITERS = DL_POS * DL_HEADS / GROUPS;
  __shared__ float sums[DL_HEADS][DL_POS + 1];
  const long t0 = (long)blockIdx.x * DL_POS;    // seq is a multiple of 128: the positions lie in one sequence
  const int h0 = blockIdx.y * DL_HEADS;
  const int lane = threadIdx.x % LANES, grp = threadIdx.x / LANES;
#pragma unroll 1
  for (int i0 = 0; i0 < ITERS; i0 += U) {
    uint4 x[U], y[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int item = (i0 + i) * GROUPS + grp, p = item / DL_HEADS, h = h0 + item % DL_HEADS;
      x[i] = y[i] = make_uint4(0, 0, 0, 0);
      if (h < hq) {
        x[i] = reinterpret_cast<const uint4*>(o + (t0 + p) * o_row + (long)h * DV)[lane];
        y[i] = reinterpret_cast<const uint4*>(d_o + (t0 + p) * do_row + (long)h * DV)[lane];
      }
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int item = (i0 + i) * GROUPS + grp;
      const __nv_bfloat162* xa = reinterpret_cast<const __nv_bfloat162*>(&x[i]);
      const __nv_bfloat162* ya = reinterpret_cast<const __nv_bfloat162*>(&y[i]);
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 a = __bfloat1622float2(xa[u]), c = __bfloat1622float2(ya[u]);
        s += a.x * c.x + a.y * c.y;
      }
#pragma unroll
      for (int k = LANES / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
      if (lane == 0) sums[item % DL_HEADS][item / DL_HEADS] = s;
    }
  }
  __syncthreads();
  const int h = h0 + threadIdx.x / DL_POS, p = threadIdx.x % DL_POS;
  if (h < hq) {
    const long b = t0 / seq;
    const long off = (b * hq + h) * seq + (t0 - b * seq) + p;
    delta[off] = sums[threadIdx.x / DL_POS][p];
    neg_lse2[off] = lse[off] * -1.4426950408889634f;
  }
}

// Gradient of the per-head sink logits: dsink[h] = - sum over the head's rows of exp(sink - lse) * delta (the sink has no
// value vector: it only enters through the softmax normaliser).  One CTA per head, fixed summation order.
__global__ void __launch_bounds__(1024)
attn_sink_grad_kernel(const float* __restrict__ delta, const float* __restrict__ lse, const float* __restrict__ sinks,
                      float* __restrict__ dsinks, int batch, int seq, int hq) {
  PB_GRID_WAIT();
  __shared__ float red[32];
  const int h = blockIdx.x;
  const float sink = sinks[h];
  float s = 0.f;
  for (int b = 0; b < batch; ++b) {
    const long off = ((long)b * hq + h) * seq;
    for (int i = threadIdx.x; i < seq; i += 1024) s += expf(sink - lse[off + i]) * delta[off + i];
  }
  s = pb::warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = pb::warp_sum(red[threadIdx.x]);
    if (threadIdx.x == 0) dsinks[h] = -s;
  }
}

struct BwdArgs {
  const void *d_o, *q, *k, *v, *o;
  const float* lse;
  float *delta, *neg_lse2;
  void *dq, *dk, *dv;
  int batch, seq, seq_k, q_off, window, hq, hkv;
  float softcap;
  long q_row, k_row, v_row, o_row, do_row, dq_row, dk_row, dv_row;
  float scale;
  int causal;
  int* status;
  cudaStream_t stream;
};

// How many CTAs (a cluster of 1, 2, 4 or 8) share the steps of one row block.  A pass takes the longer of its longest block
// and its mean load per SM; a block more costs `fixed` microseconds for start and end, with a cluster more for the exchange
// of the sums.  Few key / value heads leave long blocks and idle SMs: 4096 tokens, 32 query heads on 4 key / value heads of
// 128 have 128 blocks of up to 256 steps but work for 114 steps per SM.  Measured (us, cluster 1 / 2 / 4 / 8), dK / dV pass:
//   4096 x 32/4 x 128   399 / 221 / 264 / 395      1024 x 8/1 x 128   101 / 58 / 38 / 31     8192 x 1/1 x 128   104 / 62 / 56 / 123
//   8192 x 32/8 x 128   803 / 835 / 1013 / 1511    2048 x 16/2 x 64   140 / 77 / 46 / 56     window 128, 64/8 x 64  60 / 86 / 130 / 258
// dQ pass: 2048 x 32/8 x 128  49 / 97 / 202 / 459   8192 x 1/1 x 128  79 / 46 / 41 / 82.  The model below is within 15 % of
// these but for the window (36 / 61 / 142 / 378): its blocks of few steps cost more at their start and end than `fixed` says, and
// only the order of the choices is right there.  Clusters of 4 and 8 do not fit every GPC: 132 and 120 CTAs in flight on 148 SMs.
int bwd_cluster_size(int mode, int d_qk, int d_v, int batch, int seq, int seq_k, int q_off, int hq, int hkv, int causal,
                     int window) {
  const bool kv = mode == MODE_DKDV;
  const int bc = kv && d_qk != d_v ? BC : BR;             // rows of a step
  const int blocks = (kv ? seq_k : seq) / BR, tiles = (kv ? seq : seq_k) / bc;
  double total = 0.;
  int longest = 0;
  for (int rb = 0; rb < blocks; ++rb) {                   // the kernels' own step ranges
    int lo, hi;
    if (kv) {
      lo = causal ? (rb * BR - q_off) / bc : 0;
      hi = window > 0 ? (rb * BR + BR + window - 2 - q_off) / bc + 1 : tiles;
    } else {
      lo = window > 0 ? (rb * BR + q_off - window + 1) / bc : 0;
      hi = causal ? rb + 1 + q_off / bc : tiles;
    }
    lo = lo > 0 ? lo : 0;
    hi = hi < tiles ? hi : tiles;
    const int n = (hi > lo ? hi - lo : 0) * (kv ? hq / hkv : 1);
    total += n;
    longest = n > longest ? n : longest;
  }
  const double heads = (double)batch * (kv ? hkv : hq);
  const double step = d_qk == 64 ? (kv ? 1.1 : 1.) : d_qk == d_v ? (kv ? 1.55 : 1.2) : (kv ? 1.3 : 1.4);
  static const double fixed_kv[4] = {4., 9., 14., 20.}, fixed_q[4] = {3.5, 8., 11., 14.}, sms[4] = {1., 1., 0.89, 0.81};
  int best = 1;
  double t_best = 0.;
  for (int l = 0; l < 4; ++l) {
    const int c = 1 << l;
    const double fixed = (kv ? fixed_kv : fixed_q)[l];
    const double alone = (longest + c - 1) / c * step + fixed;
    const double mean = heads * (total * step + (double)blocks * c * fixed) / (sms[l] * pbh::sm_count());
    const double t = alone > mean ? alone : mean;
    if (l == 0 || t < 0.95 * t_best) {
      best = c;
      t_best = t;
    }
  }
  return best;
}

template <int DQK, int DV>
int launch_bwd(const BwdArgs& a) {
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  const long T = (long)a.batch * a.seq;
  const dim3 grid_delta((unsigned)(T / DL_POS), (a.hq + DL_HEADS - 1) / DL_HEADS);
  auto delta_kern = (long)grid_delta.x * grid_delta.y > 148 * 2 ? attn_delta_kernel<DV, 2> : attn_delta_kernel<DV, 8>;
  pbh::launch_dependent(delta_kern, grid_delta, DL_THREADS, 0, a.stream, (const __nv_bfloat16*)a.o, (const __nv_bfloat16*)a.d_o, a.lse,
                        a.delta, a.neg_lse2, a.seq, a.hq, a.o_row, a.do_row);
  int rc;
  CUtensorMap q128, do128, k128, v128, dq_m, dk_m, dv_m;
  const long TK = (long)a.batch * a.seq_k;
#define MK(m, p, rows, heads, d, row, br) \
  if ((rc = pbh::make_tmap_3d(&m, p, bf, 2, rows, heads, d, d, row, br, 1, 64, sw))) return rc;
  MK(q128, a.q, T, a.hq, DQK, a.q_row, 128) MK(do128, a.d_o, T, a.hq, DV, a.do_row, 128)
  MK(k128, a.k, TK, a.hkv, DQK, a.k_row, 128) MK(v128, a.v, TK, a.hkv, DV, a.v_row, 128)
  MK(dq_m, a.dq, T, a.hq, DQK, a.dq_row, 128) MK(dk_m, a.dk, TK, a.hkv, DQK, a.dk_row, 128)
  MK(dv_m, a.dv, TK, a.hkv, DV, a.dv_row, 128)
  const int var = a.softcap > 0.f ? 2 : (a.window > 0 ? 1 : 0);
  const float* lse2 = a.neg_lse2;
  auto cluster = [&](int mode) {
    return bwd_cluster_size(mode, DQK, DV, a.batch, a.seq, a.seq_k, a.q_off, a.hq, a.hkv, a.causal, a.window);
  };
  const int c_kv = cluster(MODE_DKDV), c_q = cluster(MODE_DQ);
  const dim3 grid_kv = DQK == DV ? dim3(a.hkv * c_kv, a.batch, a.seq_k / BR) : dim3(a.hkv * a.batch * c_kv, a.seq_k / BR);
  const dim3 grid_q(a.hq * c_q, a.batch, a.seq / BR);
  const BwOut out_kv{(__nv_bfloat16*)a.dk, (__nv_bfloat16*)a.dv, a.dk_row, a.dv_row};
  const BwOut out_q{(__nv_bfloat16*)a.dq, nullptr, a.dq_row, 0};
#define PB_BWD(KERN, CFG, THREADS, GRID, CSIZE, OUT, X1, X2, Y1, Y2, O1, O2)                                                        \
  {                                                                                                                     \
    static std::atomic<bool> allowed[3][pbh::MAX_DEVICES];                                                              \
    auto kern = KERN;                                                                                                   \
    if ((rc = pbh::allow_shared_memory(kern, CFG::SMEM_BYTES, allowed[var]))) return rc;                                \
    cudaLaunchConfig_t cfg = {};                                                                                        \
    cfg.gridDim = GRID;                                                                                                 \
    cfg.blockDim = dim3(THREADS);                                                                                       \
    cfg.dynamicSmemBytes = CFG::SMEM_BYTES;                                                                             \
    cfg.stream = a.stream;                                                                                              \
    cudaLaunchAttribute attr[2];                                                                                        \
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;     /* (pb::grid_wait) */                          \
    attr[0].val.programmaticStreamSerializationAllowed = 1;                                                             \
    attr[1].id = cudaLaunchAttributeClusterDimension;                                                                   \
    attr[1].val.clusterDim.x = CSIZE;                                                                                   \
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;                                                            \
    cfg.attrs = attr;                                                                                                   \
    cfg.numAttrs = CSIZE > 1 ? 2 : 1;                                                                                   \
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, X1, X2, Y1, Y2, O1, O2, lse2, (const float*)a.delta, a.seq, a.seq_k, \
                                       a.q_off, a.hq, a.hkv, a.scale, a.causal, a.window, a.softcap, OUT, a.status);    \
    if (e != cudaSuccess) return (int)e;                                                                                \
  }
  if constexpr (DQK == DV) {
    using CKV = BwWideCfg<DQK, DV, MODE_DKDV>;
    PB_BWD((var == 2   ? flash_attn_bwd_wide_kernel<DQK, DV, MODE_DKDV, 2>
            : var == 1 ? flash_attn_bwd_wide_kernel<DQK, DV, MODE_DKDV, 1> : flash_attn_bwd_wide_kernel<DQK, DV, MODE_DKDV, 0>),
           CKV, BWW_THREADS, grid_kv, c_kv, out_kv, k128, v128, q128, do128, dk_m, dv_m)
  } else {
    CUtensorMap q64, do64;                     // (streamed by 64 rows)
    MK(q64, a.q, T, a.hq, DQK, a.q_row, 64) MK(do64, a.d_o, T, a.hq, DV, a.do_row, 64)
    using CKV = BwCfg<DQK, DV>;
    PB_BWD((var ? flash_attn_bwd_kernel<DQK, DV, true> : flash_attn_bwd_kernel<DQK, DV, false>), CKV,
           BW_THREADS, grid_kv, c_kv, out_kv, k128, v128, q64, do64, dk_m, dv_m)
  }
  using CQ = BwWideCfg<DQK, DV, MODE_DQ>;
  PB_BWD((var == 2   ? flash_attn_bwd_wide_kernel<DQK, DV, MODE_DQ, 2>
          : var == 1 ? flash_attn_bwd_wide_kernel<DQK, DV, MODE_DQ, 1> : flash_attn_bwd_wide_kernel<DQK, DV, MODE_DQ, 0>),
         CQ, BWW_THREADS, grid_q, c_q, out_q, q128, do128, k128, v128, dq_m, dq_m)
#undef PB_BWD
#undef MK
  return (int)cudaGetLastError();
}

}  // namespace

// Layouts as in pb_flash_attn_fwd_ex (q / o / d_o / dq: batch*seq rows; k / v / dk / dv: batch*seq_k rows).
// delta: fp32 scratch [2, batch, hq, seq] (written here: row sums of dO*O, then minus the log-sum-exp in log2 units).
extern "C" int pb_flash_attn_bwd_cap(const void* d_o, const void* q, const void* k, const void* v, const void* o,
                                     const float* lse, float* delta, void* dq, void* dk, void* dv, int batch, int seq,
                                     int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row, long k_row,
                                     long v_row, long o_row, long do_row, long dq_row, long dk_row, long dv_row,
                                     float scale, int causal, int window, float softcap, int* status,
                                     cudaStream_t stream) {
  if (batch <= 0 || seq % 128 || seq_k % 128 || q_off % 128 || q_off < 0 || hq % hkv) return -2;
  if (causal ? (q_off + seq != seq_k) : (q_off != 0)) return -2;
  if (window < 0 || (window > 0 && (!causal || q_off != 0)) || softcap < 0.f) return -2;
  if ((q_row | k_row | v_row | o_row | do_row | dq_row | dk_row | dv_row) % 8) return -2;
  constexpr int MAX_BATCH = 65535;             // (sequences are the grid's second dimension)
  float* neg_lse2 = delta + (long)batch * hq * seq;
  for (int b = 0; b < batch; b += MAX_BATCH) {
    const long tq = (long)b * seq, tk = (long)b * seq_k;
    auto at = [](const void* p, long rows, long pitch) { return static_cast<const __nv_bfloat16*>(p) + rows * pitch; };
    auto to = [](void* p, long rows, long pitch) { return static_cast<__nv_bfloat16*>(p) + rows * pitch; };
    BwdArgs a{at(d_o, tq, do_row), at(q, tq, q_row), at(k, tk, k_row), at(v, tk, v_row), at(o, tq, o_row), lse + tq * hq,
              delta + tq * hq, neg_lse2 + tq * hq, to(dq, tq, dq_row), to(dk, tk, dk_row), to(dv, tk, dv_row),
              batch - b < MAX_BATCH ? batch - b : MAX_BATCH, seq, seq_k, q_off, window, hq, hkv, softcap, q_row, k_row, v_row,
              o_row, do_row, dq_row, dk_row, dv_row, scale, causal, status, stream};
    const int rc = d_qk == 128 && d_v == 128   ? launch_bwd<128, 128>(a)
                   : d_qk == 192 && d_v == 128 ? launch_bwd<192, 128>(a)
                   : d_qk == 64 && d_v == 64   ? launch_bwd<64, 64>(a) : -3;
    if (rc) return rc;
  }
  return 0;
}

// CTAs per row block that pb_flash_attn_bwd_cap launches: pass 0 dK / dV, 1 dQ (host only).
extern "C" int pb_flash_attn_bwd_cluster(int pass, int batch, int seq, int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v,
                                         int causal, int window) {
  return bwd_cluster_size(pass, d_qk, d_v, batch, seq, seq_k, q_off, hq, hkv, causal, window);
}

extern "C" int pb_flash_attn_bwd_win(const void* d_o, const void* q, const void* k, const void* v, const void* o,
                                     const float* lse, float* delta, void* dq, void* dk, void* dv, int batch, int seq,
                                     int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row, long k_row,
                                     long v_row, long o_row, long do_row, long dq_row, long dk_row, long dv_row,
                                     float scale, int causal, int window, int* status, cudaStream_t stream) {
  return pb_flash_attn_bwd_cap(d_o, q, k, v, o, lse, delta, dq, dk, dv, batch, seq, seq_k, q_off, hq, hkv, d_qk, d_v,
                               q_row, k_row, v_row, o_row, do_row, dq_row, dk_row, dv_row, scale, causal, window, 0.f,
                               status, stream);
}

extern "C" int pb_flash_attn_bwd_ex(const void* d_o, const void* q, const void* k, const void* v, const void* o,
                                    const float* lse, float* delta, void* dq, void* dk, void* dv, int batch, int seq,
                                    int seq_k, int q_off, int hq, int hkv, int d_qk, int d_v, long q_row, long k_row,
                                    long v_row, long o_row, long do_row, long dq_row, long dk_row, long dv_row,
                                    float scale, int causal, int* status, cudaStream_t stream) {
  return pb_flash_attn_bwd_win(d_o, q, k, v, o, lse, delta, dq, dk, dv, batch, seq, seq_k, q_off, hq, hkv, d_qk, d_v,
                               q_row, k_row, v_row, o_row, do_row, dq_row, dk_row, dv_row, scale, causal, 0, status,
                               stream);
}

extern "C" int pb_flash_attn_bwd(const void* d_o, const void* q, const void* k, const void* v, const void* o,
                                 const float* lse, float* delta, void* dq, void* dk, void* dv, int batch, int seq,
                                 int hq, int hkv, int d_qk, int d_v, long q_row, long k_row, long v_row, long o_row,
                                 long do_row, long dq_row, long dk_row, long dv_row, float scale, int causal,
                                 int* status, cudaStream_t stream) {
  return pb_flash_attn_bwd_ex(d_o, q, k, v, o, lse, delta, dq, dk, dv, batch, seq, seq, 0, hq, hkv, d_qk, d_v, q_row,
                              k_row, v_row, o_row, do_row, dq_row, dk_row, dv_row, scale, causal, status, stream);
}

// dsinks[h] from the row sums delta [batch, hq, seq] that the backward left in its scratch and the forward's lse.
extern "C" int pb_attn_sink_grad(const float* delta, const float* lse, const float* sinks, float* dsinks, int batch, int seq,
                                 int hq, cudaStream_t stream) {
  if (hq <= 0) return 0;
  pbh::launch_dependent(attn_sink_grad_kernel, hq, 1024, 0, stream, delta, lse, sinks, dsinks, batch, seq, hq);
  return (int)cudaGetLastError();
}
