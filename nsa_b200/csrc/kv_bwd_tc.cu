// Key/value-major backward of the selected branch on tcgen05 (head_dim 128, 64-key blocks): dK, dV and dQ partials.  Same work
// decomposition and reference semantics as kv_bwd.cu (nsa/selection_attn.py:151-253 through a reverse index), different engine.
//
// One CTA owns 64 keys.  Query tokens that see them arrive in batches of 8: the 8 x 16 (token, head) rows form a
// [128 x D] tile of Q and of dO in shared memory (one 4 KB TMA box per token, 128-byte swizzle).  Per batch, one
// thread issues four groups of tcgen05.mma (accumulators in TMEM):
//     S   [128 rows x 64 keys] = Qg . K^T          A = Qg (K-major),  B = K  (K-major)
//     dP  [128 rows x 64 keys] = dOg . V^T         A = dOg (K-major), B = V  (K-major)
//     dV^T[128 d    x 64 keys] += dOg^T . (g P)    A = dOg (MN-major), B = P  (MN-major, written by the soft-max warps)
//     dK^T[128 d    x 64 keys] += Qg^T . dS        A = Qg (MN-major),  B = dS (MN-major)
// Eight soft-max warps own half a row per thread (warps 4-7 take key columns 0-31, warps 8-11 columns 32-63 of the same TMEM
// lanes; a row's lse, delta, gate and number of visible keys lie in shared memory): they read S and dP
// from TMEM, form P and dS = P (g dP - delta), and store both as bf16 tiles.
// The MMA threads issue S/dP of batch n+1 before dV/dK of batch n, so the tensor core works while the soft-max
// warps compute; the exponentials start when S alone is there, dV when P alone is written.  dV^T and dK^T stay in TMEM for
// the CTA's whole token stream and are stored once.
// Optionally dQ comes out of this kernel too: dS of a batch is already in shared memory,
// so one more product  dQ_part[128 rows x 128 d] = dS . K  (A = dS K-major, B = K MN-major, a third accumulator in TMEM)
// gives the batch's contribution to dQ, which the drain warps store as bf16 tiles indexed by the batch's positions
// in the reverse-index list; a small kernel later sums every token's tiles in slot order.  That replaces the
// query-major dQ kernel, which gathers every selected block again (32 KB per visit for 16 rows) and recomputes S and dP.
//
// Bound: the round trip of the two Q/dO stages (gather 1800 cycles, S, soft-max, dV and dK: 3650 cycles per batch) and shared
// memory (3100 cycles of operands, arriving rows and stores).  A row's lse, delta and gate are fetched once, by the drain warps: both
// soft-max threads of a row fetching them, with a division by the batch count and three unrolled variants of the arithmetic, kept those
// warps busy 3500 of 4070 cycles.  The epilogue is a loop: unrolled it cost 55 000 cycles a CTA in instruction fetches.
// 8 x 8192 tokens, 64 heads: 4.90 -> 4.08 ms with both; 65536 tokens: 5.0 -> 4.1; 2 x 2080 tokens, 32 heads: 153 -> 129 us.
// Every wait is bounded; on a time-out the role records an error and leaves its loop.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int D = 128;
constexpr int kProd = 2;                   // TMA producer warps: Q, dO
constexpr int kMmaWarp = 2;                // issues S and dP
constexpr int kMma2Warp = 3;               // issues dV, dK and the dQ partials
constexpr int kSoftWarp = 4;               // eight soft-max / epilogue warps
constexpr int kDrainWarp = 12;             // four more warps read the dQ partials out of tensor memory
constexpr int kThreads = 16 * 32;          // 512: four warpgroups, registers redistributed by setmaxnreg
constexpr int kSoftThreads = 256;          // two threads per row: key columns 0-31 and 32-63
constexpr int kDrainThreads = 128;         // one thread per row
constexpr int kTokB = 8;                   // tokens per batch (x16 heads = 128 rows)
constexpr uint32_t KV_PANEL = 64 * 128;    // [64 keys][64 ch]
constexpr uint32_t KV_TILE = 2 * KV_PANEL; // 16 KB
constexpr uint32_t Q_TILE = 128 * 256;     // 32 KB: [16 row groups][2 column panels][8 rows][128 B]
constexpr uint32_t STAGE = 2 * Q_TILE;     // Q + dO
constexpr uint32_t P_TILE = 128 * 128;     // [128 rows][64 keys]
constexpr int kStages = 2;
// K, V | Q and dO stages | two P/dS pairs | barriers | a batch's row data
constexpr uint32_t kOffBar = 2 * KV_TILE + kStages * STAGE + 4 * P_TILE, kOffRow = kOffBar + 256, kSmem = kOffRow + 128 * 12 + 1024;
static_assert(kSmem <= 227 * 1024, "with the bytes that it takes to align the tiles");
constexpr uint32_t kTmemCols = 512;        // two S/dP buffers: S 0..63, dP 64..127 | 128..255; dV^T 256..319, dK^T 320..383
constexpr uint32_t kColDV = 256, kColDK = 320, kColDQ = 384;   // dQ_part: 384..511

__global__ void __launch_bounds__(kThreads, 1)
    kv_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const KvArgs a) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;   // the 128-byte swizzle repeats every 1024 bytes
  uint8_t* const sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t k_s = sbase, v_s = sbase + KV_TILE;
  const uint32_t ring = sbase + 2 * KV_TILE;
  const uint32_t p_s0 = ring + kStages * STAGE;   // two [P | dS] tile pairs
  const uint32_t bar_base = sbase + kOffBar;
  // barriers
  // sdp_* and pds_* exist twice (index = batch & 1): S/dP of batch n+1 are computed while the soft-max warps still
  // hold batch n, and P/dS of batch n+1 are written while dV/dK of batch n still read theirs
  // q* and do* by stage: Q is held until dK, dO until dP and dV
  const uint32_t qfull0 = bar_base, qempty0 = bar_base + 16, dofull0 = bar_base + 192, doempty0 = bar_base + 208, kv_bar = bar_base + 32, sdp_full = bar_base + 40,
                 sdp_free = bar_base + 56, pds_full = bar_base + 72, pds_free = bar_base + 88, acc_full = bar_base + 104,
                 tmem_slot = bar_base + 112, dq_full = bar_base + 120, dq_free = bar_base + 128, stg_full = bar_base + 240,
                 stg_free = bar_base + 144, s_full = bar_base + 160, p_full = bar_base + 176,
                 row_full = bar_base + 224, row_empty = bar_base + 232;   // stg_full, stg_free: one per P/dS pair
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(qfull0 + 8 * i, 1);
      mbar_init(qempty0 + 8 * i, 1);
      mbar_init(dofull0 + 8 * i, 1);
      mbar_init(doempty0 + 8 * i, 2);
    }
    mbar_init(kv_bar, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full + 8 * i, 1);
      mbar_init(sdp_full + 8 * i, 1);
      mbar_init(p_full + 8 * i, kSoftThreads);
      mbar_init(sdp_free + 8 * i, kSoftThreads);
      mbar_init(pds_full + 8 * i, kSoftThreads);
      mbar_init(pds_free + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(row_full, kDrainThreads);
    mbar_init(row_empty, kSoftThreads);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, kDrainThreads);
    mbar_init(stg_full, kDrainThreads);
    mbar_init(stg_full + 8, kDrainThreads);
    mbar_init(stg_free, 1);
    mbar_init(stg_free + 8, 1);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));

  // ---- decode the work item ------------------------------------------------------------------------------
  // (batch, kv head)-major: the CTAs resident at one time share one 16-head group's Q and dO rows (67 MB at T = 8192), which
  // then stay in L2; block-major order made every gather a DRAM access
  const int G16 = (a.Hq / a.Hk) / 16;
  const int NB = (a.T + 63) / 64;
  const int seg = blockIdx.x % a.nshare, item = blockIdx.x / a.nshare;
  const int nbh = a.B * a.Hk;   // shares of a list: longest lists first (few enough items for all of Q and dO to stay in L2)
  const int blk = a.nshare > 1 ? item / nbh : item % NB, bh = a.nshare > 1 ? item % nbh : item / NB, b = bh / a.Hk, hk = bh % a.Hk;
  const int* rp = a.rev_ptr + (long long)bh * (NB + 1);
  const int* list = a.rev_tok + (long long)bh * a.rev_cap;
  int lo = rp[blk], nA = rp[blk + 1] - lo;
  if (a.nshare > 1) {   // this CTA's share of the list, in whole batches
    const int ba = (nA + kTokB - 1) / kTokB;
    const int a0 = ba * seg / a.nshare * kTokB, a1 = min(nA, ba * (seg + 1) / a.nshare * kTokB);
    lo += a0;
    nA = a1 - a0;
  }
  const int key0 = blk * 64;
  const int nb_sub = (nA + kTokB - 1) / kTokB;   // batches per 16-head sub-group
  const int nb = nb_sub * G16;                   // batches of this CTA
  const bool emit_dq = a.dq_part != nullptr;     // every batch also leaves its dQ partial
  auto list_token = [&](int i) { return list[lo + min(i, nA - 1)]; };

  // 512 threads start with 128 registers each; the soft-max warps need 168.  Warps 0-3 (TMA, MMA) and 12-15 (drain)
  // give registers back, warps 4-11 take them (each instruction is executed by a whole warpgroup).
  // Each role's code follows its own setmaxnreg, so the compiler allocates registers for it under that budget.
  // Budget (setmaxnreg moves registers inside the pool the CTA was launched with, 512 x 128 = 65536; an inc that the
  // pool cannot satisfy blocks for ever): 128 x 80 + 256 x 168 + 128 x 88 = 64512.
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
  if (warp < kProd) {
    // ------------------------------- TMA producers -----------------------------------------------
    // A batch of gathered tokens (a reverse-index list) is 16 boxes of 4 KB, one per token of Q and one of dO, through a 4-D
    // view (64 columns, 8 rows, 2 column panels, row groups) as in the forward: the gather is bound by the number of
    // boxes.  Warp 0 gathers Q, warp 1 dO; lane j finds where the batch's token j is, one lane issues the eight boxes and
    // arms the stage's barrier with their byte count.  Token ids are fetched one batch ahead.
    if (warp == 0 && nb > 0 && elect_one()) {
      mbar_expect_tx(kv_bar, 2 * KV_TILE);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        tma_load_4d(k_s + p * KV_PANEL, &tmK, kv_bar, p * 64, hk, key0, b);
        tma_load_4d(v_s + p * KV_PANEL, &tmV, kv_bar, p * 64, hk, key0, b);
      }
    }
    const bool has = lane < kTokB;
    const uint32_t full0 = warp ? dofull0 : qfull0, empty0 = warp ? doempty0 : qempty0, dst0 = ring + (warp ? Q_TILE : 0);
    const CUtensorMap* const tm = warp ? &tmDO : &tmQ;
    auto batch_token = [&](int n) { return n >= nb || !has ? 0 : list_token(n % nb_sub * kTokB + lane); };
    int tk_next = batch_token(0);
    for (int n = 0; n < nb; ++n) {
      const int tk = tk_next;
      tk_next = batch_token(n + 1);
      const int hg = hk * G16 + n / nb_sub;
      const int stage = n % kStages;
      const uint32_t ph = (n / kStages) & 1;
      const uint32_t fb = full0 + 8 * stage;
      const int grp = (int)((((long long)b * a.Tq + (tk - a.q0)) * a.Hq + hg * 16) >> 3);
      int row_group[kTokB];
#pragma unroll
      for (int j = 0; j < kTokB; ++j) row_group[j] = __shfl_sync(0xffffffffu, grp, j);
      const bool good = mbar_wait(empty0 + 8 * stage, ph ^ 1, DEV_ERR_EMPTY_WAIT);
      if (!__all_sync(0xffffffffu, good)) break;
      if (elect_one()) {
        mbar_expect_tx(fb, Q_TILE);
#pragma unroll
        for (int j = 0; j < kTokB; ++j) tma_load_4d(dst0 + stage * STAGE + j * 4096, tm, fb, 0, 0, 0, row_group[j]);
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------- MMA issuer A: S and dP ----------------------------------------
    // S/dP of batch n is issued as soon as its Q/dO stage has landed and its TMEM buffer is free (the soft-max warps
    // hold batch n-2 in registers), i.e. ahead of dV/dK of batch n-1, which the second issuer handles.
    if (nb > 0 && elect_one()) {
      constexpr uint32_t idesc_kk = umma_idesc_bf16(128, 64, 0, 0);   // both operands K-major
      bool ok = mbar_wait(kv_bar, 0, DEV_ERR_FULL_WAIT);
      const uint64_t dK = umma_smem_desc(k_s, 0, 1024), dV = umma_smem_desc(v_s, 0, 1024);
      uint64_t dQk[kStages], dDOk[kStages];
#pragma unroll
      for (int i = 0; i < kStages; ++i) {
        const uint32_t q_s = ring + i * STAGE, do_s = q_s + Q_TILE;
        dQk[i] = umma_smem_desc(q_s, 0, 2048);
        dDOk[i] = umma_smem_desc(do_s, 0, 2048);
      }
      for (int n = 0; ok && n < nb; ++n) {
        ok = mbar_wait(qfull0 + 8 * (n % kStages), (n / kStages) & 1, DEV_ERR_FULL_WAIT);
        if (ok && n >= 2) ok = mbar_wait(sdp_free + 8 * (n & 1), ((n >> 1) - 1) & 1, DEV_ERR_EMPTY_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint64_t aq = (n % kStages) ? dQk[1] : dQk[0], ado = (n % kStages) ? dDOk[1] : dDOk[0];
        const uint32_t col = (n & 1) * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t aoff = (ks >> 2) * 1024 + (ks & 3) * 32, boff = (ks >> 2) * KV_PANEL + (ks & 3) * 32;
          umma_ss(tmem + col, umma_desc_advance(aq, aoff), umma_desc_advance(dK, boff), idesc_kk, ks ? 1u : 0u);
        }
        umma_commit(s_full + 8 * (n & 1));   // the exponentials need S alone
        ok = mbar_wait(dofull0 + 8 * (n % kStages), (n / kStages) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t aoff = (ks >> 2) * 1024 + (ks & 3) * 32, boff = (ks >> 2) * KV_PANEL + (ks & 3) * 32;
          umma_ss(tmem + col + 64, umma_desc_advance(ado, aoff), umma_desc_advance(dV, boff), idesc_kk, ks ? 1u : 0u);
        }
        umma_commit(sdp_full + 8 * (n & 1));
        umma_commit(doempty0 + 8 * (n % kStages));
      }
    }
  } else if (warp == kMma2Warp) {
    // ------------------------------- MMA issuer B: dV, dK, dQ partials -----------------------------
    if (nb > 0 && elect_one()) {
      constexpr uint32_t idesc_mn = umma_idesc_bf16(128, 64, 1, 1);   // both operands MN-major
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, 128, 0, 1);  // A = dS K-major, B = K MN-major
      bool ok = mbar_wait(kv_bar, 0, DEV_ERR_FULL_WAIT);
      uint64_t dQmn[kStages], dDOmn[kStages], dP[2], dDS[2], dDSk[2];
#pragma unroll
      for (int i = 0; i < kStages; ++i) {
        const uint32_t q_s = ring + i * STAGE, do_s = q_s + Q_TILE;
        dQmn[i] = umma_smem_desc(q_s, 1024, 2048);
        dDOmn[i] = umma_smem_desc(do_s, 1024, 2048);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        dP[i] = umma_smem_desc(p_s0 + i * 2 * P_TILE, 0, 1024);
        dDS[i] = umma_smem_desc(p_s0 + i * 2 * P_TILE + P_TILE, 0, 1024);
        dDSk[i] = dDS[i];   // the same tile read K-major for the dQ partial
      }
      const uint64_t dKmn = umma_smem_desc(k_s, KV_PANEL, 1024);
      for (int n = 0; ok && n < nb; ++n) {
        ok = mbar_wait(dofull0 + 8 * (n % kStages), (n / kStages) & 1, DEV_ERR_FULL_WAIT) &&
             mbar_wait(p_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint64_t aq = (n % kStages) ? dQmn[1] : dQmn[0], ado = (n % kStages) ? dDOmn[1] : dDOmn[0];
        const uint64_t bp = (n & 1) ? dP[1] : dP[0], bds = (n & 1) ? dDS[1] : dDS[0];
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)   // contraction over the 128 rows, 16 per step; dV while the soft-max warps form dS
          umma_ss(tmem + kColDV, umma_desc_advance(ado, ks * 4096), umma_desc_advance(bp, ks * 2048), idesc_mn, (n | ks) ? 1u : 0u);
        umma_commit(doempty0 + 8 * (n % kStages));
        ok = mbar_wait(pds_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_ss(tmem + kColDK, umma_desc_advance(aq, ks * 4096), umma_desc_advance(bds, ks * 2048), idesc_mn, (n | ks) ? 1u : 0u);
        umma_commit(qempty0 + 8 * (n % kStages));
        if (emit_dq) {
          // the previous partial must have been read out of its accumulator by the drain warps
          if (n > 0) ok = mbar_wait(dq_free, (n - 1) & 1, DEV_ERR_EMPTY_WAIT);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ads = (n & 1) ? dDSk[1] : dDSk[0];
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)   // contraction over the 64 keys, 16 per step
            umma_ss(tmem + kColDQ, umma_desc_advance(ads, ks * 32), umma_desc_advance(dKmn, ks * 2048), idesc_dq, ks ? 1u : 0u);
          umma_commit(dq_full);
        }
        umma_commit(pds_free + 8 * (n & 1));
      }
      umma_commit(acc_full);
    }
  }
  } else if (warp >= kDrainWarp) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
  {
    // ------------------------------- drain warps: dQ partials, one row per thread ------------------
    // dQ partial of a batch: accumulator -> bf16 -> shared memory -> one bulk store.  The staging area is that
    // batch's own P/dS tile pair (32 KB = 128 rows x 256 bytes): dq_full also says that every MMA that read the pair
    // has completed, and the soft-max warps write it again (batch n+2) only after stg_free.  The 8 tokens' [16 x D]
    // tiles sit at consecutive list positions, i.e. contiguous in dq_part when the KV head has one 16-head group.
    // Within a 128-byte half row the 16-byte chunk c is stored at position c ^ (row & 7) (conflict-free writes;
    // row & 7 == head & 7, and the reduction kernel undoes it).  Plain stores from the accumulator's layout (a thread
    // owns a row: 16 bytes per lane at a 256-byte stride) cost a tenth of the kernel in store wavefronts, and reading
    // the partials out in the soft-max warps delayed the next batch's soft-max.
    // Before that, the thread's row of the batch after next: what the soft-max warps need to know of it (the two that share a row
    // would each fetch and address it themselves, a quarter of their time).
    {
      const int quad = warp & 3;
      const int row = 32 * quad + lane;
      const int j = row >> 4;
      const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
      const bool elected = warp == kDrainWarp && lane == 0;
      const long long head0 = (long long)b * a.Tq * a.Hq + hk * G16 * 16 + (row & 15);
      float2* const row_ld = reinterpret_cast<float2*>(sgen + kOffRow) + row;
      uint32_t* const row_gn = reinterpret_cast<uint32_t*>(sgen + kOffRow + 128 * 8) + row;
      // batch to be fetched next: place in its 16-head sub-group, sub-group; its token (two batches ahead of the publication)
      int fm = 0, fsub = 0, ft = nA > 0 ? list_token(j) : 0;
      float lse = 0.f, del = 0.f;
      bf16 g = __float2bfloat16(1.f);
      int nv = 0;
      auto fetch = [&](int n) {   // row data of batch n, kept as loaded: converting them would wait for the loads
        if (n >= nb) return;
        const long long qrow = head0 + (long long)(ft - a.q0) * a.Hq + fsub * 16;
        lse = a.lse[qrow];
        del = a.delta[qrow];
        if (a.gate) g = a.gate[qrow];
        nv = fm * kTokB + j < nA ? min(64, ft - key0 + 1) : 0;   // keys that the row sees (the block's first at least)
        if (++fm == nb_sub) {
          fm = 0;
          ++fsub;
        }
        ft = list_token(fm * kTokB + j);
      };
      auto publish = [&](int n) {
        if (n >= nb) return true;
        if (n > 0 && !mbar_wait(row_empty, (n - 1) & 1, DEV_ERR_EMPTY_WAIT)) return false;
        const uint32_t gn = (uint32_t)__bfloat16_as_ushort(g) << 16 | (lse > -INFINITY ? nv : 0);   // (a row that sees nothing: none)
        *row_ld = make_float2(-lse * kLog2e, -del);
        *row_gn = gn;
        mbar_arrive(row_full);
        fetch(n + 1);
        return true;
      };
      fetch(0);
      bool ok = publish(0) && publish(1);
      for (int n = 0; ok && n < nb; ++n) {
        ok = publish(n + 2);
        if (!ok || !emit_dq) continue;
        const int sub = n / nb_sub, mloc = n % nb_sub;
        ok = mbar_wait(dq_full, n & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint32_t stg = p_s0 + (uint32_t)(n & 1) * 2 * P_TILE;
        uint8_t* sp = sgen + (stg - sbase) + row * 256;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {   // 32 columns at a time
          float vals[2][16];
          tmem_ld16(tmem + lane_addr + kColDQ + q4 * 32, vals[0]);
          tmem_ld16(tmem + lane_addr + kColDQ + q4 * 32 + 16, vals[1]);
          tmem_ld_wait();
          if (q4 == 3) {
            tc_fence_before();
            mbar_arrive(dq_free);   // the accumulator is in registers: the next partial may be issued
          }
#pragma unroll
          for (int c2 = 0; c2 < 4; ++c2) {   // four 16-byte chunks
            const float* f = &vals[c2 >> 1][(c2 & 1) * 8];
            uint4 o;
            __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e) ho[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
            const int cc = q4 * 4 + c2;       // chunk 0..15 of the row: half cc >> 3, position (cc & 7) ^ (row & 7)
            *reinterpret_cast<uint4*>(sp + (cc >> 3) * 128 + (((cc & 7) ^ (row & 7)) * 16)) = o;
          }
        }
        fence_proxy_async();
        mbar_arrive(stg_full + 8 * (n & 1));   // (two: a warp may be a batch ahead of the slowest)
        if (elected) {
          ok = mbar_wait(stg_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
          const int nvalid = min(kTokB, nA - mloc * kTokB);
          if (ok && nvalid > 0) {
            bf16* dst = a.dq_part + (((long long)bh * a.rev_cap + lo + mloc * kTokB) * G16 + sub) * (16 * D);
            if (G16 == 1) {
              bulk_store_evict_first(dst, stg, (uint32_t)nvalid * 16 * D * 2);
            } else {
              for (int i = 0; i < nvalid; ++i)
                bulk_store_evict_first(dst + (long long)i * G16 * 16 * D, stg + i * 16 * D * 2, 16 * D * 2);
            }
          }
          bulk_commit();
          bulk_wait_read();                       // the pair may be written again
          mbar_arrive(stg_free + 8 * (n & 1));
        }
      }
      if (elected) bulk_wait_all();
    }
  }
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
  {
    // ------------------------------- soft-max warps: one (token, head) row per thread --------------
    const int quad = warp & 3;
    const int half = (warp - kSoftWarp) >> 2;    // which 32 key columns this thread owns
    const int row = 32 * quad + lane;           // TMEM lane == tile row
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const float sl2 = a.scale * kLog2e;
    bool ok = true;
    // With dQ partials: the drain warps stage the partial of batch n in that batch's own P/dS pair; the pair is written again
    // for batch n+2 only after their bulk store has read it (stg_free of that pair).
    const uint64_t sl22 = pack_f32x2(sl2, sl2);
    uint8_t* const prow0 = sgen + (p_s0 - sbase) + row * 128;
    const float2* const row_ld = reinterpret_cast<const float2*>(sgen + kOffRow) + row;
    const uint32_t* const row_gn = reinterpret_cast<const uint32_t*>(sgen + kOffRow + 128 * 8) + row;
    for (int n = 0; ok && n < nb; ++n) {
      ok = mbar_wait(row_full, n & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      const float2 ri = *row_ld;
      const uint32_t gn = *row_gn;
      mbar_arrive(row_empty);
      const uint32_t buf = n & 1, use = n >> 1;
      const uint32_t scol = tmem + lane_addr + buf * 128 + half * 32;
      ok = mbar_wait(s_full + 8 * buf, use & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      float p[32];
      tmem_ld32(scol, p);
      const float gv = __uint_as_float(gn & 0xffff0000u);
      const int nrow = gn & 0xffff, nvis = nrow - 32 * half;   // visible keys of the block, of this half (0: a row that is not there)
      const uint64_t nl2 = pack_f32x2(ri.x, ri.x), g2 = pack_f32x2(gv, gv), nd2 = pack_f32x2(ri.y, ri.y);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const uint64_t x = fma_f32x2(pack_f32x2(p[e], p[e + 1]), sl22, nl2);
        p[e] = lo_f32x2(x);
        p[e + 1] = hi_f32x2(x);
      }
      if (nvis < 32) {
#pragma unroll
        for (int e = 0; e < 32; ++e) p[e] = e < nvis ? p[e] : -INFINITY;
      }
      uint32_t pw[16];   // 32 bf16
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        p[e] = ex2(p[e]);
        p[e + 1] = ex2(p[e + 1]);
        const uint64_t gp = mul_f32x2(g2, pack_f32x2(p[e], p[e + 1]));
        pw[e / 2] = pack_bf16(lo_f32x2(gp), hi_f32x2(gp));
      }
      // dV/dK of batch n-2 have read this pair, and the bulk stores of its dQ partial
      if (n >= 2) {
        ok = mbar_wait(pds_free + 8 * buf, (use - 1) & 1, DEV_ERR_EMPTY_WAIT);
        if (ok && emit_dq) ok = mbar_wait(stg_free + 8 * buf, (use - 1) & 1, DEV_ERR_EMPTY_WAIT);
        if (!ok) break;
      }
      // this thread's half of row `row` of the [128 x 64] bf16 tiles: 4 chunks of 16 bytes at swizzled positions
      uint8_t* const prow = prow0 + buf * 2 * P_TILE;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(prow + ((4 * half + c) ^ (row & 7)) * 16) = make_uint4(pw[4 * c], pw[4 * c + 1], pw[4 * c + 2], pw[4 * c + 3]);
      fence_proxy_async();
      mbar_arrive(p_full + 8 * buf);
      ok = mbar_wait(sdp_full + 8 * buf, use & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      float dpv[32];
      tmem_ld32(scol + 64, dpv);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(sdp_free + 8 * buf);   // S and dP are in registers: batch n+2 may overwrite this TMEM buffer
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const uint64_t x = fma_f32x2(g2, pack_f32x2(dpv[e], dpv[e + 1]), nd2);
        const uint64_t d2 = mul_f32x2(pack_f32x2(p[e], p[e + 1]), x);
        pw[e / 2] = pack_bf16(lo_f32x2(d2), hi_f32x2(d2));
      }
      if (nrow == 0) {   // (0 times whatever dP is)
#pragma unroll
        for (int e = 0; e < 16; ++e) pw[e] = 0u;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(prow + P_TILE + ((4 * half + c) ^ (row & 7)) * 16) = make_uint4(pw[4 * c], pw[4 * c + 1], pw[4 * c + 2], pw[4 * c + 3]);
      fence_proxy_async();
      mbar_arrive(pds_full + 8 * buf);
    }
    // ---- epilogue: dV^T / dK^T [d lanes x 64 key columns] -> global ---------------------------------------
    if (ok && nb > 0) ok = mbar_wait(acc_full, 0, DEV_ERR_FULL_WAIT);
    tc_fence_after();
    // Half 0 stores dV, half 1 dK; a thread has one channel.  The loop is not unrolled: straight-line code that a CTA runs once comes
    // from beyond the instruction cache (all 64 keys unrolled, with their variants, took 55 000 cycles beside 384 000 for 94 batches)
    const float mul = half ? a.scale : 1.f;
    const long long Nout = (long long)a.B * a.T * a.Hk * D;
    const int step = a.Hk * D, nk = ok ? min(64, a.T - key0) : 0;
    const long long off0 = (((long long)b * a.T + key0) * a.Hk + hk) * D + row;
    const float* const win = a.part + (half ? 0 : a.slabs * Nout) + off0;   // the window's part, or where a share goes
#pragma unroll 1
    for (int c = 0; c < 64; c += 16) {
      float vals[16];
      if (nb > 0) {
        tmem_ld16(tmem + lane_addr + kColDV + half * 64 + c, vals);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) vals[e] = 0.f;
      }
      if (a.nshare > 1) {
        float* const dst = const_cast<float*>(win) + seg * Nout + (long long)c * step;
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (c + e < nk) dst[e * step] = vals[e] * mul;
      } else {
        float add[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) add[e] = 0.f;
#pragma unroll 1
        for (int w = 0; w < a.nadd; ++w) {
          const float* const src = win + w * Nout + (long long)c * step;
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (c + e < nk) add[e] += src[e * step];
        }
        bf16* const dst = (half ? a.dk : a.dv) + off0 + (long long)c * step;
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (c + e < nk) dst[e * step] = __float2bfloat16(fmaf(vals[e], mul, add[e]));
      }
    }
  }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemCols);
}

int launch(const KvArgs& a, cudaStream_t s) {
  CUtensorMap tmQ, tmDO, tmK, tmV;
  const long long qrows = (long long)a.B * a.Tq * a.Hq;
  if (qrows > 0x7fffffffLL) {
    set_error("B*T*Hq exceeds the 2^31 rows a TMA coordinate can address");
    return -32;
  }
  // rows as (64 columns, 8 rows, 2 column panels, groups of 8 rows): one box = 16 rows x 128 columns of one token
  const unsigned long long qd[4] = {64, 8, 2, (unsigned long long)(qrows / 8)};
  const unsigned long long qs[3] = {(unsigned long long)D * 2, 128, (unsigned long long)D * 2 * 8};
  const unsigned qb[4] = {64, 8, 2, 2};
  int rc = make_tmap_generic(&tmQ, a.q, 4, qd, qs, qb);
  if (!rc) rc = make_tmap_generic(&tmDO, a.dout, 4, qd, qs, qb);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.k, D, a.Hk, a.T, a.B, 64);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hk, a.T, a.B, 64);
  if (rc) return rc;
  cudaError_t e = cudaFuncSetAttribute(kv_bwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return (int)e;
  const long long grid = (long long)a.B * a.Hk * ((a.T + 63) / 64) * a.nshare;
  if (grid <= 0) return 0;
  if (grid > 0x7fffffffLL) {
    set_error("kv backward: grid too large");
    return -33;
  }
  launch_next(kv_bwd_tc_kernel, (unsigned)grid, kThreads, kSmem, s, tmQ, tmDO, tmK, tmV, a);
  note_launches(1);
  return (int)cudaGetLastError();
}

}  // namespace

// head_dim 128 and 64-key blocks only; the caller falls back to launch_kv_bwd otherwise.
int launch_kv_bwd_tc(const KvArgs& a, cudaStream_t s) { return launch(a, s); }
int kv_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
