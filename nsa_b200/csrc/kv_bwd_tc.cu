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
// Eight soft-max warps own half a row per thread (lse, delta, gate and the causal mask are thread-local, no
// shuffles; warps 2-5 take key columns 0-31, warps 6-9 columns 32-63 of the same TMEM lanes): they read S and dP
// from TMEM, form P and dS = P (g dP - delta), and store both as bf16 tiles.
// The MMA threads issue S/dP of batch n+1 before dV/dK of batch n, so the tensor core works while the soft-max
// warps compute; the exponentials start when S alone is there, dV when P alone is written.  dV^T and dK^T stay in TMEM for
// the CTA's whole token stream and are stored once.
// Optionally dQ comes out of this kernel too: dS of a batch is already in shared memory,
// so one more product  dQ_part[128 rows x 128 d] = dS . K  (A = dS K-major, B = K MN-major, a third accumulator in TMEM)
// gives the batch's contribution to dQ, which the drain warps store as bf16 tiles indexed by the batch's positions
// in the reverse-index list; a small kernel later sums every token's tiles in slot order.  That replaces the
// query-major dQ kernel, which gathers every selected block again (32 KB per visit for 16 rows) and recomputes S and dP.
// Every wait is bounded; on a time-out the role records an error and leaves its loop.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int D = 128;
constexpr int kProd = 2;                   // TMA producer warps (a warp's TMA instructions run one after another,
                                           // ~900 cycles each whatever their size, so the boxes of a batch are
                                           // spread over two warps and issued by one instruction per warp)
constexpr int kMmaWarp = 2;                // issues S and dP
constexpr int kMma2Warp = 3;               // issues dV, dK and the dQ partials: tcgen05.mma costs its issuing thread
                                           // ~60 cycles per instruction, so two threads issue the kernel's 32-36 MMAs
                                           // per batch
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
constexpr uint32_t kSmem = 2 * KV_TILE + kStages * STAGE + 4 * P_TILE + 256 + 1024;
constexpr uint32_t kTmemCols = 512;        // two S/dP buffers: S 0..63, dP 64..127 | 128..255; dV^T 256..319, dK^T 320..383
constexpr uint32_t kColDV = 256, kColDK = 320, kColDQ = 384;   // dQ_part: 384..511

__global__ void __launch_bounds__(kThreads, 1)
    kv_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const KvArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t k_s = sbase, v_s = sbase + KV_TILE;
  const uint32_t ring = sbase + 2 * KV_TILE;
  const uint32_t p_s0 = ring + kStages * STAGE;   // two [P | dS] tile pairs
  const uint32_t bar_base = p_s0 + 4 * P_TILE;
  // barriers
  // sdp_* and pds_* exist twice (index = batch & 1): S/dP of batch n+1 are computed while the soft-max warps still
  // hold batch n, and P/dS of batch n+1 are written while dV/dK of batch n still read theirs
  const uint32_t full0 = bar_base, empty0 = bar_base + 16, kv_bar = bar_base + 32, sdp_full = bar_base + 40,
                 sdp_free = bar_base + 56, pds_full = bar_base + 72, pds_free = bar_base + 88, acc_full = bar_base + 104,
                 tmem_slot = bar_base + 112, dq_full = bar_base + 120, dq_free = bar_base + 128, stg_full = bar_base + 136,
                 stg_free = bar_base + 144, s_full = bar_base + 160, p_full = bar_base + 176;   // stg_free: two barriers, one per P/dS pair
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + 8 * i, kProd);
      mbar_init(empty0 + 8 * i, 1);
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
    mbar_init(dq_full, 1);
    mbar_init(dq_free, kDrainThreads);
    mbar_init(stg_full, kDrainThreads);
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
    // boxes.  Box x = 2 * lane + warp belongs to this lane; every producer warp issues its eight with a single instruction
    // and arms the stage's barrier with their byte count.  Token ids are fetched one batch ahead.
    if (warp == 0 && lane == 0 && nb > 0) {
      mbar_expect_tx(kv_bar, 2 * KV_TILE);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        tma_load_4d(k_s + p * KV_PANEL, &tmK, kv_bar, p * 64, hk, key0, b);
        tma_load_4d(v_s + p * KV_PANEL, &tmV, kv_bar, p * 64, hk, key0, b);
      }
    }
    const int x = kProd * lane + warp;          // this lane's box of every batch (none if >= 16)
    const bool has = x < 2 * kTokB;
    const int bj = x & 7, bwhich = x >> 3;
    const int nmine = 2 * kTokB / kProd;   // boxes this warp issues per batch
    auto batch_token = [&](int n) { return n >= nb || !has ? 0 : list_token(n % nb_sub * kTokB + bj); };
    int tk_next = batch_token(0);
    for (int n = 0; n < nb; ++n) {
      const int tk = tk_next;
      tk_next = batch_token(n + 1);
      const int hg = hk * G16 + n / nb_sub;
      const int stage = n % kStages;
      const uint32_t ph = (n / kStages) & 1;
      const uint32_t fb = full0 + 8 * stage;
      int good = 1;
      if (lane == 0) {
        good = mbar_wait(empty0 + 8 * stage, ph ^ 1, DEV_ERR_EMPTY_WAIT) ? 1 : 0;
        if (good) mbar_expect_tx(fb, nmine * 4096);
      }
      if (!__shfl_sync(0xffffffffu, good, 0)) break;
      if (has) {
        const uint32_t q_s = ring + stage * STAGE, do_s = q_s + Q_TILE;
        const int qrow = (int)(((long long)b * a.Tq + (tk - a.q0)) * a.Hq + hg * 16);
        tma_load_4d((bwhich ? do_s : q_s) + bj * 4096, bwhich ? &tmDO : &tmQ, fb, 0, 0, 0, qrow >> 3);
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------- MMA issuer A: S and dP ----------------------------------------
    // S/dP of batch n is issued as soon as its Q/dO stage has landed and its TMEM buffer is free (the soft-max warps
    // hold batch n-2 in registers), i.e. ahead of dV/dK of batch n-1, which the second issuer handles.
    if (lane == 0 && nb > 0) {
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
        ok = mbar_wait(full0 + 8 * (n % kStages), (n / kStages) & 1, DEV_ERR_FULL_WAIT);
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
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t aoff = (ks >> 2) * 1024 + (ks & 3) * 32, boff = (ks >> 2) * KV_PANEL + (ks & 3) * 32;
          umma_ss(tmem + col + 64, umma_desc_advance(ado, aoff), umma_desc_advance(dV, boff), idesc_kk, ks ? 1u : 0u);
        }
        umma_commit(sdp_full + 8 * (n & 1));
      }
    }
  } else if (warp == kMma2Warp) {
    // ------------------------------- MMA issuer B: dV, dK, dQ partials -----------------------------
    if (lane == 0 && nb > 0) {
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
        ok = mbar_wait(p_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint64_t aq = (n % kStages) ? dQmn[1] : dQmn[0], ado = (n % kStages) ? dDOmn[1] : dDOmn[0];
        const uint64_t bp = (n & 1) ? dP[1] : dP[0], bds = (n & 1) ? dDS[1] : dDS[0];
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)   // contraction over the 128 rows, 16 per step; dV while the soft-max warps form dS
          umma_ss(tmem + kColDV, umma_desc_advance(ado, ks * 4096), umma_desc_advance(bp, ks * 2048), idesc_mn, (n | ks) ? 1u : 0u);
        ok = mbar_wait(pds_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_ss(tmem + kColDK, umma_desc_advance(aq, ks * 4096), umma_desc_advance(bds, ks * 2048), idesc_mn, (n | ks) ? 1u : 0u);
        umma_commit(empty0 + 8 * (n % kStages));
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
    if (emit_dq) {
      const int quad = warp & 3;
      const int row = 32 * quad + lane;
      const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
      const bool elected = warp == kDrainWarp && lane == 0;
      bool ok = true;
      for (int n = 0; ok && n < nb; ++n) {
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
        mbar_arrive(stg_full);
        if (elected) {
          ok = mbar_wait(stg_full, n & 1, DEV_ERR_FULL_WAIT);
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
    const int j = row >> 4, head = row & 15;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const float sl2 = a.scale * kLog2e;
    bool ok = true;
    // per-row operands are fetched one batch ahead (token ids two ahead) so their latency hides behind the MMAs; they are kept
    // as loaded, since converting them would wait for the loads
    struct RowInfo {
      int t;
      bool live;
      float lse, del;
      bf16 g;
    };
    auto row_token = [&](int n, bool& live) {
      live = false;
      if (n >= nb) return 0;
      const int i = n % nb_sub * kTokB + j;
      live = i < nA;
      return list_token(i);
    };
    auto row_load = [&](int n, int t, bool live) {
      RowInfo r = {t, live, 0.f, 0.f, __float2bfloat16(1.f)};
      if (n < nb) {
        const long long qrow = ((long long)b * a.Tq + (t - a.q0)) * a.Hq + (hk * G16 + n / nb_sub) * 16 + head;
        r.lse = a.lse[qrow];
        r.del = a.delta[qrow];
        if (a.gate) r.g = a.gate[qrow];
      }
      return r;
    };
    // With dQ partials: the drain warps stage the partial of batch n in that batch's own P/dS pair; the pair is written again
    // for batch n+2 only after their bulk store has read it (stg_free of that pair).
    bool live1;
    int t1 = row_token(0, live1);
    RowInfo cur = row_load(0, t1, live1);
    t1 = row_token(1, live1);
    for (int n = 0; ok && n < nb; ++n) {
      const RowInfo ri = cur;
      cur = row_load(n + 1, t1, live1);     // operands of batch n+1
      t1 = row_token(n + 2, live1);         // token id of batch n+2
      const int t = ri.t;
      const bool live = ri.live;

      const uint32_t buf = n & 1, use = n >> 1;
      const uint32_t tcol = buf * 128;
      ok = mbar_wait(s_full + 8 * buf, use & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      float p[32];
      uint32_t pw[16];   // 32 bf16
      tmem_ld16(tmem + lane_addr + tcol + half * 32, *reinterpret_cast<float(*)[16]>(&p[0]));
      tmem_ld16(tmem + lane_addr + tcol + half * 32 + 16, *reinterpret_cast<float(*)[16]>(&p[16]));
      tmem_ld_wait();
      const int kfirst = key0 + half * 32, klast = kfirst + 31;
      const float lse2 = ri.lse * kLog2e, del = ri.del, gv = __bfloat162float(ri.g);
      const bool dead = !live || !(lse2 > -INFINITY);
      if (dead) {
#pragma unroll
        for (int e = 0; e < 32; ++e) p[e] = 0.f;
      } else if (klast <= t) {
        const float nl = -lse2;
#pragma unroll
        for (int e = 0; e < 32; ++e) p[e] = ex2(fmaf(p[e], sl2, nl));
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) p[e] = kfirst + e <= t ? ex2(p[e] * sl2 - lse2) : 0.f;
      }
#pragma unroll
      for (int e = 0; e < 32; e += 2) pw[e / 2] = pack_bf16(p[e] * gv, p[e + 1] * gv);
      if (n >= 2) {
        ok = mbar_wait(pds_free + 8 * buf, (use - 1) & 1, DEV_ERR_EMPTY_WAIT);   // dV/dK of batch n-2 have read this pair
        if (!ok) break;
      }
      if (emit_dq && n >= 2) {
        ok = mbar_wait(stg_free + 8 * buf, (use - 1) & 1, DEV_ERR_EMPTY_WAIT);
        if (!ok) break;
      }
      // this thread's half of row `row` of the [128 x 64] bf16 tiles: 4 chunks of 16 bytes at swizzled positions
      uint8_t* prow = sgen + (p_s0 - sbase) + buf * 2 * P_TILE + row * 128;
      uint8_t* drow = prow + P_TILE;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(prow + ((4 * half + c) ^ (row & 7)) * 16) = make_uint4(pw[4 * c], pw[4 * c + 1], pw[4 * c + 2], pw[4 * c + 3]);
      fence_proxy_async();
      mbar_arrive(p_full + 8 * buf);
      ok = mbar_wait(sdp_full + 8 * buf, use & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      float dpv[32];
      tmem_ld16(tmem + lane_addr + tcol + 64 + half * 32, *reinterpret_cast<float(*)[16]>(&dpv[0]));
      tmem_ld16(tmem + lane_addr + tcol + 64 + half * 32 + 16, *reinterpret_cast<float(*)[16]>(&dpv[16]));
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(sdp_free + 8 * buf);   // S and dP are in registers: batch n+2 may overwrite this TMEM buffer
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const uint32_t d2 = pack_bf16(p[e] * fmaf(gv, dpv[e], -del), p[e + 1] * fmaf(gv, dpv[e + 1], -del));
        pw[e / 2] = dead ? 0u : d2;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(drow + ((4 * half + c) ^ (row & 7)) * 16) = make_uint4(pw[4 * c], pw[4 * c + 1], pw[4 * c + 2], pw[4 * c + 3]);
      fence_proxy_async();
      mbar_arrive(pds_full + 8 * buf);
    }
    // ---- epilogue: dV^T / dK^T [d lanes x 64 key columns] -> global ---------------------------------------
    if (ok && nb > 0) ok = mbar_wait(acc_full, 0, DEV_ERR_FULL_WAIT);
    tc_fence_after();
    const int dch = row;  // channel owned by this thread
    {
      const int which = half;   // half 0 stores dV, half 1 dK
      const float mul = which ? a.scale : 1.f;
      const long long Nout = (long long)a.B * a.T * a.Hk * D;
      float* part = a.part + (which ? 0 : a.slabs * Nout);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float vals[16];
        if (nb > 0) {
          tmem_ld16(tmem + lane_addr + kColDV + which * 64 + c * 16, vals);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) vals[e] = 0.f;
        }
        float add[16];   // the window's part
#pragma unroll
        for (int e = 0; e < 16; ++e) add[e] = 0.f;
        for (int w = 0; a.nshare == 1 && w < a.nadd; ++w) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int kp = key0 + c * 16 + e;
            if (kp < a.T) add[e] += part[w * Nout + (((long long)b * a.T + kp) * a.Hk + hk) * D + dch];
          }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const int kp = key0 + c * 16 + e;
          if (!ok || kp >= a.T) continue;
          const long long off = (((long long)b * a.T + kp) * a.Hk + hk) * D + dch;
          if (a.nshare > 1)
            part[seg * Nout + off] = vals[e] * mul;
          else
            (which ? a.dk : a.dv)[off] = __float2bfloat16(fmaf(vals[e], mul, add[e]));
        }
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
  kv_bwd_tc_kernel<<<(unsigned)grid, kThreads, kSmem, s>>>(tmQ, tmDO, tmK, tmV, a);
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
