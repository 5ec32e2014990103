// Selected attention forward, key-major on tcgen05 (head_dim 128, 64-key blocks, 16 query heads per group).
// Same results as the query-major kernel (nsa/selection_attn.py:401-517: every query attends to the keys k <= t of
// its selected blocks), different decomposition: the 16 heads of one query are the only rows that share a gathered
// block, too few for a tensor-core tile, so here a CTA owns one 64-key block and the QUERIES that selected it arrive in
// batches of 8 tokens x 16 heads = 128 rows (the block's ascending token list from the reverse index).  Per batch:
//     S     [128 rows x 64 keys] = Qg . K^T     A = Qg (K-major, gathered by TMA), B = K (K-major)
//     O_part[128 rows x 128 d  ] = P . V        A = P (tensor memory, written by the soft-max warps), B = V (MN-major)
// with P = exp(scale S - m), m the row's maximum over the block's visible keys.  The visit leaves (m, l = sum P) per
// row and O_part as a [16 heads x D] bf16 tile at the visit's position in the reverse-index list; a second kernel
// merges a token's visits in slot order (fixed order, no atomics):  o = sum_v 2^(m_v - M) O_v / sum_v 2^(m_v - M) l_v.
// K and V of a block are read once per CTA instead of once per visiting query (32 KB per visit in the query-major
// kernel, which is bound by that gather).
// Roles (512 threads): warps 0-1 TMA producers (4-stage ring of 32 KB Q tiles; a stage is free as soon as its score MMAs
// have completed), warps 2 and 3 issue S and P.V, warps 4-7 / 8-11 two soft-max groups (even / odd batches, one
// row per thread), warps 12-15 read O_part out of tensor memory into a staging tile that one bulk store writes.
// Every wait is bounded; on a time-out the role records an error and leaves its loop.
#include <algorithm>
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int D = 128;
constexpr int kProd = 2;
constexpr int kMmaWarp = kProd;             // issues S
constexpr int kMma2Warp = kProd + 1;        // issues P.V
constexpr int kSoftWarp = kProd + 2;        // 8 soft-max warps: two groups of four
constexpr int kDrainWarp = kSoftWarp + 8;   // 4 drain warps
constexpr int kThreads = (kDrainWarp + 4) * 32;
constexpr int kTokB = 8;
constexpr uint32_t KV_PANEL = 64 * 128;     // [64 keys][64 ch]
constexpr uint32_t KV_TILE = 2 * KV_PANEL;  // 16 KB
constexpr uint32_t Q_TILE = 128 * 256;       // 32 KB: [16 row groups][2 column panels][8 rows][128 B]
constexpr uint32_t STG_TILE = 128 * 256;    // [128 rows][128 d] bf16
constexpr int kStages = 4;
constexpr uint32_t kSmem = 2 * KV_TILE + kStages * Q_TILE + 2 * STG_TILE + 256 + 1024;
constexpr uint32_t kTmemCols = 512;         // S: 0..63 | 64..127; O_part: 128..255 | 256..383; P: 384..415 | 416..447
constexpr uint32_t kColO = 128, kColP = 384;

__global__ void __launch_bounds__(kThreads, 1)
    sel_fwd_kv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const SelKvArgs a, const int nshare, const int nfirst) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t k_s = sbase, v_s = sbase + KV_TILE;
  const uint32_t ring = sbase + 2 * KV_TILE;
  const uint32_t stg = ring + kStages * Q_TILE;
  const uint32_t bar_base = stg + 2 * STG_TILE;
  // barriers (8 bytes each); the double ones are indexed by batch & 1
  const uint32_t full0 = bar_base, empty0 = bar_base + 32, kv_bar = bar_base + 64, s_full = bar_base + 72,
                 s_free = bar_base + 88, p_full = bar_base + 104, p_free = bar_base + 120, o_full = bar_base + 136,
                 o_free = bar_base + 152, stg_full = bar_base + 168, stg_free = bar_base + 184, tmem_slot = bar_base + 200;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + 8 * i, kProd);
      mbar_init(empty0 + 8 * i, 1);
    }
    mbar_init(kv_bar, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full + 8 * i, 1);
      mbar_init(s_free + 8 * i, 128);
      mbar_init(p_full + 8 * i, 128);
      mbar_init(p_free + 8 * i, 1);
      mbar_init(o_full + 8 * i, 1);
      mbar_init(o_free + 8 * i, 128);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(stg_full + 8 * i, 128);
      mbar_init(stg_free + 8 * i, 1);
    }
    fence_mbar_init();
  }
  if (warp == kMmaWarp) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));

  // ---- work item: (batch, kv head)-major so the resident CTAs share one head group's Q rows in L2; shares of a block's
  // list block-major, longest lists first (there are few enough of them for all of Q to stay in L2); nfirst > 0: shares of
  // every head group's first block before the other blocks --------------------------------------------------------------
  const int G16 = (a.Hq / a.Hk) / 16;
  const int NB = (a.T + 63) / 64;
  const int BH = a.B * a.Hk;
  int nseg = nshare, seg = (int)(blockIdx.x % nshare), item = (int)(blockIdx.x / nshare);
  int blk = nshare > 1 ? item / BH : item % NB, bh = nshare > 1 ? item % BH : item / NB;
  if (nfirst > 0) {   // (nshare = 1)
    if (item < BH * nfirst) {
      nseg = nfirst;
      seg = item % nfirst;
      blk = 0;
      bh = item / nfirst;
    } else {
      item -= BH * nfirst;
      blk = 1 + item % (NB - 1);
      bh = item / (NB - 1);
    }
  }
  const int b = bh / a.Hk, hk = bh % a.Hk;
  const int* rp = a.rev_ptr + (long long)bh * (NB + 1);
  int ta_lo = rp[blk], nA = rp[blk + 1] - ta_lo;
  if (nseg > 1) {   // this CTA's share of the list, in whole batches
    const int ba = (nA + kTokB - 1) / kTokB;
    const int a0 = (int)((long long)ba * seg / nseg) * kTokB, a1 = min(nA, (int)((long long)ba * (seg + 1) / nseg) * kTokB);
    ta_lo += a0;
    nA = a1 - a0;
  }
  const int* list = a.rev_tok + (long long)bh * a.rev_cap + ta_lo;
  const int key0 = blk * 64;
  const int nb_sub = (nA + kTokB - 1) / kTokB;
  const int nb = nb_sub * G16;   // batches of this CTA (0: nothing selected this block)
  auto token = [&](int i) { return list[min(i, nA - 1)]; };

  if (nb > 0 && warp < kProd) {
    // ------------------------------- TMA producers ------------------------------------------------------------
    // a batch is 8 boxes of 4 KB, one per token: the token's [16 heads x 128 d] rows through a 4-D view of q
    // (64 columns, 8 rows, 2 column panels, row groups) land as [row group][panel][8 rows][128 B], so the 8-row swizzle
    // atoms of one panel sit 2 KB apart over the whole tile (SBO = 2048, second panel at +1 KB).  One box per token
    // instead of one per (token, panel): the gather is bound by the number of boxes.  Lane j finds
    // where the token of the warp's box j is, one lane issues the warp's four
    if (warp == 0 && elect_one()) {
      mbar_expect_tx(kv_bar, 2 * KV_TILE);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        tma_load_4d(k_s + p * KV_PANEL, &tmK, kv_bar, p * 64, hk, key0, b);
        tma_load_4d(v_s + p * KV_PANEL, &tmV, kv_bar, p * 64, hk, key0, b);
      }
    }
    const int x = kProd * lane + warp;
    const bool has = x < kTokB;
    const int bj = x;
    constexpr int kMine = kTokB / kProd;   // boxes of this warp
    int tk_next = has ? token(bj) : 0;
    for (int n = 0; n < nb; ++n) {
      const int tk = tk_next;
      const int m1 = (n + 1) % nb_sub;
      tk_next = (has && n + 1 < nb) ? token(m1 * kTokB + bj) : 0;
      const int sub = n / nb_sub;
      const int hg = hk * G16 + sub;
      const int stage = n % kStages;
      const uint32_t ph = (n / kStages) & 1;
      const uint32_t fb = full0 + 8 * stage;
      const int grp = (int)((((long long)b * a.Tq + (tk - a.q0)) * a.Hq + hg * 16) >> 3);
      int row_group[kMine];
#pragma unroll
      for (int j = 0; j < kMine; ++j) row_group[j] = __shfl_sync(0xffffffffu, grp, j);
      const bool good = mbar_wait(empty0 + 8 * stage, ph ^ 1, DEV_ERR_EMPTY_WAIT);
      if (!__all_sync(0xffffffffu, good)) break;
      if (elect_one()) {
        mbar_expect_tx(fb, kMine * 4096);
#pragma unroll
        for (int j = 0; j < kMine; ++j)
          tma_load_4d(ring + stage * Q_TILE + (kProd * j + warp) * 4096, &tmQ, fb, 0, 0, 0, row_group[j]);
      }
    }
  } else if (nb > 0 && warp == kMmaWarp) {
    // ------------------------------- MMA issuer A: S ------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, 0, 0);    // both operands K-major
      bool ok = mbar_wait(kv_bar, 0, DEV_ERR_FULL_WAIT);
      const uint64_t dK = umma_smem_desc(k_s, 0, 1024), dQ0 = umma_smem_desc(ring, 0, 2048);
      for (int n = 0; ok && n < nb; ++n) {
        const int st = n % kStages;
        ok = mbar_wait(full0 + 8 * st, (n / kStages) & 1, DEV_ERR_FULL_WAIT) &&
             (n < 2 || mbar_wait(s_free + 8 * (n & 1), ((n >> 1) - 1) & 1, DEV_ERR_EMPTY_WAIT));
        if (!ok) break;
        tc_fence_after();
        const uint64_t aq = umma_desc_advance(dQ0, st * Q_TILE);
        const uint32_t col = (n & 1) * 64;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t aoff = (ks >> 2) * 1024 + (ks & 3) * 32, boff = (ks >> 2) * KV_PANEL + (ks & 3) * 32;
          umma_ss(tmem + col, umma_desc_advance(aq, aoff), umma_desc_advance(dK, boff), idesc_s, ks ? 1u : 0u);
        }
        umma_commit(s_full + 8 * (n & 1));
        umma_commit(empty0 + 8 * st);          // the Q tile is only needed for the scores
      }
    }
  } else if (nb > 0 && warp == kMma2Warp) {
    // ------------------------------- MMA issuer B: P.V ----------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, 128, 0, 1);   // A = P in tensor memory, B = V MN-major
      bool ok = mbar_wait(kv_bar, 0, DEV_ERR_FULL_WAIT);
      const uint64_t dVmn = umma_smem_desc(v_s, KV_PANEL, 1024);
      for (int n = 0; ok && n < nb; ++n) {
        ok = mbar_wait(p_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT) &&
             (n < 2 || mbar_wait(o_free + 8 * (n & 1), ((n >> 1) - 1) & 1, DEV_ERR_EMPTY_WAIT));
        if (!ok) break;
        tc_fence_after();
        const uint32_t ap = tmem + kColP + (n & 1) * 32;   // 16 keys = 8 packed columns per step
        const uint32_t col = kColO + (n & 1) * 128;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)   // contraction over the 64 keys, 16 per step
          umma_ts(tmem + col, ap + ks * 8, umma_desc_advance(dVmn, ks * 2048), idesc_o, ks ? 1u : 0u);
        umma_commit(o_full + 8 * (n & 1));
        umma_commit(p_free + 8 * (n & 1));
      }
    }
  } else if (nb > 0 && warp >= kDrainWarp) {
    // ------------------------------- drain warps: O_part, one row per thread -----------------------------------
    // accumulator -> bf16 -> staging tile (128 rows x 256 bytes; within a 128-byte half row the 16-byte chunk c sits at
    // position c ^ (row & 7): conflict-free writes, undone by the merge kernel) -> one bulk store: the batch's 8 tiles
    // are consecutive list positions, contiguous in the partial buffer when the KV head has one 16-head group
    const int quad = warp & 3;
    const int row = 32 * quad + lane;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    bool ok = true;
    for (int n = 0; ok && n < nb; ++n) {
      const int sub = n / nb_sub, mloc = n % nb_sub;
      ok = mbar_wait(o_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
      // the store of batch n-2 has read this staging tile
      if (ok && n >= 2) ok = mbar_wait(stg_free + 8 * (n & 1), ((n >> 1) - 1) & 1, DEV_ERR_EMPTY_WAIT);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sb = stg + (uint32_t)(n & 1) * STG_TILE;
      uint8_t* sp = sgen + (sb - sbase) + row * 256;
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {   // 32 columns at a time
        float vals[2][16];
        tmem_ld16(tmem + lane_addr + kColO + (n & 1) * 128 + q4 * 32, vals[0]);
        tmem_ld16(tmem + lane_addr + kColO + (n & 1) * 128 + q4 * 32 + 16, vals[1]);
        tmem_ld_wait();
        if (q4 == 3) {
          tc_fence_before();
          mbar_arrive(o_free + 8 * (n & 1));   // the accumulator is in registers
        }
#pragma unroll
        for (int c2 = 0; c2 < 4; ++c2) {
          const float* f = &vals[c2 >> 1][(c2 & 1) * 8];
          uint4 o;
          __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int e = 0; e < 4; ++e) ho[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
          const int cc = q4 * 4 + c2;
          *reinterpret_cast<uint4*>(sp + (cc >> 3) * 128 + (((cc & 7) ^ (row & 7)) * 16)) = o;
        }
      }
      fence_proxy_async();
      mbar_arrive(stg_full + 8 * (n & 1));   // (two: of batches 0 and 1 a warp may be at the second before the slowest is through the first)
      if (warp == kDrainWarp) {
        // one 32 KB bulk store (the tokens' tiles are contiguous), or one of 4 KB per token where the KV head has several
        // 16-head groups.  Eight 4 KB stores by eight lanes were no faster than the one (4.31 against 4.20 ms)
        bool good = mbar_wait(stg_full + 8 * (n & 1), (n >> 1) & 1, DEV_ERR_FULL_WAIT);
        const int nvalid = min(kTokB, nA - mloc * kTokB);
        if (good && G16 == 1 && lane == 0 && nvalid > 0) {
          bf16* dst = a.part + (((long long)bh * a.rev_cap + ta_lo + mloc * kTokB) * (16 * D));
          bulk_store_evict_first(dst, sb, (uint32_t)nvalid * 16 * D * 2);
        } else if (good && G16 > 1 && lane < nvalid) {
          bf16* dst = a.part + ((((long long)bh * a.rev_cap + ta_lo + mloc * kTokB + lane) * G16 + sub) * (16 * D));
          bulk_store_evict_first(dst, sb + lane * 16 * D * 2, 16 * D * 2);
        }
        bulk_commit();
        bulk_wait_read_but_one();   // batch n-1's stores have read their tile; this batch's stay in flight
        __syncwarp();
        if (lane == 0 && n > 0) mbar_arrive(stg_free + 8 * ((n - 1) & 1));
        ok = good;
      }
    }
    if (warp == kDrainWarp) bulk_wait_all();
  } else if (nb > 0 && warp >= kSoftWarp) {
    // ------------------------------- soft-max warps: one (token, head) row per thread --------------------------
    const int g = (warp - kSoftWarp) >> 2;      // group: batches n = g, g+2, ...
    const int quad = warp & 3;
    const int row = 32 * quad + lane;           // TMEM lane == tile row
    const int j = row >> 4, head = row & 15;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const float sl2 = a.scale * kLog2e;
    bool ok = true;
    int t_next = (g < nb) ? token((g % nb_sub) * kTokB + j) : 0;
    for (int n = g; ok && n < nb; n += 2) {
      const int sub = n / nb_sub, mloc = n % nb_sub;
      const int i = mloc * kTokB + j;
      const bool live = i < nA;
      const int t = t_next;
      if (n + 2 < nb) t_next = token(((n + 2) % nb_sub) * kTokB + j);
      const uint32_t use = n >> 1;
      ok = mbar_wait(s_full + 8 * g, use & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      float sv[64];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(tmem + lane_addr + g * 64 + c * 16, *reinterpret_cast<float(*)[16]>(&sv[16 * c]));
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(s_free + 8 * g);   // S is in registers: batch n+2 may overwrite this buffer
      // visible keys: key0 + c <= t (the block's first key always is, or the token would not be in this list)
      const int nvis = live ? min(64, t - key0 + 1) : 0;
      float m2 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 64; ++c) {
        sv[c] = (c < nvis) ? sv[c] * sl2 : -INFINITY;
        m2 = fmaxf(m2, sv[c]);
      }
      float l = 0.f;
      float pw[32];   // packed pairs
      if (nvis > 0) {
#pragma unroll
        for (int c = 0; c < 64; c += 2) {
          const float p0 = ex2(sv[c] - m2), p1 = ex2(sv[c + 1] - m2);
          const uint32_t pk = pack_bf16(p0, p1);
          pw[c / 2] = __uint_as_float(pk);
          // l is the sum of the rounded probabilities the tensor core multiplies, as in the query-major kernel
          const __nv_bfloat162 pr = *reinterpret_cast<const __nv_bfloat162*>(&pk);
          l += __low2float(pr) + __high2float(pr);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) pw[c] = 0.f;
      }
      if (use >= 1) {
        ok = mbar_wait(p_free + 8 * g, (use - 1) & 1, DEV_ERR_EMPTY_WAIT);   // P.V of batch n-2 has read these columns
        if (!ok) break;
      }
      tc_fence_after();
      const uint32_t p_col = tmem + lane_addr + kColP + g * 32;
      tmem_st16(p_col, *reinterpret_cast<float(*)[16]>(&pw[0]));
      tmem_st16(p_col + 16, *reinterpret_cast<float(*)[16]>(&pw[16]));
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_full + 8 * g);
      if (live) {
        float2* st = reinterpret_cast<float2*>(a.stats) + (((long long)bh * a.rev_cap + ta_lo + i) * G16 + sub) * 16 + head;
        *st = make_float2(m2, l);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemCols);
}

// Two warps per (batch, token, 16-head group), each eight of the 16 heads: the visits' (m, l) and O tiles merged in slot order,
// and the gated sum of the branches.  A load instruction of the warp covers 512 contiguous bytes of a tile.  Bound by reading
// the tiles, so by what a warp has in flight per register: the first tile and the gates are fetched ahead of the maxima.
// All slots visible, 4 x 8192 tokens, 64 heads: 1.41 ms with the gate (6.9 TB/s); half visible, 8 x 8192 tokens, three
// branches: 2.25; one sequence of 5003 tokens: 162 us; 2 x 2080 tokens: 80.  Small blocks at 64 registers keep 32 warps on an
// SM: with eight warps a block at the compiler's 76 registers (24 warps) 1.49 ms, 2.50 ms, 182 us and 85 us; seven blocks of
// four as eight, nine (spilling) 2.32 ms and 167 us.  Four heads per warp, one tile in flight: 2.60 ms and 190 us; more than
// one tile in flight leaves too few warps.
constexpr int kMergeHeads = 8, kMergeWarps = 16 / kMergeHeads, kMergeBlock = 4;   // warps per tile, per block
template <bool SUM>
__global__ void __launch_bounds__(32 * kMergeBlock, 8) sel_fwd_merge_kernel(const RevArgs a, const bf16* __restrict__ part,
                                                            const float* __restrict__ stats, const SelMerge m, const int G16) {
  after_previous();
  constexpr int NV = kMergeHeads * D / 8 / 32;   // 16-byte vectors per lane: 4
  const long long w4 = (long long)blockIdx.x * kMergeBlock + (threadIdx.x >> 5);
  const long long total = (long long)a.B * a.Tq * a.H * G16;
  const long long w = w4 / kMergeWarps;
  if (w >= total) return;
  const int hb = (int)(w4 % kMergeWarps);
  const int lane = threadIdx.x & 31;
  const int sub = (int)(w % G16);
  const long long row = w / G16;   // (b, tl, h) row of idx / counts
  const int h = (int)(row % a.H);
  const long long bt = row / a.H;
  const int tl = (int)(bt % a.Tq), b = (int)(bt / a.Tq);
  const long long bh = (long long)b * a.H + h;
  const int mypos = lane < a.S ? a.inv[row * a.S + lane] : -1;   // -1: the slot does not count
  const int Hq = a.H * G16 * 16;
  const long long orow0 = bt * Hq + (long long)(h * G16 + sub) * 16;   // first of the group's 16 (token, head) rows
  const int myhead = hb * kMergeHeads + lane % kMergeHeads;
  // vector u = 32 i + lane of this part of the tile belongs to head u / 16 = 2 i + lane / 16 (of this warp's); the staging layout
  // swizzles a tile's 16-byte chunks by its row
  int ud[NV];
  const long long vec0 = orow0 * (D / 8) + hb * (kMergeHeads * D / 8);
  bf16 graw[3];   // gates of head lane % 8
#pragma unroll
  for (int x = 0; x < 3; ++x) graw[x] = __float2bfloat16(1.f);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int u = 32 * i + lane;
    ud[i] = ((u & ~7) | ((u & 7) ^ ((hb * kMergeHeads + (u >> 4)) & 7)));
  }
  if (SUM && m.g0) graw[0] = m.g0[orow0 + myhead];
  if (SUM && m.g1) graw[1] = m.g1[orow0 + myhead];
  if (SUM && m.g2) graw[2] = m.g2[orow0 + myhead];
  const unsigned live = __ballot_sync(0xffffffffu, mypos >= 0);
  auto tile_index = [&](int s) {
    const long long pos = __shfl_sync(0xffffffffu, mypos, s);
    return (bh * a.cap + pos) * G16 + sub;
  };
  const uint4* base = reinterpret_cast<const uint4*>(part) + hb * (kMergeHeads * D / 8) + lane;
  unsigned rem = live;
  uint4 v[NV];
  float2 ml;
  auto fetch = [&]() {   // the next slot's tile and (m, l)
    const long long ti = tile_index(__ffs(rem) - 1);
    rem &= rem - 1;
    ml = reinterpret_cast<const float2*>(stats)[ti * 16 + myhead];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = __ldcs(base + ti * (16 * D / 8) + 32 * i);
  };
  if (live) fetch();
  // pass 1: M = max_v m_v per head.  Lane s fetches the maxima of slot s for this warp's heads (all slots at once, instead of
  // one dependent load per slot), a butterfly takes the maximum over the slots, and every lane keeps the value of head
  // lane % 8, the head whose (m, l) it reads in pass 2.
  float mh[kMergeHeads];
#pragma unroll
  for (int e = 0; e < kMergeHeads; ++e) mh[e] = -INFINITY;
  if (mypos >= 0) {
    const float4* sp = reinterpret_cast<const float4*>(stats) + (((bh * a.cap + mypos) * G16 + sub) * 16 + hb * kMergeHeads) / 2;
#pragma unroll
    for (int e = 0; e < kMergeHeads / 2; ++e) {
      const float4 v4 = sp[e];   // (m, l) of two heads
      mh[2 * e] = v4.x;
      mh[2 * e + 1] = v4.z;
    }
  }
#pragma unroll
  for (int e = 0; e < kMergeHeads; ++e)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mh[e] = fmaxf(mh[e], __shfl_xor_sync(0xffffffffu, mh[e], off));
  float M = mh[0];
#pragma unroll
  for (int e = 1; e < kMergeHeads; ++e) M = (lane % kMergeHeads == e) ? mh[e] : M;
  float L = 0.f;
  float acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[i][k] = 0.f;
  for (bool more = live != 0; more;) {
    const float wgt = ex2(ml.x - M);   // lanes 0-7 (and their copies): own head
    L += wgt * ml.y;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const float wi = __shfl_sync(0xffffffffu, wgt, 2 * i + (lane >> 4));
      const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(hv[k]);
        acc[i][2 * k] = fmaf(wi, f.x, acc[i][2 * k]);
        acc[i][2 * k + 1] = fmaf(wi, f.y, acc[i][2 * k + 1]);
      }
    }
    more = rem != 0;
    if (more) fetch();
  }
  const float inv = L > 0.f ? 1.f / L : 0.f;
  if (m.lse && lane < kMergeHeads) m.lse[orow0 + myhead] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -INFINITY;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int hl = 2 * i + (lane >> 4);
    const float ii = __shfl_sync(0xffffffffu, inv, hl);
    uint4 ov;
    __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
    for (int k = 0; k < 4; ++k) ho[k] = __floats2bfloat162_rn(acc[i][2 * k] * ii, acc[i][2 * k + 1] * ii);
    if (m.o) reinterpret_cast<uint4*>(m.o)[vec0 + ud[i]] = ov;
    if (SUM) {   // g0 * (this branch, as rounded) + g1 * a1 + g2 * a2
      float g[3];
#pragma unroll
      for (int x = 0; x < 3; ++x) g[x] = __shfl_sync(0xffffffffu, __bfloat162float(graw[x]), hl);
      uint4 w1 = make_uint4(0u, 0u, 0u, 0u), w2 = w1;
      if (m.a1) w1 = __ldcs(reinterpret_cast<const uint4*>(m.a1) + vec0 + ud[i]);
      if (m.a2) w2 = __ldcs(reinterpret_cast<const uint4*>(m.a2) + vec0 + ud[i]);
      const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&w1);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&w2);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f0 = __bfloat1622float2(ho[k]), f1 = __bfloat1622float2(h1[k]), f2 = __bfloat1622float2(h2[k]);
        ho[k] = __floats2bfloat162_rn(fmaf(g[2], f2.x, fmaf(g[1], f1.x, g[0] * f0.x)), fmaf(g[2], f2.y, fmaf(g[1], f1.y, g[0] * f0.y)));
      }
      reinterpret_cast<uint4*>(m.out)[vec0 + ud[i]] = ov;
    }
  }
}

}  // namespace

bool sel_fwd_kv_supported(const SelKvArgs& a, int Dh) {
  return Dh == 128 && a.BS == 64 && a.S <= 32 && a.Hq % (16 * a.Hk) == 0;
}

int launch_sel_fwd_kv(const SelKvArgs& a, const RevArgs& r, cudaStream_t s) {
  CUtensorMap tmQ, tmK, tmV;
  const long long qrows = (long long)a.B * a.Tq * a.Hq;
  if (qrows > 0x7fffffffLL) {
    set_error("B*T*Hq exceeds the 2^31 rows a TMA coordinate can address");
    return -32;
  }
  // q rows as (64 columns, 8 rows, 2 column panels, groups of 8 rows): one box = 16 rows x 128 columns of one token
  const unsigned long long qd[4] = {64, 8, 2, (unsigned long long)(qrows / 8)};
  const unsigned long long qs[3] = {(unsigned long long)D * 2, 128, (unsigned long long)D * 2 * 8};
  const unsigned qb[4] = {64, 8, 2, 2};
  int rc = make_tmap_generic(&tmQ, a.q, 4, qd, qs, qb);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.k, D, a.Hk, a.T, a.B, 64);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hk, a.T, a.B, 64);
  if (rc) return rc;
  cudaError_t e = cudaFuncSetAttribute(sel_fwd_kv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return (int)e;
  // The first block is visible to every token, the last to few: with few blocks per SM the first one's CTA would be the last to
  // end.  Up to eight CTAs then share a block's list, so that there are three or more per SM, or at least two CTAs up to six
  // blocks per SM (a visit's results have a place of
  // their own, nothing is added up; a CTA's start and end cost about two batches).  One sequence of 5003 tokens, 4 KV heads:
  // 245 us
  // with one CTA a block, 160 / 159 / 169 / 177 with 3 / 4 / 6 / 8 per SM; 2 x 2080 tokens, 2 KV heads: 140, then 76 / 80 /
  // 88 / 89.
  // Two CTAs a block, 4 KV heads: 9000 tokens (564 blocks) 374 -> 308, 14000 tokens (876) 557 -> 494, 17000 tokens (1064) 559
  // -> 616.
  const long long blocks = (long long)a.B * a.Hk * ((a.T + 63) / 64), want = 3LL * num_sms();
  if (blocks <= 0) return 0;
  const int nshare = blocks >= 2 * want ? 1 : (int)std::max(2LL, std::min(8LL, (want + blocks - 1) / blocks));
  // Many blocks: the first one may still be selected by every token (a fixed choice of it is part of the method), a list as long as
  // many others together, and the last head group's would begin last.  It goes first, in shares, about one per SM over the head
  // groups (up to twice as many blocks as a token selects every list is long).  The whole branch, block 0 and 15 drawn ones, 4 KV
  // heads: 4 x 8192 tokens 4.75 -> 3.83 ms, 8 x 8192 8.8 -> 7.9, 65536 14.8 -> 7.5; drawn ones alone 4.07 / 3.98, 7.88 / 7.85.
  const long long BH = (long long)a.B * a.Hk;
  const int nfirst = nshare == 1 && (a.T + 63) / 64 > 2 * a.S ? (int)std::max(2LL, std::min(32LL, (num_sms() + BH - 1) / BH)) : 0;
  const long long grid = nfirst ? blocks + BH * (nfirst - 1) : blocks * nshare;
  if (grid > 0x7fffffffLL) {
    set_error("selected forward: grid too large");
    return -33;
  }
  launch_next(sel_fwd_kv_kernel, (unsigned)grid, kThreads, kSmem, s, tmQ, tmK, tmV, a, nshare, nfirst);
  note_launches(1);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  const int G16 = a.Hq / a.Hk / 16;
  const long long total = (long long)a.B * a.Tq * a.Hk * G16;
  const unsigned nb = (unsigned)((kMergeWarps * total + kMergeBlock - 1) / kMergeBlock);
  if (a.merge.out)
    launch_next(sel_fwd_merge_kernel<true>, nb, 32 * kMergeBlock, 0, s, r, a.part, a.stats, a.merge, G16);
  else
    launch_next(sel_fwd_merge_kernel<false>, nb, 32 * kMergeBlock, 0, s, r, a.part, a.stats, a.merge, G16);
  note_launches(1);
  return (int)cudaGetLastError();
}

int sel_fwd_kv_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
