// dK, dV of the dense branches on tcgen05 (head_dim 64 or 128): sliding-window attention, or compressed attention (dCK, dCV).
// Semantics of parallel_nsa_bwd_kernel_dkv's window half (nsa/selection_attn.py:207-253) and of _attn_bwd_only_dkv
// (nsa/triton_attention.py:219-318).
//
// A CTA owns 128 keys and walks the queries that see them, 8 tokens x 16 heads = [128 x D] tiles of Q and dO.  Keys are the
// rows of every product, so P and dS never leave tensor memory:
//     S^T = K . Q^T,   dP^T = V . dO^T                            (both operands in shared memory)
//     P^T = exp(scale S^T - lse),  dS^T = P^T (g dP^T - delta)    (eight soft-max warps, half a row of 64 queries per thread)
//     dV += (g P^T) . dO,   dK += dS^T . Q                        (A in tensor memory, over the columns it was computed from;
//                                                                  B = dO, Q as MN-major operands)
// Tensor memory is full: S^T / P^T 128 columns, dP^T / dS^T 128, dV and dK 128 each.  So a tile is two halves of 64 queries, each
// with its own group of four soft-max warps: while one group computes, the products of the other run.  One thread issues, per
// half, dV(n), S^T(n+1), which share columns, another dK(n), dP^T(n+1), which share others, so neither pair needs a barrier of
// its own.  A query's lse, delta and gate are columns here: four warps prepare them in shared memory one tile ahead.
//
// Bound: the 48 products of a tile at about 70 cycles (shared memory delivers 320 KB to them and takes 64 KB from TMA): 3300
// cycles per tile.  Tried: whole tiles (32 products): S^T(n+1) waits for P^T(n) and dV(n), 4150; whole tiles with S^T(n+1) over
// dP^T(n) as soon as that is in registers, in one or two issuing threads: 3600.
// Window, 8 x 8192 tokens, 64 heads, 4 KV heads, window 512: 3670 us (64-key CTAs, below) -> 2260; compressed 1900 -> 1270;
// 32768 tokens, compressed 3700 -> 1970; 1024 tokens, head_dim 64 (mma.sync before), compressed 654 -> 23.  Products issued
// under elect_one instead of a lane number, so that issuing is no longer what takes the time: both together 4.11 -> 3.53 ms at
// 8 x 8192 tokens (below full clocks), 128 -> 107 us at 2 x 2080 tokens, 32 heads.
// At head_dim 64 they stay under the lane number: elected 8 x 4096 tokens, 64 heads, window 925 -> 1046 us, compressed 355 -> 382.
// The keys of a 64-row CTA with P and dS in shared memory (this kernel's predecessor, still the selected branch's) took the same
// number of products for half the keys.
//
// The window's tiles are dealt one per CTA; the tiles start at different places of their query range so that CTAs running side
// by side read the same query tile at the same time (each is read by 5 key tiles with a window of 512; walked from their own
// starts the CTAs would be 16 tiles apart and re-read from DRAM).  The compressed branch's long ranges are cut into segments
// (fp32 slabs, added in a fixed order), all key tiles of a segment side by side.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kTok = 8;
constexpr int kThreads = 512;                 // warp 0 TMA K, Q; 1 S^T, dV; 2 dP^T, dK; 3 TMA V, dO; 4-11 soft-max; 12-15 row data
constexpr int kSoft = 256;
constexpr int kRow = 128;
constexpr uint32_t PANEL = 128 * 128;         // [128 rows][64 columns] bf16
constexpr int QST = 3, DST = 2;               // slots of Q (held until dK) and of dO
constexpr uint32_t kRowStage = 128 * 4 + 128 * 4 + 128 * 2;   // -lse (log2), -delta, gate (bf16) of a tile's 128 rows
constexpr uint32_t kBars = 256;
template <int D>
constexpr uint32_t kSmem = (D / 64) * PANEL * (2 + QST + DST) + 2 * kRowStage + kBars;   // 227 KB at D = 128: no room to align
constexpr uint32_t kTmemCols = 512;           // S^T / P^T 0.., dP^T / dS^T 128.., dV 256.., dK 256 + D..

struct Item {
  long long row0, out_row;   // first query row of the sequence; output row of the tile's first key
  int hk, b, key0, keys;     // KV head, sequence, first key (position in its sequence) and keys of the tile
  int Tq, qlo, n, shift;     // query rows of the sequence; query tiles qlo .. qlo+n-1, walked from `shift` on
  int slab;
};

__device__ __forceinline__ bool decode_item(const DenseKvArgs& a, Item& it) {
  int i = blockIdx.x, sp = 0;
  if (a.mode == 0) {
    sp = i % a.nslab;
    i /= a.nslab;
  }
  const int per = (a.Lk + 127) / 128;
  const int tile = i % per;
  i /= per;
  it.hk = i % a.Hk;
  i /= a.Hk;
  it.b = i % a.seq.B;
  if (a.mode == 1) sp = a.nslab - 1 - i / a.seq.B;
  it.row0 = (long long)it.b * a.seq.Tq;
  it.Tq = a.seq.Tq;
  it.key0 = tile * 128;
  it.out_row = (long long)it.b * a.Lk + it.key0;
  it.keys = min(128, a.Lk - it.key0);
  it.slab = sp;
  long long lo, hi;   // query rows that see one of the keys
  if (a.mode == 0) {
    lo = it.key0 - a.seq.q0;
    hi = (long long)it.key0 + it.keys - 1 + a.window - a.seq.q0;
  } else {
    const long long first = a.causal ? (long long)it.key0 * a.cstride + a.cblock - a.seq.q0 : 0;
    lo = max(first, (long long)sp * a.seg_len);
    hi = (long long)(sp + 1) * a.seg_len;
  }
  lo = max(lo, 0LL);
  hi = min(hi, (long long)it.Tq);
  it.qlo = (int)lo / kTok;
  it.n = hi > lo ? ((int)hi + kTok - 1) / kTok - it.qlo : 0;
  it.shift = 0;
  if (a.mode == 0) {
    const int b0 = (int)((long long)it.n * sp / a.nslab), b1 = (int)((long long)it.n * (sp + 1) / a.nslab);
    it.qlo += b0;
    it.n = b1 - b0;
    if (it.n > 0) it.shift = (it.n - it.qlo % it.n) % it.n;
  } else if (it.n == 0 && a.part) {
    return false;   // a segment that sees nothing of the tile: the reduction skips it too
  }
  return true;
}

template <int D, bool BYSEQ>   // BYSEQ: the query rows come by sequence (see launch)
__global__ void __launch_bounds__(kThreads, 1)
    dense_kv_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                       const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const DenseKvArgs a) {
  after_previous();
  constexpr int NP = D / 64;
  constexpr uint32_t TILE = NP * PANEL;
  constexpr uint32_t kColDV = 256, kColDK = 256 + D;
  extern __shared__ __align__(1024) uint8_t dense_kv_smem[];
  const uint32_t sbase = smem_u32(dense_kv_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (sbase & 1023u) {   // the 128-byte swizzle repeats every 1024 bytes
    if (threadIdx.x == 0) atomicCAS(&g_dev_error, 0, 330);
    return;
  }
  Item it;
  if (!decode_item(a, it)) return;
  const uint32_t k_s = sbase, v_s = sbase + TILE, q_ring = sbase + 2 * TILE, do_ring = q_ring + QST * TILE;
  const uint32_t rows_s = do_ring + DST * TILE, bars = rows_s + 2 * kRowStage;
  const uint32_t k_full = bars, v_full = bars + 8, q_full0 = bars + 16, q_empty0 = bars + 40, do_full0 = bars + 64,
                 do_empty0 = bars + 80, row_full0 = bars + 96, row_empty0 = bars + 112, s_full0 = bars + 128, p_full0 = bars + 144,
                 dp_full0 = bars + 160, ds_full0 = bars + 176, acc_full = bars + 192, tmem_slot = bars + 200;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(dense_kv_smem + (bars - sbase) + 208);
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int i = 0; i < QST; ++i) {
      mbar_init(q_full0 + 8 * i, 1);
      mbar_init(q_empty0 + 8 * i, 1);
    }
    for (int i = 0; i < DST; ++i) {
      mbar_init(do_full0 + 8 * i, 1);
      mbar_init(do_empty0 + 8 * i, 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(row_full0 + 8 * i, kRow);
      mbar_init(row_empty0 + 8 * i, kSoft);
      mbar_init(s_full0 + 8 * i, 1);
      mbar_init(p_full0 + 8 * i, kSoft / 2);
      mbar_init(dp_full0 + 8 * i, 1);
      mbar_init(ds_full0 + 8 * i, kSoft / 2);
    }
    mbar_init(acc_full, 2);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(dense_kv_smem + (tmem_slot - sbase));

  const int G16 = (a.Hq / a.Hk) / 16;
  const int N = it.n * G16;   // query tiles, one 16-head group of the KV head after the other
  auto tile_of = [&](int c, int& hg) {   // first query row of the c-th tile
    const int sub = c / it.n;
    int s = c - sub * it.n + it.shift;
    if (s >= it.n) s -= it.n;
    hg = it.hk * G16 + sub;
    return (it.qlo + s) * kTok;
  };

  // Registers: 512 threads are launched with 128 each (65536); 128 x 64 + 256 x 168 + 128 x 48 = 57344 (an inc that the launch
  // pool cannot satisfy blocks for ever).
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 0 || warp == 3) {
      // ------------------------------- TMA producers: K and Q (warp 0), V and dO (warp 3) --------------------
      const bool is_k = warp == 0;
      const uint32_t full0 = is_k ? q_full0 : do_full0, empty0 = is_k ? q_empty0 : do_empty0, ring = is_k ? q_ring : do_ring;
      const uint32_t nst = is_k ? QST : DST;
      const CUtensorMap* tmX = is_k ? &tmQ : &tmDO;
      if (N > 0 && elect_one()) {
        mbar_expect_tx(is_k ? k_full : v_full, TILE);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d((is_k ? k_s : v_s) + p * PANEL, is_k ? &tmK : &tmV, is_k ? k_full : v_full, p * 64, it.hk, it.key0, it.b);
        for (int c = 0; c < N; ++c) {
          int hg;
          const int t0 = tile_of(c, hg);
          const uint32_t sl = c % nst;
          if (!mbar_wait_abortable(empty0 + 8 * sl, ((c / nst) & 1) ^ 1, 331, abort_flag)) break;
          mbar_expect_tx(full0 + 8 * sl, TILE);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            if (BYSEQ)
              tma_load_4d(ring + sl * TILE + p * PANEL, tmX, full0 + 8 * sl, p * 64, hg * 16, t0, it.b);
            else
              tma_load_3d(ring + sl * TILE + p * PANEL, tmX, full0 + 8 * sl, p * 64, hg * 16, (int)it.row0 + t0);
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer: dV(n), S^T(n+1) -----------------------------------------
      if (N > 0 && (D == 64 ? lane == 0 : elect_one())) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, 0, 0), idesc_dv = umma_idesc_bf16(128, D, 0, 1);
        const uint64_t dk = umma_smem_desc(k_s, 0, 1024), dq_base = umma_smem_desc(q_ring, 0, 1024);
        const uint64_t ddo_base = umma_smem_desc(do_ring, PANEL, 1024);
        auto issue_s = [&](int c, int h) {
          const uint64_t dq = umma_desc_advance(dq_base, (c % QST) * TILE + h * 8192);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks >> 2) * PANEL + (ks & 3) * 32;
            umma_ss(tmem + h * 64, umma_desc_advance(dk, off), umma_desc_advance(dq, off), idesc_s, ks ? 1u : 0u);
          }
          umma_commit(s_full0 + 8 * h);
        };
        bool ok = mbar_wait_abortable(k_full, 0, 332, abort_flag) && mbar_wait_abortable(q_full0, 0, 333, abort_flag);
        if (ok) {
          tc_fence_after();
          issue_s(0, 0);
          issue_s(0, 1);
        }
        for (int c = 0; ok && c < N; ++c) {
          const uint32_t sl = c % DST;
          ok = mbar_wait_abortable(do_full0 + 8 * sl, (c / DST) & 1, 334, abort_flag);
          if (ok && c + 1 < N) ok = mbar_wait_abortable(q_full0 + 8 * ((c + 1) % QST), ((c + 1) / QST) & 1, 336, abort_flag);
          const uint64_t ddo = umma_desc_advance(ddo_base, sl * TILE);
          for (int h = 0; ok && h < 2; ++h) {
            ok = mbar_wait_abortable(p_full0 + 8 * h, c & 1, 335, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)   // 16 queries = 8 packed columns per step
              umma_ts(tmem + kColDV, tmem + h * 64 + ks * 8, umma_desc_advance(ddo, (4 * h + ks) * 2048), idesc_dv, (c | h | ks) ? 1u : 0u);
            if (h == 1) umma_commit(do_empty0 + 8 * sl);
            if (c + 1 < N) issue_s(c + 1, h);
          }
        }
        umma_commit(acc_full);
      }
    } else {
      // ------------------------------- MMA issuer: dK(n), dP^T(n+1) ----------------------------------------
      if (N > 0 && (D == 64 ? lane == 0 : elect_one())) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, 0, 0), idesc_dk = umma_idesc_bf16(128, D, 0, 1);
        const uint64_t dv = umma_smem_desc(v_s, 0, 1024), ddo_base = umma_smem_desc(do_ring, 0, 1024);
        const uint64_t dq_base = umma_smem_desc(q_ring, PANEL, 1024);
        auto issue_dp = [&](int c, int h) {
          const uint64_t ddo = umma_desc_advance(ddo_base, (c % DST) * TILE + h * 8192);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks >> 2) * PANEL + (ks & 3) * 32;
            umma_ss(tmem + 128 + h * 64, umma_desc_advance(dv, off), umma_desc_advance(ddo, off), idesc_s, ks ? 1u : 0u);
          }
          umma_commit(dp_full0 + 8 * h);
          if (h == 1) umma_commit(do_empty0 + 8 * (c % DST));
        };
        bool ok = mbar_wait_abortable(v_full, 0, 337, abort_flag) && mbar_wait_abortable(do_full0, 0, 338, abort_flag);
        if (ok) {
          tc_fence_after();
          issue_dp(0, 0);
          issue_dp(0, 1);
        }
        for (int c = 0; ok && c < N; ++c) {
          const uint32_t sl = c % QST;
          ok = mbar_wait_abortable(q_full0 + 8 * sl, (c / QST) & 1, 339, abort_flag);
          if (ok && c + 1 < N) ok = mbar_wait_abortable(do_full0 + 8 * ((c + 1) % DST), ((c + 1) / DST) & 1, 341, abort_flag);
          const uint64_t dq = umma_desc_advance(dq_base, sl * TILE);
          for (int h = 0; ok && h < 2; ++h) {
            ok = mbar_wait_abortable(ds_full0 + 8 * h, c & 1, 340, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ts(tmem + kColDK, tmem + 128 + h * 64 + ks * 8, umma_desc_advance(dq, (4 * h + ks) * 2048), idesc_dk, (c | h | ks) ? 1u : 0u);
            if (h == 1) umma_commit(q_empty0 + 8 * sl);
            if (c + 1 < N) issue_dp(c + 1, h);
          }
        }
        umma_commit(acc_full);
      }
    }
  } else if (warp >= 12) {
    // ------------------------------- row data: one query row per thread -----------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    const int row = threadIdx.x - 384;
    float lse = -INFINITY, del = 0.f;
    bf16 g = __float2bfloat16(0.f);
    auto load = [&](int c) {   // as loaded: converting here would wait for the loads
      lse = -INFINITY;
      del = 0.f;
      g = __float2bfloat16(0.f);
      if (c >= N) return;
      int hg;
      const int r = tile_of(c, hg) + (row >> 4);
      if (r >= it.Tq) return;   // no such row: all of its terms are zero
      const long long qrow = (it.row0 + r) * a.Hq + hg * 16 + (row & 15);
      lse = a.lse[qrow];
      del = a.delta[qrow];
      g = a.gate ? a.gate[qrow] : __float2bfloat16(1.f);
    };
    bool ok = true;
    load(0);
    for (int c = 0; ok && c < N; ++c) {
      const uint32_t st = c & 1;
      ok = mbar_wait_abortable(row_empty0 + 8 * st, ((c >> 1) & 1) ^ 1, 342, abort_flag);
      uint8_t* p = dense_kv_smem + (rows_s - sbase) + st * kRowStage;
      reinterpret_cast<float*>(p)[row] = lse > -INFINITY ? -lse * kLog2e : -INFINITY;   // a row without a visible key: P = 0
      reinterpret_cast<float*>(p + 512)[row] = -del;
      reinterpret_cast<bf16*>(p + 1024)[row] = g;
      mbar_arrive(row_full0 + 8 * st);
      load(c + 1);
    }
  } else {
    // ------------------------------- soft-max warps: one key, half of the tile's query rows per thread -----------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int quad = warp & 3, half = (warp - 4) >> 2;
    const int key = it.key0 + 32 * quad + lane;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const uint32_t s_col = tmem + lane_addr + half * 64, dp_col = s_col + 128;
    const float sl2 = a.scale * kLog2e;
    const uint64_t sl22 = pack_f32x2(sl2, sl2);
    bool ok = true;
    for (int c = 0; c < N; ++c) {
      int hg;
      const int t0 = a.seq.q0 + tile_of(c, hg);   // positions of the tile's tokens: t0 .. t0 + 7
      const uint32_t st = c & 1;
      const uint8_t* rp = dense_kv_smem + (rows_s - sbase) + st * kRowStage;
      const float4* nl4 = reinterpret_cast<const float4*>(rp) + half * 16;
      const float4* nd4 = reinterpret_cast<const float4*>(rp + 512) + half * 16;
      const uint4* g8 = reinterpret_cast<const uint4*>(rp + 1024) + half * 8;
      bool all;                                    // no column of the tile is masked for any key
      if (a.mode == 0)
        all = it.key0 + 127 <= t0 && it.key0 > t0 + kTok - 1 - a.window;
      else
        all = !a.causal || (long long)(it.key0 + 127) * a.cstride + a.cblock <= t0;
      ok = mbar_wait_abortable(row_full0 + 8 * st, (c >> 1) & 1, 343, abort_flag) && ok;
      ok = mbar_wait_abortable(s_full0 + 8 * half, c & 1, 344, abort_flag) && ok;
      tc_fence_after();
      float s[64];
      tmem_ld32(s_col, *reinterpret_cast<float(*)[32]>(&s[0]));
      tmem_ld32(s_col + 32, *reinterpret_cast<float(*)[32]>(&s[32]));
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 64; e += 4) {
        const float4 nl = nl4[e >> 2];
        const uint64_t x0 = fma_f32x2(pack_f32x2(s[e], s[e + 1]), sl22, pack_f32x2(nl.x, nl.y));
        const uint64_t x1 = fma_f32x2(pack_f32x2(s[e + 2], s[e + 3]), sl22, pack_f32x2(nl.z, nl.w));
        s[e] = lo_f32x2(x0);
        s[e + 1] = hi_f32x2(x0);
        s[e + 2] = lo_f32x2(x1);
        s[e + 3] = hi_f32x2(x1);
      }
      if (!all) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // four tokens of this thread's half, 16 heads each
          const int t = t0 + half * 4 + j;
          const bool valid = a.mode == 0 ? (key <= t && key > t - a.window) : (long long)key * a.cstride + a.cblock <= t;
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (!valid) s[16 * j + e] = -INFINITY;
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float w[16];
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          const uint4 g = g8[(32 * q + e) >> 3];
          const uint32_t gg[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float& p0 = s[32 * q + e + 2 * u];
            float& p1 = s[32 * q + e + 2 * u + 1];
            p0 = ex2(p0);
            p1 = ex2(p1);
            const uint64_t gp = mul_f32x2(pack_f32x2(__uint_as_float(gg[u] << 16), __uint_as_float(gg[u] & 0xffff0000u)), pack_f32x2(p0, p1));
            w[(e >> 1) + u] = __uint_as_float(pack_bf16(lo_f32x2(gp), hi_f32x2(gp)));
          }
        }
        tmem_st16(s_col + q * 16, w);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_full0 + 8 * half);
      ok = mbar_wait_abortable(dp_full0 + 8 * half, c & 1, 345, abort_flag) && ok;
      tc_fence_after();
      float dp[64];
      tmem_ld32(dp_col, *reinterpret_cast<float(*)[32]>(&dp[0]));
      tmem_ld32(dp_col + 32, *reinterpret_cast<float(*)[32]>(&dp[32]));
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float w[16];
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          const int b = 32 * q + e;
          const uint4 g = g8[b >> 3];
          const uint32_t gg[4] = {g.x, g.y, g.z, g.w};
          const float4 na = nd4[b >> 2], nb = nd4[(b >> 2) + 1];
          const uint64_t nd[4] = {pack_f32x2(na.x, na.y), pack_f32x2(na.z, na.w), pack_f32x2(nb.x, nb.y), pack_f32x2(nb.z, nb.w)};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint64_t g2 = pack_f32x2(__uint_as_float(gg[u] << 16), __uint_as_float(gg[u] & 0xffff0000u));
            const uint64_t x = fma_f32x2(g2, pack_f32x2(dp[b + 2 * u], dp[b + 2 * u + 1]), nd[u]);
            const uint64_t d2 = mul_f32x2(pack_f32x2(s[b + 2 * u], s[b + 2 * u + 1]), x);
            w[(e >> 1) + u] = __uint_as_float(pack_bf16(lo_f32x2(d2), hi_f32x2(d2)));
          }
        }
        tmem_st16(dp_col + q * 16, w);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(ds_full0 + 8 * half);
      mbar_arrive(row_empty0 + 8 * st);
    }
    // ---- epilogue: dV (half 0), dK (half 1); rows become whole lines by a transpose among eight lanes ----
    if (N > 0) ok = mbar_wait_abortable(acc_full, 0, 346, abort_flag) && ok;
    tc_fence_after();
    const float mul = half ? a.scale : 1.f;
    float* part = a.part ? a.part + ((half ? 0 : (long long)a.slabs) + a.slab0 + it.slab) * a.n_out : nullptr;
    bf16* out = half ? a.dk : a.dv;
#pragma unroll 1
    for (int q = 0; q < D / 32; ++q) {
      float v[32];
      if (N > 0) {
        tmem_ld32(tmem + lane_addr + (half ? kColDK : kColDV) + q * 32, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = 0.f;
      }
      float4 x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = make_float4(v[4 * e] * mul, v[4 * e + 1] * mul, v[4 * e + 2] * mul, v[4 * e + 3] * mul);
      transpose8(x, lane);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = 32 * quad + (lane & ~7) + k;
        if (!ok || r >= it.keys) continue;
        const long long off = ((it.out_row + r) * a.Hk + it.hk) * D + q * 32 + (lane & 7) * 4;
        if (part)
          *reinterpret_cast<float4*>(part + off) = x[k];
        else
          *reinterpret_cast<uint2*>(out + off) = make_uint2(pack_bf16(x[k].x, x[k].y), pack_bf16(x[k].z, x[k].w));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// dk, dv (bf16) = sum over the segments that see the row's key tile of part [2][nslab][n_out]
__global__ void __launch_bounds__(256) dense_kv_reduce_kernel(const DenseKvArgs a, int D) {
  after_previous();
  const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= a.n_out) return;
  const long long row = i / (a.Hk * D);
  const int key = (int)(row % a.Lk), Tq = a.seq.Tq;
  const long long first = a.causal ? (long long)(key / 128 * 128) * a.cstride + a.cblock - a.seq.q0 : 0;
  const float* p = a.part + (blockIdx.y ? (long long)a.nslab * a.n_out : 0) + i;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  const int k0 = first > 0 ? (int)min(first / a.seg_len, (long long)a.nslab) : 0, k1 = min(a.nslab, (Tq + a.seg_len - 1) / a.seg_len);
#pragma unroll 4
  for (int k = first < Tq ? k0 : k1; k < k1; ++k) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p + k * a.n_out));
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  *reinterpret_cast<uint2*>((blockIdx.y ? a.dv : a.dk) + i) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
}

template <int D>
int launch(const DenseKvArgs& a, cudaStream_t s) {
  CUtensorMap tmQ, tmDO, tmK, tmV;
  // Where a sequence's last tile of query rows reaches into the next sequence, rows come by sequence and those past the end
  // are zeros:
  // they enter the products over the rows with P = 0, and the next sequence's dO or Q there could be NaN or infinite.  (Not
  // everywhere: the fourth coordinate costs 4 % of the kernel, 65536 tokens 9.9 -> 10.3 ms; a branch in the loop 1 %.)
  const bool by_seq = a.seq.B > 1 && a.seq.Tq % kTok != 0;
  const int nq = by_seq ? a.seq.B : 1;
  const unsigned long long qrows = (unsigned long long)(seq_rows(a.seq) / nq), HD2 = (unsigned long long)a.Hq * D * 2;
  const unsigned long long qd[4] = {(unsigned long long)D, (unsigned long long)a.Hq, qrows, (unsigned long long)nq};
  const unsigned long long qs[3] = {(unsigned long long)D * 2, HD2, qrows * HD2};
  const unsigned qb[4] = {64, 16, (unsigned)kTok, 1};
  int rc = make_tmap_generic(&tmQ, a.q, by_seq ? 4 : 3, qd, qs, qb);
  if (!rc) rc = make_tmap_generic(&tmDO, a.dout, by_seq ? 4 : 3, qd, qs, qb);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.k, D, a.Hk, a.Lk, a.seq.B, 128);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hk, a.Lk, a.seq.B, 128);
  if (rc) return rc;
  const auto kern = by_seq ? dense_kv_tc_kernel<D, true> : dense_kv_tc_kernel<D, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem<D>);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)a.seq.B * ((a.Lk + 127) / 128);
  const long long grid = tiles * a.Hk * a.nslab;
  if (grid <= 0) return 0;
  if (grid > 0x7fffffffLL) {
    set_error("dense dK, dV: grid too large");
    return -33;
  }
  launch_next(kern, (unsigned)grid, kThreads, kSmem<D>, s, tmQ, tmDO, tmK, tmV, a);
  note_launches(1);
  if (a.mode == 1 && a.part) {
    launch_next(dense_kv_reduce_kernel, dim3((unsigned)((a.n_out / 4 + 255) / 256), 2), 256, 0, s, a, D);
    note_launches(1);
  }
  return (int)cudaGetLastError();
}

}  // namespace

int launch_dense_kv_tc(const DenseKvArgs& args, int head_dim, cudaStream_t s) {
  DenseKvArgs a = args;
  a.n_out = (long long)a.seq.B * a.Lk * a.Hk * head_dim;
  return head_dim == 64 ? launch<64>(a, s) : launch<128>(a, s);
}

// Parts of a key tile's query range.  Window: all tiles are alike, so the count (of 1 .. 16) is the one whose waves of CTAs
// take the least, a CTA's start and end counted as four query tiles (10 us).
int dense_kv_window_slabs(int B, int T, int Hk, int window) {
  const long long tiles = (long long)B * Hk * ((T + 127) / 128);
  const long long n = (std::min<long long>((long long)window + 127, T) + kTok - 1) / kTok;
  int best = 1;
  long long cost = -1;
  for (int ns = 1; ns <= 16 && ns <= n; ++ns) {
    const long long c = (tiles * ns + num_sms() - 1) / num_sms() * ((n + ns - 1) / ns + 4);
    if (cost < 0 || c < cost) {
      cost = c;
      best = ns;
    }
  }
  return best;
}
// Compressed: with w query tiles of work per SM in all (half of all pairs: causal) and segments of x tiles, starts and ends
// cost 4 / x of the time and the last wave about x / (2 w), least at x = sqrt(8 w).  Never more than 32 segments (they are
// memory).
int dense_kv_segment_rows(int B, int T, int Tc, int Hk) {
  const double w = (double)B * Hk * ((Tc + 127) / 128) * T / (2 * kTok) / num_sms();
  long long rows = ((long long)std::sqrt(8 * w) + 1) * kTok;
  rows = std::max<long long>(rows, ((T + 31) / 32 + kTok - 1) / kTok * kTok);
  return (int)std::min<long long>(rows, (T + kTok - 1) / kTok * kTok);
}

int dense_kv_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
