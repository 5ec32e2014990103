// dQ of the dense branches on tcgen05 (head_dim 64 or 128): sliding-window attention, compressed attention, or both in one
// pass.  Semantics of parallel_nsa_bwd_kernel_dq's window half (nsa/selection_attn.py:358-398) and of _attn_bwd_only_dq
// (nsa/triton_attention.py:321-416).
//
// A persistent CTA owns 8 consecutive tokens x 16 heads = [128 x D] tiles of Q and dO (resident for the item).  [128 keys x
// D] tiles of K and V (then of the compressed keys and values) stream through two rings.  Per tile
//     S  = Q . K^T,   dP = dO . V^T        (accumulators in TMEM, issued by one thread)
// eight soft-max warps (half a row of 64 key columns per thread; lse, delta, gate and the mask are thread-local)
// form  dS = P (g dP - delta)  with  P = exp(scale S - lse), packed as bf16 in tensor memory, and a second thread issues
//     dQ += dS . K                          (A = dS from tensor memory, B = K as an MN-major operand)
// dQ stays in tensor memory over both branches and is stored once.
//
// Bound: the MMAs, 24 per tile at about 90 cycles (an SS product of this shape reads 8 KB of shared memory, 64 cycles' worth),
// 2050 cycles per tile; the soft-max takes about 1500.  So nothing may make the tensor core wait: the next tile's S and dP are
// issued each as soon as this tile's is in registers (P is formed while dP is still being computed); dS in tensor memory
// leaves room for a third K slot (with two stages of
// K and V together a stage came back 2500 cycles after its dQ, 3700 per tile); Q and dO of the next item load as soon as the
// last S and dP have read them; the epilogue has its own four warps.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kTok = 8;
constexpr int kThreads = 512;                 // warp 0 TMA Q, K; 1 S/dP; 2 dQ; 3 TMA dO, V; 4-11 soft-max; 12-15 epilogue
constexpr int kSoft = 256;
constexpr int kEpi = 128;
constexpr uint32_t PANEL = 128 * 128;         // [128 rows][64 columns] bf16
constexpr int KST = 3, VST = 2;
constexpr uint32_t kTmemCols = 512;           // S 0..127, dP 128..255, dQ 256.., dS 384..447 (packed bf16)
constexpr uint32_t kMisc = 256;
template <int D>
constexpr uint32_t kSmem = (D / 64) * PANEL * (2 + KST + VST) + kMisc + 2 * 128 * 4 + 1024;   // [2][128] floats: row pre-pass

struct Sched {
  int first, nw, n;   // first window tile, window tiles, tiles in all
};

template <bool WIN, bool CMP>
__device__ __forceinline__ Sched make_sched(const DenseArgs& a, const SeqTile& st) {
  Sched s = {0, 0, 0};
  if (st.t0 >= st.Tq) return s;
  const int t0 = a.seq.q0 + st.t0;                        // positions in the sequence
  const int tmax = min(a.seq.q0 + st.Tq - 1, t0 + kTok - 1);
  if (WIN) {
    s.first = max(0, t0 - a.window + 1) / 128;
    s.nw = tmax / 128 - s.first + 1;
  }
  s.n = s.nw;
  if (CMP) {
    int nvis = st.Tc;
    if (a.causal) nvis = (tmax < a.cblock) ? 0 : min(st.Tc, (tmax - a.cblock) / a.cstride + 1);
    s.n += (nvis + 127) / 128;
  }
  return s;
}

struct Maps {
  CUtensorMap q, dout, k, v, ck, cv;
};

template <int D, bool WIN, bool CMP>
__global__ void __launch_bounds__(kThreads, 1)
    dense_dq_tc_kernel(const __grid_constant__ Maps maps, const DenseArgs a) {
  after_previous();
  constexpr int NP = D / 64;
  constexpr uint32_t TILE = NP * PANEL;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q_s = sbase, do_s = sbase + TILE, k_ring = sbase + 2 * TILE, v_ring = k_ring + KST * TILE;
  const uint32_t misc = v_ring + VST * TILE;
  const uint32_t q_full = misc, q_free = misc + 8, do_full = misc + 16, do_free = misc + 24, k_full0 = misc + 32,
                 k_empty0 = misc + 56, v_full0 = misc + 80, v_empty0 = misc + 96, s_full = misc + 112, s_free = misc + 120,
                 dp_full = misc + 128, dp_free = misc + 136, ds_full = misc + 144, ds_free = misc + 152, dq_full = misc + 160,
                 dq_free = misc + 168, tmem_slot = misc + 176;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + (misc - sbase) + 184);
  float* xpre = reinterpret_cast<float*>(sgen + (misc - sbase) + kMisc);   // [2 branches][128 rows] exchange of the row pre-pass
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    mbar_init(q_free, 1);
    mbar_init(do_full, 1);
    mbar_init(do_free, 1);
    for (int i = 0; i < KST; ++i) {
      mbar_init(k_full0 + 8 * i, 1);
      mbar_init(k_empty0 + 8 * i, 1);
    }
    for (int i = 0; i < VST; ++i) {
      mbar_init(v_full0 + 8 * i, 1);
      mbar_init(v_empty0 + 8 * i, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, kSoft);
    mbar_init(dp_full, 1);
    mbar_init(dp_free, kSoft);
    mbar_init(ds_full, kSoft);
    mbar_init(ds_free, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, kEpi);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));

  const int HG = a.Hq / 16;
  const int G16 = (a.Hq / a.Hk) / 16;
  const int ntile = seq_tiles_dev(a.seq, kTok);
  const int total = HG * ntile;   // (checked on the host: fits 31 bits)

  // Registers: 512 threads are launched with 128 each (65536); 128 x 56 + 256 x 168 + 128 x 120 = 65536 (an inc that the
  // launch pool cannot satisfy blocks for ever).
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp == 0 || warp == 3) {
    // ------------------------------- TMA producers: Q and K (warp 0), dO and V (warp 3) --------------------
    // The first K (V) tile of an item goes out before its Q (dO), whose buffer comes back last.
    const bool is_k = warp == 0;
    const uint32_t full0 = is_k ? k_full0 : v_full0, empty0 = is_k ? k_empty0 : v_empty0, ring = is_k ? k_ring : v_ring;
    const uint32_t x_full = is_k ? q_full : do_full, x_free = is_k ? q_free : do_free, x_s = is_k ? q_s : do_s;
    const CUtensorMap* tmX = is_k ? &maps.q : &maps.dout;
    const uint32_t nst = is_k ? KST : VST;
    uint32_t c = 0, ic = 0;
    if (elect_one()) {
      bool good = true;
      for (int item = blockIdx.x; good && item < total; item += gridDim.x) {
        const int hg = item % HG;
        const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
        if (st.t0 >= st.Tq) continue;
        const Sched sc = make_sched<WIN, CMP>(a, st);
        const int hk = hg / G16;
        for (int i = 0; good && i < max(sc.n, 1); ++i) {
          if (i < sc.n) {
            const uint32_t sl = c % nst;
            good = mbar_wait_abortable(empty0 + 8 * sl, ((c / nst) & 1) ^ 1, 202, abort_flag);
            if (!good) break;
            mbar_expect_tx(full0 + 8 * sl, TILE);
            const bool win = WIN && (!CMP || i < sc.nw);
            const CUtensorMap* tm = is_k ? (win ? &maps.k : &maps.ck) : (win ? &maps.v : &maps.cv);
            const int row = win ? (sc.first + i) * 128 : (i - sc.nw) * 128;
#pragma unroll
            for (int p = 0; p < NP; ++p) tma_load_4d(ring + sl * TILE + p * PANEL, tm, full0 + 8 * sl, p * 64, hk, row, st.b);
            ++c;
          }
          if (i == 0) {
            good = mbar_wait_abortable(x_free, (ic & 1) ^ 1, 201, abort_flag);
            if (!good) break;
            mbar_expect_tx(x_full, TILE);
#pragma unroll
            for (int p = 0; p < NP; ++p) tma_load_3d(x_s + p * PANEL, tmX, x_full, p * 64, hg * 16, (int)st.row0 + st.t0);
          }
        }
        ++ic;
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer: S and dP ---------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      uint32_t c = 0, ic = 0;
      bool ok = true;
      const uint64_t dq_desc = umma_smem_desc(q_s, 0, 1024), ddo_desc = umma_smem_desc(do_s, 0, 1024);
      const uint64_t dk_base = umma_smem_desc(k_ring, 0, 1024), dv_base = umma_smem_desc(v_ring, 0, 1024);
      for (int item = blockIdx.x; ok && item < total; item += gridDim.x) {
        const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
        if (st.t0 >= st.Tq) continue;
        const int n = make_sched<WIN, CMP>(a, st).n;
        ok = mbar_wait_abortable(q_full, ic & 1, 203, abort_flag);
        // (an item without a tile still waits for both of its loads: a buffer is handed back only when they have landed)
        if (ok && n == 0) ok = mbar_wait_abortable(do_full, ic & 1, 215, abort_flag);
        for (int i = 0; ok && i < n; ++i, ++c) {
          const uint32_t ks_ = c % KST, vs = c % VST;
          ok = mbar_wait_abortable(k_full0 + 8 * ks_, (c / KST) & 1, 204, abort_flag);
          // the soft-max warps hold the previous tile's S in registers
          if (ok && c > 0) ok = mbar_wait_abortable(s_free, (c - 1) & 1, 205, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t dk = umma_desc_advance(dk_base, ks_ * TILE), dv = umma_desc_advance(dv_base, vs * TILE);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks >> 2) * PANEL + (ks & 3) * 32;
            umma_ss(tmem + 0, umma_desc_advance(dq_desc, off), umma_desc_advance(dk, off), idesc_s, ks ? 1u : 0u);
          }
          umma_commit(s_full);
          if (i == n - 1) umma_commit(q_free);
          if (ok && i == 0) ok = mbar_wait_abortable(do_full, ic & 1, 214, abort_flag);
          if (ok) ok = mbar_wait_abortable(v_full0 + 8 * vs, (c / VST) & 1, 206, abort_flag);
          if (ok && c > 0) ok = mbar_wait_abortable(dp_free, (c - 1) & 1, 212, abort_flag);   // and its dP
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks >> 2) * PANEL + (ks & 3) * 32;
            umma_ss(tmem + 128, umma_desc_advance(ddo_desc, off), umma_desc_advance(dv, off), idesc_s, ks ? 1u : 0u);
          }
          umma_commit(dp_full);
          umma_commit(v_empty0 + 8 * vs);
        }
        umma_commit(do_free);
        if (n == 0) umma_commit(q_free);
        ++ic;
      }
    }
  } else {
    // ------------------------------- MMA issuer: dQ ---------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, D, 0, 1);
      uint32_t c = 0, ic = 0;
      bool ok = true;
      const uint64_t dk_base = umma_smem_desc(k_ring, PANEL, 1024);
      for (int item = blockIdx.x; ok && item < total; item += gridDim.x) {
        const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
        if (st.t0 >= st.Tq) continue;
        const int n = make_sched<WIN, CMP>(a, st).n;
        if (ic > 0) ok = mbar_wait_abortable(dq_free, (ic - 1) & 1, 207, abort_flag);   // the previous item's dQ has been read
        for (int i = 0; ok && i < n; ++i, ++c) {
          const uint32_t ks_ = c % KST;
          ok = mbar_wait_abortable(ds_full, c & 1, 208, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t dk = umma_desc_advance(dk_base, ks_ * TILE);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)   // A = dS from tensor memory: 16 keys = 8 packed columns per step
            umma_ts(tmem + 256, tmem + 384 + ks * 8, umma_desc_advance(dk, ks * 2048), idesc_dq, (i | ks) ? 1u : 0u);
          umma_commit(k_empty0 + 8 * ks_);
          umma_commit(ds_free);
        }
        umma_commit(dq_full);
        ++ic;
      }
    }
  }
  } else if (warp < 12) {
    // ------------------------------- soft-max warps ------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int quad = warp & 3;
    const int half = (warp - 4) >> 2;
    const int row = 32 * quad + lane;
    const int tl = row >> 4, head = row & 15;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const uint32_t ds_col = tmem + lane_addr + 384 + half * 32;
    const float sl2 = (D == 64 && a.scale == 0.f ? 1e-30f : a.scale) * kLog2e;   // (head_dim 64: scales of any sign, see the forward)
    const float hidden = D == 64 && a.scale < 0.f ? INFINITY : -INFINITY;        // a masked column: scaled it is -inf
    uint32_t c = 0;
    bool ok = true;
    struct Row {   // operands of this thread's row for the (first) branch and, with both, for the compressed one, as loaded:
      float lse, del, lse_c, del_c;   // converting them here would wait for the loads
      bf16 g, g_c;
    };
    auto load_row = [&](int item, const SeqTile& st) {
      Row r = {-INFINITY, 0.f, -INFINITY, 0.f, __float2bfloat16(1.f), __float2bfloat16(1.f)};
      if (item >= total || st.t0 + tl >= st.Tq) return r;   // no such row: lse = -inf makes all of its terms zero
      const long long qrow = (st.row0 + st.t0 + tl) * a.Hq + (item % HG) * 16 + head;
      r.lse = a.lse[qrow];
      if (a.gate) r.g = a.gate[qrow];
      if (!a.pre_o[0]) r.del = a.delta[qrow];
      if (WIN && CMP) {
        r.lse_c = a.lse_c[qrow];
        if (a.gate_c) r.g_c = a.gate_c[qrow];
        r.del_c = a.delta_c[qrow];
      }
      return r;
    };
    SeqTile nst = seq_tile(a.seq, kTok, max(ntile - 1 - (int)blockIdx.x / HG, 0));
    Row next = load_row(blockIdx.x, nst);
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      const int hg = item % HG;
      const SeqTile st = nst;
      Row rw = next;
      const int item1 = item + gridDim.x;
      nst = seq_tile(a.seq, kTok, max(ntile - 1 - item1 / HG, 0));
      next = load_row(item1, nst);   // under way during this item
      if (st.t0 >= st.Tq) continue;
      const Sched sc = make_sched<WIN, CMP>(a, st);
      const int tloc = st.t0 + tl;             // local query row
      const int t = a.seq.q0 + tloc;           // its sequence position
      const bool live = tloc < st.Tq;
      if (a.pre_o[0]) {
        // Row pre-pass folded in (parallel_nsa_bwd_kernel_preprocess, nsa/selection_attn.py:520-530; _attn_bwd_preprocess,
        // nsa/triton_attention.py:184-199; the gate gradients of nsa/nsa.py:133): rowsum(o_x * dO) over this thread's half of
        // the channels, the two halves of a row meet in shared memory, the first half finishes and publishes the row's delta.
        const long long qrow = (st.row0 + (live ? tloc : 0)) * a.Hq + hg * 16 + head;
        float part[2] = {0.f, 0.f};
        const uint4* pd = reinterpret_cast<const uint4*>(a.dout + qrow * D + half * (D / 2));
        uint4 dv[D / 16];
#pragma unroll
        for (int e = 0; e < D / 16; ++e) dv[e] = pd[e];
#pragma unroll
        for (int br = 0; br < 2; ++br) {
          if (!a.pre_o[br]) continue;
          const uint4* po = reinterpret_cast<const uint4*>(a.pre_o[br] + qrow * D + half * (D / 2));
#pragma unroll
          for (int e = 0; e < D / 16; ++e) {
            const uint4 ov = po[e];
            const __nv_bfloat162* ho2 = reinterpret_cast<const __nv_bfloat162*>(&ov);
            const __nv_bfloat162* hd2 = reinterpret_cast<const __nv_bfloat162*>(&dv[e]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float2 x = __bfloat1622float2(ho2[u]), y = __bfloat1622float2(hd2[u]);
              part[br] = fmaf(x.x, y.x, fmaf(x.y, y.y, part[br]));
            }
          }
        }
        if (half == 1) {
          xpre[row] = part[0];
          xpre[128 + row] = part[1];
        }
        named_bar_sync(1, kSoft);
        if (half == 0) {
          float own = 0.f;
#pragma unroll
          for (int br = 0; br < 2; ++br) {
            if (!a.pre_o[br]) continue;
            const float tot = part[br] + xpre[br * 128 + row];
            const float gb = a.pre_gate[br] ? __bfloat162float(a.pre_gate[br][qrow]) : 1.f;
            if (live) {
              a.pre_delta[br][qrow] = gb * tot;
              if (a.pre_dgate[br]) a.pre_dgate[br][qrow] = __float2bfloat16(tot);
            }
            if (br == 0) own = gb * tot;
          }
          xpre[row] = own;
          rw.del = own;
        }
        named_bar_sync(1, kSoft);
        if (half == 1) rw.del = xpre[row];
      }
      for (int i = 0; i < sc.n; ++i, ++c) {
        const bool win = WIN && (!CMP || i < sc.nw);
        int lo = 0, hi;                          // this thread's valid columns of the tile
        if (win) {
          const int j0 = (sc.first + i) * 128 + half * 64;
          lo = t - a.window + 1 - j0;
          hi = t + 1 - j0;
        } else {
          int nvis = st.Tc;
          if (a.causal) nvis = (t < a.cblock) ? 0 : min(st.Tc, (t - a.cblock) / a.cstride + 1);
          hi = nvis - (i - sc.nw) * 128 - half * 64;
        }
        const bool first = !WIN || !CMP || win;
        const float lse2 = (first ? rw.lse : rw.lse_c) * kLog2e, gv = __bfloat162float(first ? rw.g : rw.g_c),
                    del = first ? rw.del : rw.del_c;
        if (!live || !(lse2 > -INFINITY)) hi = 0;
        ok = mbar_wait_abortable(s_full, c & 1, 209, abort_flag) && ok;
        tc_fence_after();
        float s[64];
        tmem_ld32(tmem + lane_addr + half * 64, *reinterpret_cast<float(*)[32]>(&s[0]));
        tmem_ld32(tmem + lane_addr + half * 64 + 32, *reinterpret_cast<float(*)[32]>(&s[32]));
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(s_free);   // S of this tile is in registers: the next tile's may overwrite it
        if (!__all_sync(0xffffffffu, lo <= 0 && hi >= 64)) {   // masked columns: exp(-inf) = 0
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int l0 = min(max(lo - 32 * q, 0), 32), h0 = min(max(hi - 32 * q, 0), 32);
            const unsigned valid = h0 > l0 ? (0xffffffffu >> (32 - (h0 - l0))) << l0 : 0u;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (!(valid & (1u << e))) s[32 * q + e] = hidden;
          }
        }
        const float nl = lse2 > -INFINITY ? -lse2 : 0.f;
        const uint64_t sl22 = pack_f32x2(sl2, sl2), nl2 = pack_f32x2(nl, nl), gv2 = pack_f32x2(gv, gv), nd2 = pack_f32x2(-del, -del);
#pragma unroll
        for (int e = 0; e < 64; e += 2) {   // P, while dP is still being computed
          const uint64_t x = fma_f32x2(pack_f32x2(s[e], s[e + 1]), sl22, nl2);
          s[e] = ex2(lo_f32x2(x));
          s[e + 1] = ex2(hi_f32x2(x));
        }
        ok = mbar_wait_abortable(dp_full, c & 1, 213, abort_flag) && ok;
        tc_fence_after();
        float dp[64];
        tmem_ld32(tmem + lane_addr + 128 + half * 64, *reinterpret_cast<float(*)[32]>(&dp[0]));
        tmem_ld32(tmem + lane_addr + 128 + half * 64 + 32, *reinterpret_cast<float(*)[32]>(&dp[32]));
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(dp_free);
        float dw[32];
#pragma unroll
        for (int e = 0; e < 64; e += 2) {
          const uint64_t w = fma_f32x2(gv2, pack_f32x2(dp[e], dp[e + 1]), nd2);
          const uint64_t d2 = mul_f32x2(pack_f32x2(s[e], s[e + 1]), w);
          dw[e >> 1] = __uint_as_float(pack_bf16(lo_f32x2(d2), hi_f32x2(d2)));
        }
        if (c > 0) ok = mbar_wait_abortable(ds_free, (c - 1) & 1, 210, abort_flag) && ok;   // dQ of the previous tile read dS
        tc_fence_after();
        tmem_st16(ds_col, *reinterpret_cast<float(*)[16]>(&dw[0]));
        tmem_st16(ds_col + 16, *reinterpret_cast<float(*)[16]>(&dw[16]));
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(ds_full);
      }
    }
  } else {
    // ------------------------------- epilogue warps: dq = scale * dQ (+ previous contents) -----------------------
    // One row per thread while the soft-max warps are already at the next item (an item's epilogue took 4300 of its 15000
    // cycles when they did it).  Rows become whole 128-byte lines by a transpose among eight lanes: lane l then holds piece l
    // of the group's rows 0..7.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;");
    const int quad = warp & 3;
    const uint32_t o_col = tmem + ((uint32_t)(32 * quad) << 16) + 256;
    uint32_t ic = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      const int hg = item % HG;
      const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
      if (st.t0 >= st.Tq) continue;
      const int n = make_sched<WIN, CMP>(a, st).n;
      auto line = [&](int p, int k) -> uint4* {   // this lane's piece of panel p of the k-th row of its group; null: no such row
        const int r = 32 * quad + (lane & ~7) + k;
        if (st.t0 + (r >> 4) >= st.Tq) return nullptr;
        return reinterpret_cast<uint4*>(a.dq + ((st.row0 + st.t0 + (r >> 4)) * a.Hq + hg * 16 + (r & 15)) * D + p * 64) + (lane & 7);
      };
      ok = mbar_wait_abortable(dq_full, ic & 1, 211, abort_flag) && ok;
      tc_fence_after();
#pragma unroll 1
      for (int p = 0; p < NP; ++p) {
        uint4 out[8];
        if (a.accumulate) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint4* src = line(p, k);
            out[k] = src ? *src : make_uint4(0u, 0u, 0u, 0u);
          }
          transpose8(out, lane);   // row mapping: lane = row, piece k
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) out[k] = make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // 32 channels, four pieces
          float o[32];
          if (n > 0) {
            tmem_ld32(o_col + p * 64 + h * 32, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0.f;
          }
          if (p == NP - 1 && h == 1) {
            tc_fence_before();
            mbar_arrive(dq_free);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&out[4 * h + e]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float2 x = __bfloat1622float2(ho[u]);
              ho[u] = __floats2bfloat162_rn(fmaf(o[8 * e + 2 * u], a.scale, x.x), fmaf(o[8 * e + 2 * u + 1], a.scale, x.y));
            }
          }
        }
        transpose8(out, lane);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint4* dst = line(p, k);
          if (dst && ok) *dst = out[k];
        }
      }
      ++ic;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

template <int D, bool WIN, bool CMP>
int launch(const DenseArgs& a, cudaStream_t s) {
  Maps m;
  const unsigned long long qd[3] = {(unsigned long long)D, (unsigned long long)a.Hq, (unsigned long long)seq_rows(a.seq)};
  const unsigned long long qs[2] = {(unsigned long long)D * 2, (unsigned long long)a.Hq * D * 2};
  const unsigned qb[3] = {64, 16, (unsigned)kTok};
  int rc = make_tmap_generic(&m.q, a.q, 3, qd, qs, qb);
  if (!rc) rc = make_tmap_generic(&m.dout, a.dout, 3, qd, qs, qb);
  if (WIN && !rc) {
    rc = make_tmap_rows4d(&m.k, a.k, D, a.Hk, a.T, a.B, 128);
    if (!rc) rc = make_tmap_rows4d(&m.v, a.v, D, a.Hk, a.T, a.B, 128);
  }
  if (CMP && !rc) {
    rc = make_tmap_rows4d(&m.ck, WIN ? a.ck : a.k, D, a.Hk, a.seq.Tc, a.B, 128);
    if (!rc) rc = make_tmap_rows4d(&m.cv, WIN ? a.cv : a.v, D, a.Hk, a.seq.Tc, a.B, 128);
  }
  if (rc) return rc;
  if (!WIN) m.k = m.v = m.ck;
  if (!CMP) m.ck = m.cv = m.k;
  auto kern = dense_dq_tc_kernel<D, WIN, CMP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem<D>);
  if (e != cudaSuccess) return (int)e;
  const long long total = (long long)(a.Hq / 16) * seq_tiles(a.seq, kTok);
  if (total > 0x7fffffffLL - num_sms()) {
    set_error("dense dQ: too many tokens");
    return -33;
  }
  const int grid = (int)(total < num_sms() ? total : num_sms());
  if (grid <= 0) return 0;
  launch_next(kern, grid, kThreads, kSmem<D>, s, m, a);
  note_launches(1);
  return (int)cudaGetLastError();
}

template <int D>
int dispatch(const DenseArgs& a, cudaStream_t s) {
  if (a.mode == 1) return launch<D, false, true>(a, s);
  return a.ck ? launch<D, true, true>(a, s) : launch<D, true, false>(a, s);
}

}  // namespace

int launch_dense_dq_tc(const DenseArgs& args, int head_dim, cudaStream_t s) {
  DenseArgs a = args;
  a.seq = {a.B, a.Tq, a.q0, a.mode == 1 ? a.Lk : a.seq.Tc};
  return head_dim == 64 ? dispatch<64>(a, s) : dispatch<128>(a, s);
}
int dense_dq_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
