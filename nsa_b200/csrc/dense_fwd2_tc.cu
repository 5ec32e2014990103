// Dense query-major attention FORWARD on tcgen05, two query tiles per CTA (head_dim 64 or 128): sliding-window attention
// (mode 0) and compressed attention (mode 1).  Semantics and result layouts of nsa/selection_attn.py:484-516 (window),
// nsa/triton_attention.py:87-181,465-475 (compressed attention) and, optionally, the gate projection nn.Linear(head_dim, 3)
// of nsa/nsa.py:117 computed from the resident query tiles.  The block selection has its own kernel (score_tc.cu).
//
// A persistent CTA owns 16 consecutive tokens x the 16 heads of a GQA group = two [128 x D] Q tiles that share one
// stream of [128 keys x D] K and V tiles (K and V in separate mbarrier rings).  Each Q tile has its own soft-max group of
// 128 threads, one thread per (token, head) row holding all 128 key columns of its TMEM lane: no shuffles, no exchange, no
// CTA-wide barrier in the tile loop.  Per group and tile
//     S = Q.K^T (TMEM)  ->  soft-max  ->  P (bf16, shared memory, 64 keys at a time)  ->  O += P.V (TMEM)
// with one thread issuing the S products and another the P.V products.  At head_dim 128 O is rescaled in TMEM only when a row
// maximum grew by more than 2^8; at head_dim 64 whenever it grew (kLazy below).
//
// Bound: the special-function unit (one exponential per (row, key): 2048 cycles per pair of tiles) and the 32 MMAs of the
// pair (about 90 cycles each).  What has to be kept out of the way is the chain S -> soft-max -> P.V: with P written back
// over S in tensor memory the next S could not start before the last P.V, and the chain (5600 cycles per pair, the same
// without any exponential) was what the kernel took.  P in shared memory frees S as soon as it is in registers, so the next
// tile's S runs under this tile's soft-max and P.V under the next one's.  64 keys of P per group leave room for two K and
// two V tiles.  Multiply-adds and sums take two columns per instruction.  Measured at Hq = 64, B = 8, T = 8192: window 512
// 2.13 -> 1.35 ms, compressed (without the selection) 1.32 -> 0.88 ms; the tile loop is at 3900 cycles per pair.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kTokT = 8;                      // tokens per Q tile
constexpr int kTok = 16;                      // tokens per item (two Q tiles)
constexpr int kThreads = 384;                 // warps 0, 3 TMA, 1 S products, 2 P.V products, 4-7 / 8-11 soft-max groups
constexpr int kGroup = 128;
constexpr uint32_t PANEL = 128 * 128;         // [128 rows][64 columns] bf16
constexpr uint32_t kTmemCols = 512;           // S0 0..127, S1 128..255, O0 256.., O1 384..
constexpr int KST = 2, VST = 2;               // ring slots (the producers index them with c & 1)
constexpr uint32_t kMisc = 256;               // barriers, tmem slot, abort flag
template <int D>
constexpr uint32_t kSmem = (D / 64) * PANEL * (2 + KST + VST) + 2 * PANEL + kMisc + 3 * D * 4 + 1024;
// By how much (log2) a row's maximum may outgrow the one its exponentials refer to.  With 0 the largest P of a row is 1, which
// bf16 holds exactly; with 8 it is rounded like the others.  Window 512, 1024 tokens, N(0,1), error of o against fp64:
// 2.01 to 2.03e-3 with 0, 2.05 to 2.07e-3 with 8.  The mma.sync kernel that did head_dim 64 before had 0, so that stays.
template <int D>
constexpr float kLazy = D == 64 ? 0.f : 8.f;

struct Sched {
  int first, n;   // first key tile of the item and their number
};

template <int MODE>
__device__ __forceinline__ Sched make_sched(const DenseArgs& a, const SeqTile& st) {
  Sched s = {0, 0};
  if (st.t0 >= st.Tq) return s;
  const int t0 = a.seq.q0 + st.t0;                        // positions in the sequence
  const int tmax = min(a.seq.q0 + st.Tq - 1, t0 + kTok - 1);
  if (MODE == 0) {
    s.first = max(0, t0 - a.window + 1) / 128;
    s.n = tmax / 128 - s.first + 1;
  } else {
    int nvis = st.Tc;
    if (a.causal) nvis = (tmax < a.cblock) ? 0 : min(st.Tc, (tmax - a.cblock) / a.cstride + 1);
    s.n = (nvis + 127) / 128;
  }
  return s;
}

template <int D, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    dense_fwd2_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const DenseArgs a) {
  after_previous();
  constexpr int NP = D / 64;                  // 64-channel panels
  constexpr uint32_t TILE = NP * PANEL;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q_s = sbase, p_s = sbase + 2 * TILE, k_ring = p_s + 2 * PANEL, v_ring = k_ring + KST * TILE,
                 misc = v_ring + VST * TILE;
  // barriers (8 bytes each); pairs are indexed by group or ring slot
  const uint32_t q_full = misc, q_free = misc + 8, k_full0 = misc + 16, k_empty0 = misc + 32, v_full0 = misc + 48,
                 v_empty0 = misc + 64, s_full0 = misc + 80, s_free0 = misc + 96, p_full0 = misc + 112, p_free0 = misc + 128,
                 o_free0 = misc + 144, tmem_slot = misc + 160;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + (misc - sbase) + 168);
  float* gw = reinterpret_cast<float*>(sgen + (misc - sbase) + kMisc);         // [3][D] gate weights (fp32), mode 1
  const bool do_gate = MODE == 1 && a.gate_w != nullptr;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    // the Q tiles go back to the producer when the item's last score MMA has completed and, when the gate projection
    // is fused in, every soft-max thread has read its Q row
    mbar_init(q_free, do_gate ? 1 + 2 * kGroup : 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(k_full0 + 8 * i, 1);
      mbar_init(k_empty0 + 8 * i, 1);
      mbar_init(v_full0 + 8 * i, 1);
      mbar_init(v_empty0 + 8 * i, 1);
      mbar_init(s_full0 + 8 * i, 1);
      mbar_init(s_free0 + 8 * i, kGroup);
      mbar_init(p_full0 + 8 * i, kGroup);     // two phases per tile: P of keys 0-63, of keys 64-127
      mbar_init(p_free0 + 8 * i, 1);          // the same two phases: that half's P.V has completed
      mbar_init(o_free0 + 8 * i, kGroup);
    }
    fence_mbar_init();
  }
  if (do_gate)
    for (int i = threadIdx.x; i < 3 * D; i += kThreads) gw[i] = __bfloat162float(a.gate_w[i]);
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));

  const int HG = a.Hq / 16;
  const int G16 = (a.Hq / a.Hk) / 16;
  const int ntile = seq_tiles_dev(a.seq, kTok);
  const int total = HG * ntile;   // (checked on the host: fits 31 bits)

  // Registers: 384 threads are launched with 168 each (64512); 128 x 72 + 256 x 216 = 64512 (an inc that the launch pool
  // cannot satisfy blocks for ever).
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 0 || warp == 3) {
    // ------------------------------- TMA producers: Q and K (warp 0), V (warp 3) -------------------------
    // These, the products P.V and at head_dim 64 also S are issued under a lane number, not elected (elect_one).  Compressed branch, 64
    // heads, 8 x 8192 tokens: all elected 1037 us, none 975, P.V alone 1069, TMA alone 980, S alone 979; 2 x 4096 tokens 99.3, 95.7, 100.9,
    // 98.8, 95.8; 2 x 2080 tokens, 32 heads 23.3, 24.2, 24.5, 24.0, 23.9.  P.V issued in one go gets ahead of the other group's S, which the
    // soft-max waits for.  head_dim 64, window, 8 x 4096 tokens, 64 heads: all elected 658, none 639, S alone 646; 3 x 1999, 32 heads: 66.5,
    // 67.8, 67.5.
    const bool is_k = warp == 0;
    const uint32_t full0 = is_k ? k_full0 : v_full0, empty0 = is_k ? k_empty0 : v_empty0, ring = is_k ? k_ring : v_ring;
    const CUtensorMap* tm = is_k ? &tmK : &tmV;
    uint32_t c = 0, ic = 0;
    int good = 1;
    for (int item = blockIdx.x; good && item < total; item += gridDim.x) {
      const int hg = item % HG;
      const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
      if (st.t0 >= st.Tq) continue;
      const Sched sc = make_sched<MODE>(a, st);
      const int hk = hg / G16;
      if (is_k) {
        if (lane == 0) {
          good = mbar_wait_abortable(q_free, (ic & 1) ^ 1, 101, abort_flag) ? 1 : 0;
          if (good) mbar_expect_tx(q_full, 2 * TILE);
        }
        good = __shfl_sync(0xffffffffu, good, 0);
        if (good && lane < 2 * NP)   // lane = NP * tile + panel
          tma_load_3d(q_s + (lane / NP) * TILE + (lane % NP) * PANEL, &tmQ, q_full, (lane % NP) * 64, hg * 16,
                      (int)st.row0 + st.t0 + (lane / NP) * kTokT);
      }
      for (int i = 0; good && i < sc.n; ++i, ++c) {
        const uint32_t sl = c & 1;
        if (lane == 0) {
          good = mbar_wait_abortable(empty0 + 8 * sl, ((c >> 1) & 1) ^ 1, 102, abort_flag) ? 1 : 0;
          if (good) mbar_expect_tx(full0 + 8 * sl, TILE);
        }
        good = __shfl_sync(0xffffffffu, good, 0);
        if (good && lane < NP)
          tma_load_4d(ring + sl * TILE + lane * PANEL, tm, full0 + 8 * sl, lane * 64, hk, (sc.first + i) * 128, st.b);
      }
      ++ic;
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer: S ---------------------------------------------------
    // S of a group's tile c as soon as its K tile has landed and the group holds tile c - 1 in registers
    if (D == 128 ? elect_one() : lane == 0) {   // (see the producers)
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      uint32_t c = 0, ic = 0;     // tiles so far; items so far
      bool ok = true;
      const uint64_t dq_base = umma_smem_desc(q_s, 0, 1024), dk_base = umma_smem_desc(k_ring, 0, 1024);
      for (int item = blockIdx.x; ok && item < total; item += gridDim.x) {
        const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
        if (st.t0 >= st.Tq) continue;
        const int nt = make_sched<MODE>(a, st).n;
        ok = mbar_wait_abortable(q_full, ic & 1, 103, abort_flag);
        for (int i = 0; ok && i < nt; ++i, ++c) {
          const uint32_t ks_ = c % KST;
          ok = mbar_wait_abortable(k_full0 + 8 * ks_, (c / KST) & 1, 104, abort_flag);
          const uint64_t dk = umma_desc_advance(dk_base, ks_ * TILE);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (ok && c > 0) ok = mbar_wait_abortable(s_free0 + 8 * g, (c - 1) & 1, 105, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint64_t dq = umma_desc_advance(dq_base, g * TILE);
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
              const uint32_t off = (ks >> 2) * PANEL + (ks & 3) * 32;
              umma_ss(tmem + g * 128, umma_desc_advance(dq, off), umma_desc_advance(dk, off), idesc_s, ks ? 1u : 0u);
            }
            umma_commit(s_full0 + 8 * g);
          }
          umma_commit(k_empty0 + 8 * ks_);
        }
        umma_commit(q_free);
        ++ic;
      }
    }
  } else if (warp == 2) {
    // ------------------------------- MMA issuer: P.V -------------------------------------------------
    if (lane == 0) {   // (see the producers)
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, D, 0, 1);
      uint32_t c0 = 0;            // tiles of the items before
      uint32_t npi = 0;           // items with tiles so far (= o_free phases the groups will have arrived on)
      bool ok = true;
      const uint64_t dp_base = umma_smem_desc(p_s, 0, 1024), dv_base = umma_smem_desc(v_ring, PANEL, 1024);
      for (int item = blockIdx.x; ok && item < total; item += gridDim.x) {
        const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
        if (st.t0 >= st.Tq) continue;
        const int nt = make_sched<MODE>(a, st).n;
        int n[2] = {0, 0};        // halves issued, per group
        uint64_t t_idle = 0;
        while (ok && (n[0] < 2 * nt || n[1] < 2 * nt)) {
          bool progressed = false;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (n[g] >= 2 * nt || !mbar_test(p_full0 + 8 * g, n[g] & 1)) continue;
            const uint32_t c = c0 + (n[g] >> 1), vs = c % VST;
            const int half = n[g] & 1;
            if (!half && !mbar_test(v_full0 + 8 * vs, (c / VST) & 1)) continue;
            // the epilogue of the group's previous item must have read O before this item's first P.V overwrites it
            if (n[g] == 0 && npi > 0 && !mbar_test(o_free0 + 8 * g, (npi - 1) & 1)) continue;
            tc_fence_after();
            const uint64_t dp = umma_desc_advance(dp_base, g * PANEL), dv = umma_desc_advance(dv_base, vs * TILE + half * 8192);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ss(tmem + 256 + g * 128, umma_desc_advance(dp, ks * 32), umma_desc_advance(dv, ks * 2048), idesc_pv,
                      (n[g] > 0 || ks) ? 1u : 0u);
            umma_commit(p_free0 + 8 * g);
            ++n[g];
            if (half && n[g ^ 1] >= n[g]) umma_commit(v_empty0 + 8 * vs);   // the other group is done with this V tile too
            progressed = true;
          }
          if (progressed) {
            t_idle = 0;
          } else {   // bounded: the abort flag of another role, or ~2 s without progress, ends the loop
            if (*abort_flag) ok = false;
            const uint64_t now = global_timer_ns();
            if (t_idle == 0) t_idle = now;
            else if (now - t_idle > 2000000000ull) {
              atomicCAS(&g_dev_error, 0, 110);
              *abort_flag = 1;
              ok = false;
            }
          }
        }
        c0 += nt;
        if (nt > 0) ++npi;
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------- soft-max groups ------------------------------------------------
    const int quad = warp & 3;
    const int g = (warp - 4) >> 2;                // group = Q tile
    const int row = 32 * quad + lane;             // TMEM lane == Q tile row = (token, head)
    const int tl = row >> 4, head = row & 15;
    const uint32_t lane_addr = (uint32_t)(32 * quad) << 16;
    const uint32_t s_col = tmem + lane_addr + g * 128, o_col = tmem + lane_addr + 256 + g * 128;
    // (head_dim 64 takes scales of any sign, as it did on mma.sync: negative ones by negating the scores, zero as nearly so,
    // since
    // masked scores are -inf)
    const bool neg = D == 64 && a.scale < 0.f;
    const float sl2 = (D == 128 ? a.scale : a.scale == 0.f ? 1e-30f : fabsf(a.scale)) * kLog2e;
    const uint64_t sl22 = pack_f32x2(sl2, sl2);
    const uint32_t s_full = s_full0 + 8 * g, s_free = s_free0 + 8 * g, p_full = p_full0 + 8 * g, p_free = p_free0 + 8 * g,
                   o_free = o_free0 + 8 * g;
    uint8_t* prow = sgen + (p_s - sbase) + g * PANEL + row * 128;
    uint32_t c = 0, ic = 0;     // tiles so far; items so far
    bool ok = true;
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      const int hg = item % HG;
      const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
      if (st.t0 >= st.Tq) continue;
      const Sched sc = make_sched<MODE>(a, st);
      const int tloc = st.t0 + g * kTokT + tl;   // local query row
      const int t = a.seq.q0 + tloc;             // its sequence position
      const bool live = tloc < st.Tq;
      const long long orow = (st.row0 + tloc) * a.Hq + hg * 16 + head;
      // the row's valid keys are one interval [klo, khi)
      int klo = 0, khi;
      if (MODE == 0) {
        klo = t - a.window + 1;
        khi = t + 1;
      } else {
        khi = st.Tc;
        if (a.causal) khi = (t < a.cblock) ? 0 : min(st.Tc, (t - a.cblock) / a.cstride + 1);
      }
      if (!live) khi = 0;
      float m_run = -INFINITY, l_run = 0.f;     // soft-max state (log2 domain)
      if (do_gate) {
        // gate projection of this row from the resident Q tile (nn.Linear(head_dim, 3), no activation)
        ok = mbar_wait_abortable(q_full, ic & 1, 106, abort_flag) && ok;
        float acc0 = 0.f, acc1 = 0.f, acc2 = 0.f;
        const uint8_t* qrow = sgen + (q_s - sbase) + g * TILE + row * 128;
#pragma unroll
        for (int ch = 0; ch < D / 8; ++ch) {
          const uint4 qq = *reinterpret_cast<const uint4*>(qrow + (ch >> 3) * PANEL + (((ch & 7) ^ (row & 7)) << 4));
          const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&qq);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h2[e]);
            const int d0 = ch * 8 + 2 * e;
            acc0 = fmaf(f.x, gw[d0], fmaf(f.y, gw[d0 + 1], acc0));
            acc1 = fmaf(f.x, gw[D + d0], fmaf(f.y, gw[D + d0 + 1], acc1));
            acc2 = fmaf(f.x, gw[2 * D + d0], fmaf(f.y, gw[2 * D + d0 + 1], acc2));
          }
        }
        mbar_arrive(q_free);
        if (live && ok) {
          const float b0 = a.gate_b ? __bfloat162float(a.gate_b[0]) : 0.f, b1 = a.gate_b ? __bfloat162float(a.gate_b[1]) : 0.f,
                      b2 = a.gate_b ? __bfloat162float(a.gate_b[2]) : 0.f;
          a.g_out[0][orow] = __float2bfloat16(acc0 + b0);
          a.g_out[1][orow] = __float2bfloat16(acc1 + b1);
          a.g_out[2][orow] = __float2bfloat16(acc2 + b2);
        }
      }
      for (int i = 0; i < sc.n; ++i, ++c) {
        const int j0 = (sc.first + i) * 128;
        const int lo = klo - j0, hi = khi - j0;
        ok = mbar_wait_abortable(s_full, c & 1, 107, abort_flag) && ok;
        tc_fence_after();
        float s[128];
#pragma unroll
        for (int q = 0; q < 4; ++q) tmem_ld32(s_col + q * 32, *reinterpret_cast<float(*)[32]>(&s[q * 32]));
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(s_free);   // S is in registers: the next tile's S may overwrite it
        if (D == 64 && neg) {
#pragma unroll
          for (int e = 0; e < 128; ++e) s[e] = -s[e];
        }
        // One straight block of code for whole and masked tiles: every branch inside it would drain the exponentials in
        // flight (per-chunk branches that skipped empty chunks cost 800 of 2600 cycles per tile).
        if (!__all_sync(0xffffffffu, lo <= 0 && hi >= 128)) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int l0 = min(max(lo - 32 * q, 0), 32), h0 = min(max(hi - 32 * q, 0), 32);   // valid columns of this chunk
            const unsigned valid = h0 > l0 ? (0xffffffffu >> (32 - (h0 - l0))) << l0 : 0u;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (!(valid & (1u << e))) s[32 * q + e] = -INFINITY;
          }
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 128; e += 8)
#pragma unroll
          for (int q = 0; q < 4; ++q) mx[q] = max3f(mx[q], s[e + 2 * q], s[e + 2 * q + 1]);
        const float mtile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2;   // sl2 > 0: the maximum of the scaled scores
        // Lazy rescale (head_dim 128): the reference maximum follows the true maximum only when that has grown by more than
        // 2^8, so exponentials stay below 256 and the TMEM round trip that rescales O is rare.
        const float mtrue = fmaxf(m_run, mtile);
        const float mnew = (mtrue > m_run + kLazy<D> || m_run == -INFINITY) ? mtrue : m_run;
        const float muse = (mnew == -INFINITY) ? 0.f : mnew;
        const float alpha = ex2(m_run - muse);   // 0 when m_run = -inf
        const bool moved = (mnew != m_run) && (m_run > -INFINITY);
        m_run = mnew;
        if (i > 0 && __any_sync(0xffffffffu, moved)) {
          ok = mbar_wait_abortable(p_free, 1, 108, abort_flag) && ok;   // the previous tile's P.V has completed
          tc_fence_after();
#pragma unroll 1
          for (int q = 0; q < D / 16; ++q) {
            float o[16];
            tmem_ld16(o_col + q * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] *= alpha;
            tmem_st16(o_col + q * 16, o);
          }
          tmem_st_wait();
          tc_fence_before();
        }
        const uint64_t nm2 = pack_f32x2(-muse, -muse);
        uint64_t r0 = 0, r1 = 0;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {   // 64 keys at a time
          uint32_t pk[32];
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float* x = s + 64 * hh + 2 * e;
            const uint64_t x0 = fma_f32x2(pack_f32x2(x[0], x[1]), sl22, nm2), x1 = fma_f32x2(pack_f32x2(x[2], x[3]), sl22, nm2);
            const float p0 = ex2(lo_f32x2(x0)), p1 = ex2(hi_f32x2(x0)), p2 = ex2(lo_f32x2(x1)), p3 = ex2(hi_f32x2(x1));
            r0 = add_f32x2(r0, pack_f32x2(p0, p1));
            r1 = add_f32x2(r1, pack_f32x2(p2, p3));
            pk[e] = pack_bf16(p0, p1);
            pk[e + 1] = pack_bf16(p2, p3);
          }
          // the P.V of the half before has read this buffer
          if (c > 0 || hh) ok = mbar_wait_abortable(p_free, hh ^ 1, 108, abort_flag) && ok;
#pragma unroll
          for (int ch = 0; ch < 8; ++ch)
            *reinterpret_cast<uint4*>(prow + ((ch ^ (row & 7)) << 4)) = make_uint4(pk[4 * ch], pk[4 * ch + 1], pk[4 * ch + 2], pk[4 * ch + 3]);
          fence_proxy_async();
          mbar_arrive(p_full);
        }
        l_run = l_run * alpha + ((lo_f32x2(r0) + hi_f32x2(r0)) + (lo_f32x2(r1) + hi_f32x2(r1)));
      }
      // ---- epilogue of the item ----------------------------------------------------------------------
      {
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        if (sc.n > 0) {
          ok = mbar_wait_abortable(p_free, 1, 109, abort_flag) && ok;   // the last P.V has completed
          tc_fence_after();
        }
        // A warp's 32 rows are two tokens x 16 heads.  They are turned through the warp's part of the
        // P buffer, 64 channels at a time, so that a store instruction writes whole 128-byte lines (a thread storing its own
        // row, 16 bytes at a 256-byte stride between lanes, took 6000 cycles per item).
        const int n_live = min(max(st.Tq - (st.t0 + g * kTokT + 2 * quad), 0), 2) * 16;   // rows of this warp that exist
        bf16* obase = a.o + ((st.row0 + st.t0 + g * kTokT + 2 * quad) * a.Hq + hg * 16) * D;   // the first of them
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          uint32_t ov[32];
          if (sc.n > 0) {
            float o[64];
            tmem_ld32(o_col + p * 64, *reinterpret_cast<float(*)[32]>(&o[0]));
            tmem_ld32(o_col + p * 64 + 32, *reinterpret_cast<float(*)[32]>(&o[32]));
            tmem_ld_wait();
            if (p == NP - 1) {
              tc_fence_before();
              mbar_arrive(o_free);   // O has been read: the next item may overwrite it
            }
#pragma unroll
            for (int e = 0; e < 32; ++e) ov[e] = pack_bf16(o[2 * e] * inv, o[2 * e + 1] * inv);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) ov[e] = 0u;
          }
#pragma unroll
          for (int ch = 0; ch < 8; ++ch)
            *reinterpret_cast<uint4*>(prow + ((ch ^ (row & 7)) << 4)) = make_uint4(ov[4 * ch], ov[4 * ch + 1], ov[4 * ch + 2], ov[4 * ch + 3]);
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int r = it * 4 + (lane >> 3), ch = lane & 7;   // row of the warp, 16-byte chunk
            const uint4 x = *reinterpret_cast<const uint4*>(prow + (r - lane) * 128 + ((ch ^ (r & 7)) << 4));
            if (r < n_live && ok) *reinterpret_cast<uint4*>(obase + (long long)((r >> 4) * a.Hq + (r & 15)) * D + p * 64 + ch * 8) = x;
          }
          __syncwarp();
        }
        if (live && ok) a.lse[orow] = l_run > 0.f ? (m_run + log2f(l_run)) * kLn2 : -INFINITY;
      }
      ++ic;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

template <int D, int MODE>
int launch(const DenseArgs& a, cudaStream_t s) {
  CUtensorMap tmQ, tmK, tmV;
  const unsigned long long qd[3] = {(unsigned long long)D, (unsigned long long)a.Hq, (unsigned long long)seq_rows(a.seq)};
  const unsigned long long qs[2] = {(unsigned long long)D * 2, (unsigned long long)a.Hq * D * 2};
  const unsigned qb[3] = {64, 16, (unsigned)kTokT};
  int rc = make_tmap_generic(&tmQ, a.q, 3, qd, qs, qb);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.k, D, a.Hk, a.Lk, a.B, 128);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hk, a.Lk, a.B, 128);
  if (rc) return rc;
  auto kern = dense_fwd2_tc_kernel<D, MODE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem<D>);
  if (e != cudaSuccess) return (int)e;
  const long long total = (long long)(a.Hq / 16) * seq_tiles(a.seq, kTok);
  if (total > 0x7fffffffLL - num_sms()) {
    set_error("dense attention: too many tokens");
    return -33;
  }
  const int grid = (int)(total < num_sms() ? total : num_sms());
  if (grid <= 0) return 0;
  launch_next(kern, grid, kThreads, kSmem<D>, s, tmQ, tmK, tmV, a);
  note_launches(1);
  return (int)cudaGetLastError();
}

}  // namespace

// True when the tcgen05 forward covers this configuration (otherwise the caller uses launch_dense_fwd).
bool dense_fwd_tc_supported(const DenseArgs& a, int head_dim) {
  if (head_dim != 128 && head_dim != 64) return false;
  return a.mode == 0 || a.n_sel <= 0 || score_tc_supported(head_dim, a.pool_k, a.pool_s, a.pool_p, a.n_pool);
}
int launch_dense_fwd2_tc(const DenseArgs& args, int head_dim, cudaStream_t s) {
  DenseArgs a = args;
  a.seq = {a.B, a.Tq, a.q0, a.Lk};
  if (head_dim == 64) return a.mode == 0 ? launch<64, 0>(a, s) : launch<64, 1>(a, s);
  return a.mode == 0 ? launch<128, 0>(a, s) : launch<128, 1>(a, s);
}
int dense_tc2_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
