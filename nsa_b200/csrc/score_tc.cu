// Block selection on tcgen05 (head_dim 128, the 5/4/0 pooling of the default block sizes): for every token and 16-head
// group the top n of the pooled soft-max scores over all compressed keys (nsa/torch_attention.py:121-125,51-62 as called
// from nsa/triton_attention.py:465-475).  The [B,Hq,T,Tc] score tensor never exists.
//
// A persistent CTA owns 16 consecutive tokens x 16 heads = two [128 x 128] Q tiles that share one stream of [128 keys x 128]
// tiles of the compressed keys, walked twice: pass A collects every row's maximum and sum, pass B recomputes S, forms
// p = exp(s - max) / sum, pools the 5-wide stride-4 windows inside the thread, sums the 16 heads of a token with a halving
// shuffle butterfly and writes the result to a per-token score vector in shared memory, from which four further warps pick
// the top n (ties to the lower index) while the next item is already being scored.
//
// Bound: the special-function unit, two exponentials per (row, key): 2048 cycles per pair of tiles and pass.  Everything
// else is arranged to stay under that: each group of 128 soft-max threads (one row per thread, all 128 columns of its TMEM
// lane) has two S accumulators, so the tensor core writes the next tile while the group exponentiates this one; the sums of
// pass A go two at a time (fma/add.rn.f32x2, which round like the scalar instructions); the two contributions to a pooled
// block meet by shuffles and plain stores (fp32 atomics in shared memory are compare-and-swap loops).  Measured at Hq = 64,
// B = 8, T = 8192: 1.79 ms (3850 cycles per pair and pass; 3300 at T = 32768).  Scoring inside the compressed attention
// kernel, with one accumulator per group shared with that branch's P, took 3.4 ms (6600 cycles).  The order of every sum
// (four interleaved chains per tile, tiles in order) is fixed: a last-bit change of a score can exchange two blocks.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int D = 128;
constexpr int kTokT = 8;                      // tokens per Q tile
constexpr int kTok = 16;                      // tokens per item
// warpgroup 0: TMA, MMA, two idle warps; warpgroups 1, 2: soft-max groups 0, 1; warpgroup 3: top-n
constexpr int kThreads = 512;
constexpr int kGroup = 128;
constexpr uint32_t PANEL = 128 * 128;
constexpr uint32_t TILE = 2 * PANEL;          // 32 KB
constexpr uint32_t kTmemCols = 512;           // S of (group g, buffer b) at 256 g + 128 b
constexpr uint32_t kMisc = 256;
constexpr int kMaxRing = 4;

// The top n of NT tokens' scores at once (their rounds are independent: one token alone is a chain of about 430 cycles per
// round).  Scores are >= 0, so their bit patterns order like the values.  A lane holds the blocks lane, lane + 32, ... in
// registers (0: none; a score's pattern + 1 otherwise) and its best of them; a round is two warp reductions.
template <int NV, int NT>
__device__ __forceinline__ void pick_top(const float* pl, int pool_floats, int Tc, int n_pool, int n_sel, int* out, long long ostride,
                                         float* dump, int nlive, int lane) {
  unsigned v[NT][NV], best[NT];
  int bi[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    best[t] = 0u;
    bi[t] = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int blk = lane + 32 * i;
      v[t][i] = 0u;
      if (blk < n_pool && t < nlive) {
        const float x = pl[t * pool_floats + blk] / (float)(min(4 * blk + 5, Tc) - 4 * blk);   // average over the window
        if (dump) dump[(long long)t * n_pool + blk] = x;
        v[t][i] = x >= 0.f ? __float_as_uint(x) + 1u : 0u;
      }
      if (v[t][i] > best[t]) {   // the first of equal ones: the lower block
        best[t] = v[t][i];
        bi[t] = i;
      }
    }
  }
  for (int r = 0; r < n_sel; ++r) {
    unsigned top[NT];
    int win[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) top[t] = __reduce_max_sync(0xffffffffu, best[t]);
#pragma unroll
    for (int t = 0; t < NT; ++t) win[t] = __reduce_min_sync(0xffffffffu, (best[t] == top[t] && top[t]) ? lane + 32 * bi[t] : 0x7fffffff);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      if (lane == t && t < nlive) out[t * ostride + r] = top[t] ? win[t] : -1;
      const bool owner = top[t] && (win[t] & 31) == lane;   // retires the block and finds its next best
      unsigned b = 0u;
      int x = 0;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (owner && i == (win[t] >> 5)) v[t][i] = 0u;
        if (v[t][i] > b) {
          b = v[t][i];
          x = i;
        }
      }
      best[t] = b;
      bi[t] = x;
    }
  }
}

// Exchange step of the sum over 16 lanes: lanes differing in bit BIT split the first 2 W values between them.
template <int W, int BIT>
__device__ __forceinline__ void halve(float (&v)[32], int lane) {
  const bool up = (lane & BIT) != 0;
#pragma unroll
  for (int x = 0; x < W; ++x) {
    const float send = up ? v[x] : v[x + W], keep = up ? v[x + W] : v[x];
    v[x] = keep + __shfl_xor_sync(0xffffffffu, send, BIT);
  }
}

__global__ void __launch_bounds__(kThreads, 1)
    score_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const ScoreArgs a,
                    const int QST, const int KST, const int nslot, const int pool_floats) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q_s = sbase, k_ring = sbase + QST * 2 * TILE, misc = k_ring + KST * TILE;
  const uint32_t q_full0 = misc, q_free0 = misc + 16, k_full0 = misc + 32, k_empty0 = misc + 64, s_full0 = misc + 96,
                 s_free0 = misc + 128, pool_full0 = misc + 160, pool_free0 = misc + 176, tmem_slot = misc + 192;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + (misc - sbase) + 200);
  float* pool = reinterpret_cast<float*>(sgen + (misc - sbase) + kMisc);   // [nslot][kTok][pool_floats]
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kMaxRing; ++i) {
      mbar_init(k_full0 + 8 * i, 1);
      mbar_init(k_empty0 + 8 * i, 1);
    }
    for (int i = 0; i < 4; ++i) {   // (group, buffer)
      mbar_init(s_full0 + 8 * i, 1);
      mbar_init(s_free0 + 8 * i, kGroup);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full0 + 8 * i, 1);
      mbar_init(q_free0 + 8 * i, 1);
      mbar_init(pool_full0 + 8 * i, 2 * kGroup);
      mbar_init(pool_free0 + 8 * i, kGroup);
    }
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
  const bool causal = a.score_mode == 1;
  // compressed tiles of one pass: all of the sequence's, or (causal scores) up to the item's last visible key
  auto tiles_of = [&](const SeqTile& st) {
    if (!causal) return (st.Tc + 127) / 128;
    const int tmax = min(a.seq.q0 + st.Tq - 1, a.seq.q0 + st.t0 + kTok - 1);
    const int nvis = tmax < a.cblock ? 0 : min(st.Tc, (tmax - a.cblock) / a.cstride + 1);
    return (nvis + 127) / 128;
  };

  // Registers: 512 threads are launched with 128 each (65536); 128 x 72 + 256 x 176 + 128 x 88 = 65536 (an inc that the
  // launch pool cannot satisfy blocks for ever).
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------- TMA producer ------------------------------------------------
      uint32_t ck = 0, ic = 0;
      if (elect_one()) {
        bool good = true;
        for (int item = blockIdx.x; good && item < total; item += gridDim.x) {
          const int hg = item % HG;
          const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
          const int nt = tiles_of(st);
          if (st.t0 >= st.Tq || nt == 0) continue;
          const uint32_t qs = ic % (uint32_t)QST;   // two Q slots: the next item's tiles land while this one is scored
          good = mbar_wait_abortable(q_free0 + 8 * qs, ((ic / (uint32_t)QST) & 1) ^ 1, 301, abort_flag);
          if (!good) break;
          mbar_expect_tx(q_full0 + 8 * qs, 2 * TILE);
#pragma unroll
          for (int x = 0; x < 4; ++x)   // x = 2 * tile + panel
            tma_load_3d(q_s + (2 * qs + (x >> 1)) * TILE + (x & 1) * PANEL, &tmQ, q_full0 + 8 * qs, (x & 1) * 64, hg * 16,
                        (int)(st.row0 + st.t0) + (x >> 1) * kTokT);
          for (int i = 0; i < 2 * nt; ++i, ++ck) {
            const uint32_t ks = ck % (uint32_t)KST;
            good = mbar_wait_abortable(k_empty0 + 8 * ks, ((ck / (uint32_t)KST) & 1) ^ 1, 302, abort_flag);
            if (!good) break;
            mbar_expect_tx(k_full0 + 8 * ks, TILE);
            const int jt = i < nt ? i : i - nt;
#pragma unroll
            for (int p = 0; p < 2; ++p)
              tma_load_4d(k_ring + ks * TILE + p * PANEL, &tmK, k_full0 + 8 * ks, p * 64, hg / G16, jt * 128, st.b);
          }
          ++ic;
        }
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer ----------------------------------------------------
      if (elect_one()) {
        constexpr uint32_t idesc = umma_idesc_bf16(128, 128, 0, 0);
        uint32_t ck = 0, ic = 0;
        bool ok = true;
        const uint64_t dq0 = umma_smem_desc(q_s, 0, 1024), dk0 = umma_smem_desc(k_ring, 0, 1024);
        for (int item = blockIdx.x; ok && item < total; item += gridDim.x) {
          const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
          const int nt = tiles_of(st);
          if (st.t0 >= st.Tq || nt == 0) continue;
          const uint32_t qs = ic % (uint32_t)QST;
          ok = mbar_wait_abortable(q_full0 + 8 * qs, (ic / (uint32_t)QST) & 1, 303, abort_flag);
          for (int i = 0; ok && i < 2 * nt; ++i, ++ck) {
            const uint32_t ks = ck % (uint32_t)KST, buf = ck & 1;
            ok = mbar_wait_abortable(k_full0 + 8 * ks, (ck / (uint32_t)KST) & 1, 304, abort_flag);
            const uint64_t dk = umma_desc_advance(dk0, ks * TILE);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              // the group holds tile ck - 2 in registers
              if (ok && ck >= 2) ok = mbar_wait_abortable(s_free0 + 8 * (2 * g + buf), ((ck >> 1) - 1) & 1, 305, abort_flag);
              if (!ok) break;
              tc_fence_after();
              const uint64_t dq = umma_desc_advance(dq0, (2 * qs + g) * TILE);
#pragma unroll
              for (int s = 0; s < 8; ++s) {
                const uint32_t off = (s >> 2) * PANEL + (s & 3) * 32;
                umma_ss(tmem + g * 256 + buf * 128, umma_desc_advance(dq, off), umma_desc_advance(dk, off), idesc, s ? 1u : 0u);
              }
              umma_commit(s_full0 + 8 * (2 * g + buf));
            }
            umma_commit(k_empty0 + 8 * ks);
          }
          umma_commit(q_free0 + 8 * qs);
          ++ic;
        }
      }
    }
  } else if (warp >= 12) {
    // ------------------------------- top-n ---------------------------------------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    const int w = warp - 12;
    uint32_t ic = 0;
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      const int hg = item % HG;
      const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
      if (st.t0 >= st.Tq) continue;
      const int n_pool = pool_len_54(st.Tc);
      const int nt = tiles_of(st);
      const uint32_t slot = ic % (uint32_t)nslot;
      float* pl = pool + slot * kTok * pool_floats;
      if (nt == 0) {   // causal scores, nothing visible yet: every score is zero and the lowest blocks win
        for (int tw = w; tw < kTok && st.t0 + tw < st.Tq; tw += 4) {
          const int tt = st.t0 + tw;
          int* out = a.sel_idx + ((st.row0 + tt) * HG + hg) * a.n_sel;
          for (int r = lane; r < a.n_sel; r += 32) out[r] = r < n_pool ? r : -1;
          if (a.sel_scores)
            for (int blk = lane; blk < n_pool; blk += 32)
              a.sel_scores[((long long)(st.b * HG + hg) * st.Tq + tt) * n_pool + blk] = 0.f;
        }
        continue;
      }
      const bool ok = mbar_wait_abortable(pool_full0 + 8 * slot, (ic / (uint32_t)nslot) & 1, 306, abort_flag);
      const int t_w = st.t0 + w * 4, nlive = min(4, st.Tq - t_w);   // this warp's four tokens
      if (ok && nlive > 0) {
        const float* src = pl + w * 4 * pool_floats;
        int* out = a.sel_idx + ((st.row0 + t_w) * HG + hg) * a.n_sel;
        float* dump = a.sel_scores ? a.sel_scores + ((long long)(st.b * HG + hg) * st.Tq + t_w) * n_pool : nullptr;
        const long long os = (long long)HG * a.n_sel;
        if (n_pool <= 128) {
          pick_top<4, 4>(src, pool_floats, st.Tc, n_pool, a.n_sel, out, os, dump, nlive, lane);
        } else if (n_pool <= 512) {
#pragma unroll 1
          for (int u = 0; u < nlive; u += 2)
            pick_top<16, 2>(src + u * pool_floats, pool_floats, st.Tc, n_pool, a.n_sel, out + u * os, os,
                            dump ? dump + (long long)u * n_pool : nullptr, nlive - u, lane);
        } else {
#pragma unroll 1
          for (int u = 0; u < nlive; ++u)
            pick_top<32, 1>(src + u * pool_floats, pool_floats, st.Tc, n_pool, a.n_sel, out + u * os, os,
                            dump ? dump + (long long)u * n_pool : nullptr, 1, lane);
        }
      }
      mbar_arrive(pool_free0 + 8 * slot);
      ++ic;
    }
  } else {
    // ------------------------------- soft-max groups ------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    const int quad = warp & 3;
    const int g = (warp - 4) >> 2;
    const int row = 32 * quad + lane;             // TMEM lane == Q tile row = (token, head)
    const int tl = row >> 4;
    const uint32_t s_col = tmem + ((uint32_t)(32 * quad) << 16) + g * 256;
    const float cmul = causal ? a.scale * kLog2e : kLog2e;
    const uint64_t cmul2 = pack_f32x2(cmul, cmul);   // pass A works on pairs of columns
    uint32_t cs = 0, ic = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      const SeqTile st = seq_tile(a.seq, kTok, ntile - 1 - item / HG);
      const int nt = tiles_of(st);
      if (st.t0 >= st.Tq || nt == 0) continue;
      const int tloc = st.t0 + g * kTokT + tl, t = a.seq.q0 + tloc;
      const bool live = tloc < st.Tq;
      // columns that count: all compressed keys (reference scores) or the row's visible ones (causal)
      int ncol = st.Tc;
      if (causal) ncol = t < a.cblock ? 0 : min(st.Tc, (t - a.cblock) / a.cstride + 1);
      float m = -INFINITY, l = 0.f;
      float s[128];
      auto load_tile = [&](int j0) {
        const uint32_t bar = 8 * (2 * g + (cs & 1));
        ok = mbar_wait_abortable(s_full0 + bar, (cs >> 1) & 1, 307, abort_flag) && ok;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(s_col + (cs & 1) * 128 + c * 32, *reinterpret_cast<float(*)[32]>(&s[c * 32]));
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(s_free0 + bar);   // S is in registers: tile cs + 2 may overwrite this accumulator
        ++cs;
        const int nval = ncol - j0;
        if (nval < 128) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (nval < 32 * (c + 1)) {
#pragma unroll
              for (int e = 32 * c; e < 32 * c + 32; ++e)
                if (e >= nval) s[e] = -INFINITY;
            }
        }
      };
      // ---- pass A: maximum and sum of the soft-max -----------------------------------------------------------
      for (int i = 0; i < nt; ++i) {
        load_tile(i * 128);
        float mx = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
        for (int e = 0; e < 128; e += 8) {
          mx = max3f(mx, s[e], s[e + 1]);
          m1 = max3f(m1, s[e + 2], s[e + 3]);
          m2 = max3f(m2, s[e + 4], s[e + 5]);
          m3 = max3f(m3, s[e + 6], s[e + 7]);
        }
        const float mnew = fmaxf(m, fmaxf(fmaxf(mx, m1), fmaxf(m2, m3)));
        if (mnew > -INFINITY) {
          const float nm = -mnew * cmul;
          const uint64_t nm2 = pack_f32x2(nm, nm);
          uint64_t r01 = 0, r23 = 0;   // four chains of sums, two per register pair
#pragma unroll
          for (int e = 0; e < 128; e += 4) {
            const uint64_t x01 = fma_f32x2(pack_f32x2(s[e], s[e + 1]), cmul2, nm2);
            const uint64_t x23 = fma_f32x2(pack_f32x2(s[e + 2], s[e + 3]), cmul2, nm2);
            r01 = add_f32x2(r01, pack_f32x2(ex2(lo_f32x2(x01)), ex2(hi_f32x2(x01))));
            r23 = add_f32x2(r23, pack_f32x2(ex2(lo_f32x2(x23)), ex2(hi_f32x2(x23))));
          }
          l = l * ex2((m - mnew) * cmul) + ((lo_f32x2(r01) + hi_f32x2(r01)) + (lo_f32x2(r23) + hi_f32x2(r23)));
          m = mnew;
        }
      }
      const float inv = (live && l > 0.f) ? 1.f / l : 0.f;
      const float nm = m > -INFINITY ? -m * cmul : 0.f;
      // ---- pass B: p, pooled per thread, summed over the heads ------------------------------------------------
      const uint32_t slot = ic % (uint32_t)nslot;
      ok = mbar_wait_abortable(pool_free0 + 8 * slot, ((ic / (uint32_t)nslot) & 1) ^ 1, 308, abort_flag) && ok;
      float* pt = pool + (slot * kTok + g * kTokT + tl) * pool_floats;
      const int m8 = lane & 7;
      for (int i = 0; i < nt; ++i) {
        load_tile(i * 128);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          float v[32];   // v[k] = columns 4k..4k+3 of this half, v[16+k] = column 4k (it also ends block k-1)
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float pe[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) pe[u] = ex2(fmaf(s[hh * 64 + 4 * k + u], cmul, nm)) * inv;
            v[k] = (pe[0] + pe[1]) + (pe[2] + pe[3]);
            v[16 + k] = pe[0];
          }
          halve<16, 8>(v, lane);   // sum over the token's 16 heads
          halve<8, 4>(v, lane);
          halve<4, 2>(v, lane);
          halve<2, 1>(v, lane);
          // Lanes 0-7 of the 16 hold the sums of blocks 2 m8, 2 m8 + 1 of this half, lanes 8-15 those of their first columns,
          // which complete the block before: one add each (the last block of a half gets its from the next half).
          const float f1 = __shfl_sync(0xffffffffu, v[1], (lane & 16) + 8 + m8);
          const float f0 = __shfl_sync(0xffffffffu, v[0], (lane & 16) + 8 + ((m8 + 1) & 7));
          float* p0 = pt + i * 32 + hh * 16;
          if (!(lane & 8)) *reinterpret_cast<float2*>(p0 + 2 * m8) = make_float2(v[0] + f1, m8 < 7 ? v[1] + f0 : v[1]);
          __syncwarp();
          if ((lane & 15) == 8 && i + hh > 0) p0[-1] += v[0];
        }
      }
      // Causal scores: behind the item's last visible key lies what the slot held before, and every score is zero.  (Cleared
      // here and
      // not by the warp that reads them: that took 3 % of the kernel in the other mode too.)
      if (causal) {
        const int n_pool = pool_len_54(st.Tc);
        for (int blk = 32 * nt + (lane & 15); blk < n_pool; blk += 16) pt[blk] = 0.f;
      }
      mbar_arrive(pool_full0 + 8 * slot);
      ++ic;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

bool score_tc_supported(int head_dim, int pool_k, int pool_s, int pool_p, int n_pool) {
  return head_dim == 128 && pool_k == 5 && pool_s == 4 && pool_p == 0 && n_pool <= 1024;
}

int launch_score_tc(const ScoreArgs& a, cudaStream_t s) {
  CUtensorMap tmQ, tmK;
  const long long rows = seq_rows(a.seq);
  const unsigned long long qd[3] = {(unsigned long long)D, (unsigned long long)a.Hq, (unsigned long long)rows};
  const unsigned long long qs[2] = {(unsigned long long)D * 2, (unsigned long long)a.Hq * D * 2};
  const unsigned qb[3] = {64, 16, (unsigned)kTokT};
  int rc = make_tmap_generic(&tmQ, a.q, 3, qd, qs, qb);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.ck, D, a.Hk, a.seq.Tc, a.seq.B, 128);
  if (rc) return rc;
  int dev = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  // Two pairs of Q tiles with two slots of compressed keys (sequences up to about 32 K tokens), else one pair with three or
  // two; two score vectors per token if they fit
  const int pool_floats = (a.Tc_max + 127) / 128 * 32;   // whole tiles of 128 compressed keys are stored
  int QST = 2, KST = 2, nslot = 2;
  auto bytes = [&]() { return QST * (int)(2 * TILE) + KST * (int)TILE + (int)kMisc + nslot * kTok * pool_floats * 4 + 1024; };
  if (bytes() > max_smem) {
    QST = 1;
    KST = 3;
  }
  if (bytes() > max_smem) nslot = 1;
  if (bytes() > max_smem) KST = 2;
  if (bytes() > max_smem) {
    set_error("block selection: the pooled-score vector (%d compressed positions) does not fit in shared memory", a.Tc_max);
    return -31;
  }
  const int smem = bytes();
  cudaError_t e = cudaFuncSetAttribute(score_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const long long total = (long long)(a.Hq / 16) * seq_tiles(a.seq, kTok);
  if (total > 0x7fffffffLL - num_sms()) {
    set_error("block selection: too many tokens");
    return -33;
  }
  const int grid = (int)(total < num_sms() ? total : num_sms());
  if (grid <= 0) return 0;
  launch_next(score_tc_kernel, grid, kThreads, smem, s, tmQ, tmK, a, QST, KST, nslot, pool_floats);
  note_launches(1);
  return (int)cudaGetLastError();
}
int score_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
