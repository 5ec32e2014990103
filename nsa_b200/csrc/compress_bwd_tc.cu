// Compression backward as tcgen05 GEMMs, K and V in the same launches, equal-length or ragged sequences (the gradients of
// y[i] = bias + sum_{j<l} x[i*d + j] . W_j; nsa/compression_kv.py:62-171,219-266 and the Conv1d backward of :298-307).
// Rows are (position, head) pairs, heads innermost, as in the forward.  No atomics: every dX element has one writer, the
// dW partials of the splits are added in a fixed order.
//
//   dX[u*d + jj, :] = sum_{r < l/d} dY[u - r, :] . W_{jj + r*d}^T      one CTA: 128 rows (u, head) x a range of the d
//     in-chunk offsets jj.  The l/d shifted dY tiles stay in shared memory (at most 64 KB, so l/d <= 2 here) while W
//     streams; dY rows outside the sequence are cleared after the copy has landed.
//   dW[(j, c), :]   = sum_i x[i*d + j, c] * dY[i, :]                   one CTA: 256 rows (j, c) of dW x a share of the
//     positions; both operands MN-major, two [128 x D] accumulators in TMEM fed by one dY tile.  The four warps that clear
//     rows past a sequence's end also add up the columns of dY (dbias).
//
// Against the mma.sync kernels these replace at such geometries (8 ragged sequences, 38 K tokens, 4 heads, both tensors):
// dX 101 us, dW 100 us + 20 us of reduction.
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kThreads = 256;   // warps 0, 1 TMA, warp 2 MMA, warps 4-7 row fix-up and epilogue

struct Maps {
  CUtensorMap x[2][2];   // x [tok,H,D] as (64 channels, head, jj, u, panel): jj >= tok % d, jj < tok % d
  CUtensorMap w[2];      // [l*D, D] as (64 columns, row), boxes of D rows
  CUtensorMap y[2];      // dY [out_tok,H,D] as (64 channels, head, position, panel)
};

struct Tile {
  long long in0, out0;
  int i0, nin, nout;     // first position of the tile; tokens and positions of the sequence
};

// Tile `t` of P positions: equal lengths by division, else sequence s owns the indices from cu[s] / G + s on.
__device__ __forceinline__ Tile find_tile(const CompressBwdArgs& a, const int* cu, int len, int G, int P, int t) {
  Tile r;
  int s, base;
  if (!cu) {
    const int per = (len + G - 1) / G;
    s = t / per;
    base = s * per;
    r.in0 = (long long)s * a.T;
    r.out0 = (long long)s * a.Tc;
    r.nin = a.T;
    r.nout = a.Tc;
  } else {
    int lo = 0, hi = a.nseq - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (cu[mid] / G + mid <= t) lo = mid; else hi = mid - 1;
    }
    s = lo;
    base = cu[s] / G + s;
    r.in0 = a.cu_in[s];
    r.out0 = a.cu_out[s];
    r.nin = a.cu_in[s + 1] - (int)r.in0;
    r.nout = a.cu_out[s + 1] - (int)r.out0;
  }
  r.i0 = (t - base) * P;
  return r;
}

// clears one 128-byte-swizzled row of NP panels
template <int NP>
__device__ __forceinline__ void clear_row(uint8_t* tile, uint32_t panel, int row) {
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(tile + p * panel + row * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
}

// ------------------------------------------------------------------------------------------------------------------
// dX
// ------------------------------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
    compress_dx_tc_kernel(const __grid_constant__ Maps maps, const CompressBwdArgs a, const int P, const int HB, const int NS) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  constexpr int NP = D / 64;
  constexpr uint32_t PANEL = 128 * 128, A_TILE = NP * PANEL, W_PANEL = D * 128, W_TILE = NP * W_PANEL;
  constexpr int NR = 4;
  const int R = a.l / a.d;                       // 1 or 2
  const uint32_t ring = sbase + 2 * A_TILE, misc = ring + NR * W_TILE;
  auto full_bar = [&](int i) { return misc + 8u * i; };
  auto empty_bar = [&](int i) { return misc + 8u * (NR + i); };
  const uint32_t a_full = misc + 16u * NR, a_ready = a_full + 8, acc_full = a_full + 16, acc_free = a_full + 32,
                 tmem_slot = a_full + 48;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z;
  const int nhg = (a.H + HB - 1) / HB;
  const int h0 = (blockIdx.x % nhg) * HB;
  const Tile t = find_tile(a, a.cu_in, a.T, a.d * P, P, blockIdx.x / nhg);
  if ((long long)t.i0 * a.d >= t.nin || !a.dx[z]) return;
  const int j_lo = a.d * blockIdx.y / NS, j_hi = a.d * (blockIdx.y + 1) / NS;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NR; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(a_full, 1);
    mbar_init(a_ready, 128);
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_free + 8 * i, 128);
    }
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(tmem_slot, 2 * D);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(a_full, (uint32_t)(R * NP * P * HB) * 128);
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sbase + r * A_TILE + p * PANEL, &maps.y[z], a_full, 0, h0, (int)t.out0 + t.i0 - r, p);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      for (int n = 0; n < (j_hi - j_lo) * R; ++n) {
        const int jj = j_lo + n / R, r = n % R;
        const int stage = n % NR;
        if (!mbar_wait(empty_bar(stage), ((n / NR) & 1) ^ 1, DEV_ERR_EMPTY_WAIT)) break;
        mbar_expect_tx(full_bar(stage), W_TILE);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_2d(ring + stage * W_TILE + p * W_PANEL, &maps.w[z], full_bar(stage), p * 64, (jj + r * a.d) * D);
      }
    }
  } else if (warp == 2) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, D, 0, 0);   // both operands K-major (contraction over the outputs)
      bool ok = mbar_wait(a_ready, 0, DEV_ERR_FULL_WAIT);
      int n = 0;
      for (int jj = j_lo; ok && jj < j_hi; ++jj) {
        const int it = jj - j_lo, buf = it & 1;
        if (it >= 2) ok = mbar_wait(acc_free + 8 * buf, ((it >> 1) - 1) & 1, DEV_ERR_EMPTY_WAIT);
        for (int r = 0; ok && r < R; ++r, ++n) {
          const int stage = n % NR;
          ok = mbar_wait(full_bar(stage), (n / NR) & 1, DEV_ERR_FULL_WAIT);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad = umma_smem_desc(sbase + r * A_TILE, 0, 1024), wd = umma_smem_desc(ring + stage * W_TILE, 0, 1024);
#pragma unroll
          for (int s = 0; s < D / 16; ++s)
            umma_ss(tmem + buf * D, umma_desc_advance(ad, (s >> 2) * PANEL + (s & 3) * 32),
                    umma_desc_advance(wd, (s >> 2) * W_PANEL + (s & 3) * 32), idesc, (r | s) ? 1u : 0u);
          umma_commit(empty_bar(stage));
        }
        umma_commit(acc_full + 8 * buf);
      }
    }
  } else if (warp >= 4) {
    const int row = 32 * (warp & 3) + lane;
    const int pos = row / HB, h = h0 + row % HB;
    bool ok = mbar_wait(a_full, 0, DEV_ERR_FULL_WAIT);
    for (int r = 0; r < R; ++r) {
      const int i = t.i0 + pos - r;
      if (row >= P * HB || i < 0 || i >= t.nout) clear_row<NP>(sgen + r * A_TILE, PANEL, row);
    }
    fence_proxy_async();
    mbar_arrive(a_ready);
    for (int jj = j_lo; ok && jj < j_hi; ++jj) {
      const int it = jj - j_lo, buf = it & 1;
      const int tok = (t.i0 + pos) * a.d + jj;
      const bool live = row < P * HB && tok < t.nin && h < a.H;
      uint4* dst = reinterpret_cast<uint4*>(a.dx[z] + ((t.in0 + tok) * a.H + h) * D);
      // All on their way at once, while the products run: two by two between the accumulator's columns each pair cost a round trip
      // to memory (8 x 8192 tokens, 4 KV heads 204 us, now 115; 18530 packed tokens 92 / 55; 2 x 2080 tokens, 2 heads 16.0 / 10.4).
      // Rows gathered into whole lines through shared memory: 225 us, more work per row than the lines saved.
      uint4 prev[D / 8];
      if (a.accumulate && live) {
#pragma unroll
        for (int c = 0; c < D / 8; ++c) prev[c] = dst[c];
      }
      ok = mbar_wait(acc_full + 8 * buf, (it >> 1) & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + buf * D + c * 16, v);
        tmem_ld_wait();
        if (c == D / 16 - 1) {
          tc_fence_before();
          mbar_arrive(acc_free + 8 * buf);
        }
        if (!live) continue;
        if (a.accumulate) {
          const __nv_bfloat162* hp = reinterpret_cast<const __nv_bfloat162*>(prev + 2 * c);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 f = __bfloat1622float2(hp[e]);
            v[2 * e] += f.x;
            v[2 * e + 1] += f.y;
          }
        }
        uint4 o[2];
        __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
        for (int e = 0; e < 8; ++e) ho[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
        dst[2 * c] = o[0];
        dst[2 * c + 1] = o[1];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 2 * D);
}

// ------------------------------------------------------------------------------------------------------------------
// dW: rows of dW in units of 128 = two 64-row panels; a panel is (j, 64 channels).  D = 64: the panels of a unit are two
// different j.
// ------------------------------------------------------------------------------------------------------------------
constexpr int kUnits = 2;   // units per CTA

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
    compress_dw_tc_kernel(const __grid_constant__ Maps maps, const CompressBwdArgs a, const int P, const int HB, const int ntile,
                          const int nsplit) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  constexpr int NP = D / 64;
  constexpr int XP = 2 * kUnits;                 // x panels per stage
  constexpr uint32_t PANEL = 128 * 128, STAGE = (XP + NP) * PANEL;
  constexpr int NR = 2;
  const uint32_t misc = sbase + NR * STAGE;
  auto full_bar = [&](int i) { return misc + 8u * i; };
  auto ready_bar = [&](int i) { return misc + 8u * (NR + i); };
  auto empty_bar = [&](int i) { return misc + 8u * (2 * NR + i); };
  const uint32_t acc_full = misc + 24u * NR, tmem_slot = acc_full + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z, grp = blockIdx.x, split = blockIdx.y;
  const int nhg = (a.H + HB - 1) / HB;
  const long long total = (long long)ntile * nhg;
  const long long n_lo = total * split / nsplit, n_hi = total * (split + 1) / nsplit;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NR; ++i) {
      mbar_init(full_bar(i), 2);
      mbar_init(ready_bar(i), 128);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(acc_full, 1);
    fence_mbar_init();
  }
  if (P * HB < 128) {   // rows that no copy ever writes take part in the contraction: they must be zero
    for (uint32_t i = threadIdx.x * 16; i < NR * STAGE; i += kThreads * 16)
      *reinterpret_cast<uint4*>(sgen + i) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
  }
  if (warp == 2) tmem_alloc(tmem_slot, kUnits * D);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));
  auto tile_of = [&](long long n) { return find_tile(a, a.cu_out, a.Tc, P, P, (int)(n / nhg)); };

  if (warp < 2) {
    // warp 0: the x panels, warp 1: dY
    if (elect_one()) {
      const int rem = (int)(a.total_in % a.d);
      uint32_t k = 0;
      for (long long n = n_lo; n < n_hi; ++n) {
        const Tile t = tile_of(n);
        if (t.i0 >= t.nout) continue;
        const int h0 = (int)(n % nhg) * HB;
        const int stage = k % NR;
        if (!mbar_wait(empty_bar(stage), ((k / NR) & 1) ^ 1, DEV_ERR_EMPTY_WAIT)) break;
        mbar_expect_tx(full_bar(stage), (uint32_t)(P * HB) * 128 * (warp == 0 ? XP : NP));
        const uint32_t st = sbase + stage * STAGE;
        if (warp == 0) {
          const int jj0 = (int)(t.in0 % a.d), u0 = (int)(t.in0 / a.d) + t.i0;
#pragma unroll
          for (int p = 0; p < XP; ++p) {
            const int r = (grp * XP + p) * 64, j = jj0 + r / D, c0 = r % D;   // first dW row of the panel
            const int jj = j % a.d;
            tma_load_5d(st + p * PANEL, &maps.x[z][jj < rem ? 1 : 0], full_bar(stage), 0, h0, jj, u0 + j / a.d, c0 / 64);
          }
        } else {
#pragma unroll
          for (int p = 0; p < NP; ++p)
            tma_load_4d(st + (XP + p) * PANEL, &maps.y[z], full_bar(stage), 0, h0, (int)t.out0 + t.i0, p);
        }
        ++k;
      }
    }
  } else if (warp == 2) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, D, 1, 1);   // both operands MN-major (contraction over the rows)
      uint32_t k = 0;
      bool ok = true;
      for (long long n = n_lo; ok && n < n_hi; ++n) {
        const Tile t = tile_of(n);
        if (t.i0 >= t.nout) continue;
        const int stage = k % NR;
        ok = mbar_wait(ready_bar(stage), (k / NR) & 1, DEV_ERR_FULL_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = sbase + stage * STAGE;
        const uint64_t yd = umma_smem_desc(st + XP * PANEL, PANEL, 1024);
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          const uint64_t xd = umma_smem_desc(st + 2 * u * PANEL, PANEL, 1024);
#pragma unroll
          for (int s = 0; s < 8; ++s)
            umma_ss(tmem + u * D, umma_desc_advance(xd, s * 2048), umma_desc_advance(yd, s * 2048), idesc, (k > 0 || s) ? 1u : 0u);
        }
        umma_commit(empty_bar(stage));
        ++k;
      }
      umma_commit(acc_full);
    }
  } else if (warp >= 4) {
    const int tid = threadIdx.x - 128;
    const int row = 32 * (warp & 3) + lane;      // tile row to clear; TMEM lane in the epilogue
    const int pos = row / HB;
    const int ngrp = gridDim.x;
    float db = 0.f;                              // column tid % D of dY, rows grp, grp + ngrp, ... (tid / D of them)
    uint32_t k = 0;
    bool ok = true;
    for (long long n = n_lo; ok && n < n_hi; ++n) {
      const Tile t = tile_of(n);
      if (t.i0 >= t.nout) continue;
      const int stage = k % NR;
      ok = mbar_wait(full_bar(stage), (k / NR) & 1, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      uint8_t* st = sgen + stage * STAGE;
      const int h0 = (int)(n % nhg) * HB;
      const int npos = min(P, t.nout - t.i0);    // positions of the tile that exist
      if (npos < P && pos >= npos) {
        clear_row<XP + NP>(st, PANEL, row);
        fence_proxy_async();
      }
      if (a.dbias[z]) {
        const int nrow = npos * HB;
        for (int r = grp + (tid / D) * ngrp; r < nrow; r += (128 / D) * ngrp) {
          const int c = tid % D;
          if (h0 + r % HB < a.H)
            db += __bfloat162float(*reinterpret_cast<const bf16*>(st + (XP + (c >> 6)) * PANEL + r * 128 +
                                                                  ((((c & 63) >> 3) ^ (r & 7)) << 4) + (c & 7) * 2));
        }
      }
      mbar_arrive(ready_bar(stage));
      ++k;
    }
    ok = ok && mbar_wait(acc_full, 0, DEV_ERR_FULL_WAIT);
    tc_fence_after();
    const long long nW = (long long)a.l * D * D;
    float* part = a.ws + ((long long)z * nsplit + split) * nW;
    // (the ring is idle: every MMA that read it has completed.)  Whole lines: 2 x 2080 tokens 16.1 -> 14.0 us, 8 x 8192 70.5 -> 67.
    uint8_t* const rows = sgen + (warp & 3) * 32 * D * 4;
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        float v[16];
        if (k > 0) {
          tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + u * D + c * 16, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          *reinterpret_cast<float4*>(staged(rows, D * 4, lane, 4 * c + e)) = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
      }
      __syncwarp();
      const long long r0 = (long long)(grp * kUnits + u) * 128 + 32 * (warp & 3);
      uint4* dst = reinterpret_cast<uint4*>(part + r0 * D);   // the 32 rows are contiguous
#pragma unroll 8
      for (int i = lane; i < 32 * D / 4; i += 32)
        if (r0 + i / (D / 4) < (long long)a.l * D) dst[i] = *staged(rows, D * 4, i / (D / 4), i % (D / 4));
      __syncwarp();
    }
    if (a.dbias[z]) {   // [tensor][split][group][128] behind the dW partials
      float* dp = a.ws + 2 * nsplit * nW + (((long long)z * nsplit + split) * ngrp + grp) * 128;
      dp[tid] = db;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, kUnits * D);
}

// dW = sum of the splits in order, in the caller's layout; the last block of every tensor adds up dbias.
// mode 0: [l*D, D] fp32; 1: [l*D, D] bf16; 2: Conv1d [o][c][j] bf16.  Block = one channel c: rows j*D + c of all j.
template <int D>
__global__ void __launch_bounds__(256) compress_dw_finish_kernel(const CompressBwdArgs a, const int nsplit, const int ngrp) {
  after_previous();
  __shared__ float t[32][D + 1];
  const int z = blockIdx.y, c = blockIdx.x;
  const long long nW = (long long)a.l * D * D;
  if (c == D) {
    if (a.dbias[z] && threadIdx.x < D) {
      const float* dp = a.ws + 2 * nsplit * nW + (long long)z * nsplit * ngrp * 128;
      float s = 0.f;
      for (int i = 0; i < nsplit * ngrp; ++i)
        for (int x = threadIdx.x; x < 128; x += D) s += dp[i * 128 + x];
      if (a.mode == 0)
        static_cast<float*>(a.dbias[z])[threadIdx.x] = s;
      else
        static_cast<bf16*>(a.dbias[z])[threadIdx.x] = __float2bfloat16(s);
    }
    return;
  }
  if (!a.dw[z]) return;
  const float* part = a.ws + (long long)z * nsplit * nW;
  for (int j0 = 0; j0 < a.l; j0 += 32) {
    const int nj = min(32, a.l - j0);
    for (int e = threadIdx.x; e < nj * (D / 4); e += 256) {
      const int j = e / (D / 4), o = (e % (D / 4)) * 4;
      const long long off = ((long long)(j0 + j) * D + c) * D + o;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int k = 0; k < nsplit; ++k) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(part + k * nW + off));
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      if (a.mode == 0) {
        *reinterpret_cast<float4*>(static_cast<float*>(a.dw[z]) + off) = s;
      } else if (a.mode == 1) {
        *reinterpret_cast<uint2*>(static_cast<bf16*>(a.dw[z]) + off) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
      } else {
        t[j][o] = s.x; t[j][o + 1] = s.y; t[j][o + 2] = s.z; t[j][o + 3] = s.w;
      }
    }
    if (a.mode == 2) {
      __syncthreads();
      for (int e = threadIdx.x; e < 32 * D; e += 256) {
        const int o = e >> 5, j = e & 31;
        if (j < nj) static_cast<bf16*>(a.dw[z])[((long long)o * D + c) * a.l + j0 + j] = __float2bfloat16(t[j][o]);
      }
      __syncthreads();
    }
  }
}

struct Geo {
  int HB, P, nhg, ntile_w, ngrp, nsplit;
};

Geo geometry(int nseq, int Tc, long long total_out, bool ragged, int H, int D, int l) {
  Geo g;
  g.HB = H < 128 ? H : 128;
  g.P = compress_tile_positions(H);
  g.nhg = (H + g.HB - 1) / g.HB;
  g.ntile_w = (int)(ragged ? total_out / g.P + nseq : (long long)nseq * ((Tc + g.P - 1) / g.P));
  g.ngrp = (l * D + kUnits * 128 - 1) / (kUnits * 128);
  // as many splits of the positions as keep one CTA per SM over both tensors, but at least two tiles each
  long long ns = num_sms() / (2 * g.ngrp);
  if (ns > (long long)g.ntile_w * g.nhg / 2) ns = (long long)g.ntile_w * g.nhg / 2;
  g.nsplit = (int)(ns < 1 ? 1 : ns);
  return g;
}

template <int D>
int launch(const CompressBwdArgs& a, cudaStream_t s) {
  const Geo g = geometry(a.nseq, a.Tc, a.total_out, a.cu_in != nullptr, a.H, D, a.l);
  Maps m;
  const long long U = a.total_in / a.d, rem = a.total_in % a.d;
  const unsigned long long H = a.H;
  for (int t = 0; t < 2; ++t) {
    const unsigned long long xs[4] = {(unsigned long long)D * 2, H * D * 2, (unsigned long long)a.d * H * D * 2, 128};
    const unsigned long long x0[5] = {64, H, (unsigned long long)a.d, (unsigned long long)U, D / 64};
    const unsigned long long x1[5] = {64, H, (unsigned long long)(rem ? rem : a.d), (unsigned long long)(rem ? U + 1 : U), D / 64};
    const unsigned xb[5] = {64, (unsigned)g.HB, 1, (unsigned)g.P, 1};
    const unsigned long long ys[3] = {(unsigned long long)D * 2, H * D * 2, 128};
    const unsigned long long y0[4] = {64, H, (unsigned long long)a.total_out, D / 64};
    const unsigned yb[4] = {64, (unsigned)g.HB, (unsigned)g.P, 1};
    int rc = make_tmap_generic(&m.x[t][0], a.x[t], 5, x0, xs, xb);
    if (!rc) rc = make_tmap_generic(&m.x[t][1], a.x[t], 5, x1, xs, xb);
    if (!rc) rc = make_tmap_rows2d(&m.w[t], a.w[t], D, (long long)a.l * D, D);
    if (!rc) rc = make_tmap_generic(&m.y[t], a.dy[t], 4, y0, ys, yb);
    if (rc) return rc;
  }
  cudaError_t e;
  if (a.dx[0] || a.dx[1]) {
    const int smem = (2 * 128 + 4 * D) * (D / 64) * 128 + 1024 + 256;
    auto kern = compress_dx_tc_kernel<D>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    const long long gtok = (long long)a.d * g.P;
    const long long gx = (a.cu_in ? a.total_in / gtok + a.nseq : (long long)a.nseq * ((a.T + gtok - 1) / gtok)) * g.nhg;
    // split of the in-chunk offsets: waves times (the shifted dY tiles, about two W tiles' worth, + the W tiles of a share)
    const int R = a.l / a.d;
    int ns = 1;
    long long best = -1;
    for (int k = 1; k <= a.d && k <= 16; k *= 2) {
      const long long cost = (gx * 2 * k + num_sms() - 1) / num_sms() * ((long long)(a.d + k - 1) / k * R + 8);
      if (best < 0 || cost < best) {
        best = cost;
        ns = k;
      }
    }
    launch_next(kern, dim3((unsigned)gx, (unsigned)ns, 2), kThreads, smem, s, m, a, g.P, g.HB, ns);
    note_launches(1);
  }
  if (a.dw[0] || a.dw[1] || a.dbias[0] || a.dbias[1]) {
    const int smem = 2 * (2 * kUnits + D / 64) * 128 * 128 + 1024 + 256;
    auto kern = compress_dw_tc_kernel<D>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    launch_next(kern, dim3((unsigned)g.ngrp, (unsigned)g.nsplit, 2), kThreads, smem, s, m, a, g.P, g.HB, g.ntile_w, g.nsplit);
    launch_next(compress_dw_finish_kernel<D>, dim3(D + 1, 2), 256, 0, s, a, g.nsplit, g.ngrp);
    note_launches(2);
  }
  return (int)cudaGetLastError();
}

}  // namespace

bool compress_bwd_tc_supported(int D, int l, int d) { return (D == 64 || D == 128) && l % d == 0 && l / d <= 2 && l * D % 256 == 0; }

size_t compress_bwd_tc_workspace_bytes(int nseq, int Tc, long long total_out, bool ragged, int H, int D, int l) {
  const Geo g = geometry(nseq, Tc, total_out, ragged, H, D, l);
  return ((size_t)2 * g.nsplit * l * D * D + (size_t)2 * g.nsplit * g.ngrp * 128) * sizeof(float);
}

int launch_compress_bwd_tc(const CompressBwdArgs& a, cudaStream_t s) {
  if (a.total_out <= 0 || a.total_in <= 0) return 0;
  return a.D == 128 ? launch<128>(a, s) : launch<64>(a, s);
}
int compress_bwd_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
