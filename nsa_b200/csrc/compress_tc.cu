// Compression forward as one tcgen05 GEMM, K and V in the same launch, equal-length or ragged sequences:
//     Y[i, :] = bias + sum_{j<l} X[i*d + j, :] . W_j          (nsa/compression_kv.py:21-57 and :298-307)
// The overlapping windows are never materialised and sequences may start at any token.  x [tok,H,D] is viewed as
// (channel, head, offset-in-stride jj, stride chunk u, 64-channel panel): window i of a sequence that starts at token in0
// is, at in-block offset j, the row (u = (in0 + j) / d + i, jj = (in0 + j) % d), so the A tile of one j -- 128 rows =
// (positions x heads), heads innermost -- is one TMA box per panel whose positions are d tokens apart.  The view needs
// tok % d handled: chunks jj < tok % d have one more u than the others, hence two maps.  Rows past a sequence's end read
// the next sequence's tokens (or zeros) and are not stored.  The D rows of W [l*D, D] of that j are the MN-major B operand
// (rows = contraction index, 128-byte swizzled; in its descriptor the leading byte offset is the distance between the two
// 64-column panels and the stride byte offset the 1024 bytes between 8-row groups).
// Warps 0 and 1 stream the A and W tiles, 64 channels of a j per stage, through an mbarrier ring, one thread of warp 2 issues
// tcgen05.mma into [128 x columns] fp32 accumulators in TMEM, warps 4-7 read them back with tcgen05.ld, add the bias and store
// bf16.
//
// A CTA is a serial chain of l * D / 64 stages however few rows there are; one stage takes 300 cycles with half of the columns,
// about what its 24 KB take from L2 (600 with a 64-bit division per stage and TMA instructions whose operands differ by lane;
// without these, and with the tile that fits the rows, below: 5008 tokens of 4 heads 22.6 -> 15.6 us, eight sequences with 38100
// tokens in all 54 -> 43 us).
// Where the caller allows it (`split`) the contraction is split over a cluster of up to eight CTAs when
// that shortens the waves; the partial accumulators meet in distributed shared memory and are added in rank order.  The
// package does not allow it anywhere: a block selection turns last-bit differences of ck into other blocks, and with one
// order of summation (the same bits as a chain of mma.sync steps, whatever tile a call gets) a sequence selects the same blocks
// whatever batch it is in and however its cache was built.
#include <algorithm>

#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxRing = 8;
constexpr uint32_t A_TILE = 128 * 128;   // [128 rows][64 channels]
constexpr uint32_t W_TILE = 64 * 128;    // [64 channels of x][64 channels of y]

// A CTA's tile: MT times 128 rows (or the first P * HB of each) x NC of the D output channels.  A stage is 64 channels of one j.
template <int MT, int NC>
constexpr uint32_t kStage = MT * A_TILE + NC / 64 * W_TILE;
template <int MT, int NC>
constexpr int kRing = 200 * 1024 / kStage<MT, NC> < kMaxRing ? 200 * 1024 / kStage<MT, NC> : kMaxRing;

struct Maps {
  CUtensorMap x[2][2];   // [tensor][jj >= tok % d, jj < tok % d]
  CUtensorMap w[2];
};

__device__ __forceinline__ float4 cluster_ld4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int D, int MT, int NC>
__global__ void __launch_bounds__(kThreads, 1)
    compress_fwd_tc_kernel(const __grid_constant__ Maps maps, const CompressFwdArgs a, const int P, const int HB, const int ks) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  constexpr int NP = D / 64;                       // 64-channel panels of x
  constexpr int NCOL = D / NC;                     // CTAs that share a tile's columns
  constexpr uint32_t STAGE = kStage<MT, NC>;
  constexpr int NR = kRing<MT, NC>;
  constexpr int RS = D + 4;                        // row stride of the partial tile in shared memory (floats)
  static_assert(MT > 1 || NC < D || 128 * RS * 4 <= NR * STAGE, "the partial tile reuses the ring");
  const uint32_t bar_base = sbase + NR * STAGE;
  auto full_bar = [&](int i) { return bar_base + 8u * i; };
  auto empty_bar = [&](int i) { return bar_base + 8u * (NR + i); };
  const uint32_t acc_bar = bar_base + 16u * NR;
  const uint32_t tmem_slot = acc_bar + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z / NCOL, col0 = blockIdx.z % NCOL * NC, rank = blockIdx.y;
  const int nhg = (a.H + HB - 1) / HB;
  const int tile = blockIdx.x / nhg, h0 = (blockIdx.x % nhg) * HB;

  // ---- the tile's sequence, first position and limits -----------------------------------------------------------
  long long in0, out0;
  int i0, iend;
  if (!a.cu_in) {
    const int tps = (a.Tc + MT * P - 1) / (MT * P);
    const int s = tile / tps;
    in0 = (long long)s * a.T;
    out0 = (long long)s * a.Tc;
    i0 = (tile % tps) * (MT * P);
    iend = a.Tc;
  } else {
    // sequence s owns the tile indices from cu_row[s] / (MT P) + s on (never fewer than it has tiles)
    int lo = 0, hi = a.nseq - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.cu_row[mid] / (MT * P) + mid <= tile) lo = mid; else hi = mid - 1;
    }
    const int r0 = a.cu_row[lo], first = a.first ? a.first[lo] : 0;
    in0 = a.cu_in[lo];
    out0 = a.cu_out[lo];
    i0 = first + (tile - (r0 / (MT * P) + lo)) * (MT * P);
    iend = first + a.cu_row[lo + 1] - r0;
  }
  if (i0 >= iend) return;   // every CTA of the cluster works on the same tile

  if (threadIdx.x == 0) {
    for (int i = 0; i < NR; ++i) {
      mbar_init(full_bar(i), 2);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(acc_bar, 1);
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(tmem_slot, MT * NC);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));
  const int j_lo = a.l * rank / ks, j_hi = a.l * (rank + 1) / ks;   // this CTA's share of the contraction
  const int nst = (j_hi - j_lo) * NP;                               // its stages

  const int row = 32 * (warp & 3) + lane;
  const int pos = row / HB, h = h0 + row % HB;
  bool ok = true;
  if (warp == 0) {
    if (elect_one()) {
      const int rem = (int)(a.total_in % a.d);
      int jj = (int)((in0 + j_lo) % a.d), u = (int)((in0 + j_lo) / a.d) + i0;
      for (int n = 0; n < nst; ++n) {
        const int stage = n % NR, p = n % NP;
        if (!mbar_wait(empty_bar(stage), (n / NR & 1) ^ 1, DEV_ERR_EMPTY_WAIT)) break;
        mbar_expect_tx(full_bar(stage), (uint32_t)(P * HB) * 128 * MT);
        const CUtensorMap* map = &maps.x[z][jj < rem ? 1 : 0];
#pragma unroll
        for (int t = 0; t < MT; ++t)
          tma_load_5d(sbase + stage * STAGE + t * A_TILE, map, full_bar(stage), 0, h0, jj, u + t * P, p);
        if (p == NP - 1 && ++jj == a.d) {
          jj = 0;
          ++u;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      for (int n = 0; n < nst; ++n) {
        const int stage = n % NR;
        if (!mbar_wait(empty_bar(stage), (n / NR & 1) ^ 1, DEV_ERR_EMPTY_WAIT)) break;
        mbar_expect_tx(full_bar(stage), NC / 64 * W_TILE);
#pragma unroll
        for (int c = 0; c < NC / 64; ++c)
          tma_load_2d(sbase + stage * STAGE + MT * A_TILE + c * W_TILE, &maps.w[z], full_bar(stage), col0 + c * 64, j_lo * D + n * 64);
      }
    }
  } else if (warp == 2) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, NC, 0, 1);
      for (int n = 0; n < nst; ++n) {
        const int stage = n % NR;
        if (!mbar_wait(full_bar(stage), (n / NR) & 1, DEV_ERR_FULL_WAIT)) break;
        tc_fence_after();
        const uint32_t a_s = sbase + stage * STAGE;
        const uint64_t wd = umma_smem_desc(a_s + MT * A_TILE, W_TILE, 1024);
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const uint64_t ad = umma_smem_desc(a_s + t * A_TILE, 0, 1024);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            umma_ss(tmem + t * NC, umma_desc_advance(ad, s * 32), umma_desc_advance(wd, s * 2048), idesc, (n | s) ? 1u : 0u);
        }
        umma_commit(empty_bar(stage));
      }
      umma_commit(acc_bar);
    }
  } else if (warp >= 4) {
    ok = mbar_wait(acc_bar, 0, DEV_ERR_FULL_WAIT);
    tc_fence_after();
    float* part = reinterpret_cast<float*>(sgen) + row * RS;
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const int i = i0 + t * P + pos;
      const bool live = row < P * HB && i < iend && h < a.H;
      bf16* dst = a.y[z] + ((out0 + i) * a.H + h) * D + col0;
      const bf16* bias = a.bias[z] ? a.bias[z] + col0 : nullptr;   // (of any alignment)
#pragma unroll
      for (int c = 0; c < NC / 16; ++c) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + t * NC + c * 16, v);
        tmem_ld_wait();
        if (ks > 1) {   // (MT = 1, NC = D) the ring is idle: every MMA that read it has completed
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<float4*>(part + c * 16 + 4 * e) = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
        } else if (ok && live) {
          uint4 o[2];
          __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float x0 = v[2 * e], x1 = v[2 * e + 1];
            if (bias) {
              x0 += __bfloat162float(bias[c * 16 + 2 * e]);
              x1 += __bfloat162float(bias[c * 16 + 2 * e + 1]);
            }
            ho[e] = __floats2bfloat162_rn(x0, x1);
          }
          *reinterpret_cast<uint4*>(dst + c * 16) = o[0];
          *reinterpret_cast<uint4*>(dst + c * 16 + 8) = o[1];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, MT * NC);
  if (ks > 1) {
    cluster_sync_all();
    if (warp >= 4) {
      // rank r finishes the rows r*128/ks ..: a thread takes four columns of every (128 / (D/4))-th row
      constexpr int CT = D / 4;
      const int et = threadIdx.x - 128, col = (et % CT) * 4;
      const int rows = 128 / ks;
      for (int rr = et / CT; rr < rows; rr += 128 / CT) {
        const int r = rank * rows + rr;
        const int p2 = r / HB, h2 = h0 + r % HB;
        if (r >= P * HB || i0 + p2 >= iend || h2 >= a.H) continue;
        const uint32_t addr = sbase + (uint32_t)(r * RS + col) * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < ks; ++k) {
          const float4 v = cluster_ld4(map_cta(addr, (uint32_t)k));
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (a.bias[z]) {
          const bf16* b = a.bias[z] + col;   // (of any alignment)
          s.x += __bfloat162float(b[0]); s.y += __bfloat162float(b[1]); s.z += __bfloat162float(b[2]); s.w += __bfloat162float(b[3]);
        }
        uint2 o = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
        *reinterpret_cast<uint2*>(a.y[z] + ((out0 + i0 + p2) * a.H + h2) * D + col) = o;
      }
    }
    cluster_sync_all();   // no CTA leaves while another still reads its partial tile
  }
}

template <int D, int MT, int NC>
int launch_tile(const Maps& m, const CompressFwdArgs& a, int P, int HB, int ks, long long gx, cudaStream_t s) {
  if (gx > 0x7fffffffLL) {
    set_error("compression: grid too large");
    return -33;
  }
  const int smem = kRing<MT, NC> * kStage<MT, NC> + 1024 + 256;
  auto kern = compress_fwd_tc_kernel<D, MT, NC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = next_config(dim3((unsigned)gx, (unsigned)ks, (unsigned)(a.ntensor * (D / NC))), dim3(kThreads), smem, s, at);
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1;
  at[1].val.clusterDim.y = (unsigned)ks;
  at[1].val.clusterDim.z = 1;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, kern, m, a, P, HB, ks);
  if (e != cudaSuccess) return (int)e;
  note_launches(1);
  return (int)cudaGetLastError();
}

template <int D>
int launch(const CompressFwdArgs& a, cudaStream_t s) {
  const int HB = a.H < 128 ? a.H : 128, nhg = (a.H + HB - 1) / HB, P0 = compress_tile_positions(a.H);
  // tile indices of a CTA tile of PP positions, and how many of them have work.  Ragged: of the nseq spare ones at most one per
  // position (a generation step completes few positions).
  auto tiles = [&](int PP) { return a.cu_in ? a.rows / PP + a.nseq : (long long)a.nseq * ((a.Tc + PP - 1) / PP); };
  auto busy = [&](int PP) { return (a.cu_in && a.rows < a.nseq ? a.rows / PP + a.rows : tiles(PP)) * nhg * a.ntensor; };
  // Split of the contraction: waves of CTAs times the stages of one, plus about six stages' worth of fixed cost (launch,
  // barrier set-up, epilogue, the cluster's reduction) per wave.
  int ks = 1;
  long long best = -1;
  for (int k = 1; k <= (a.split ? 8 : 1) && k <= a.l; k *= 2) {
    const long long cost = (busy(P0) * k + num_sms() - 1) / num_sms() * ((a.l + k - 1) / k + 6);
    if (best < 0 || cost < best) {
      best = cost;
      ks = k;
    }
  }
  // The tile.  Few rows: half of the columns per CTA while that still makes at most one CTA per SM (x is then read twice, W by
  // halves; 516 rows 14.9 us against 19.1, 1248 rows 15.6 / 19.5, 2040 rows 16.5 / 20.5, 4092 rows 19.8 / 22.8; with 8176 rows
  // it makes two waves, 38.4 / 30.3).  A little more than one CTA per SM: two row tiles in a CTA, one wave (9480 rows, 156 CTAs:
  // 42.9 against 49.2, 12488 rows, 198 CTAs: 52.0 / 53.4; at 256 the second wave is full enough, 60.5 / 56.7; 32 sequences whose 128
  // tiles fit one wave 40.1 / 31.2).  Of ragged sequences the host knows how many full tiles there are at least and expects half
  // a tile more of each.
  const long long full = a.cu_in ? a.rows / P0 * nhg * a.ntensor : busy(P0);
  const long long ctas = a.cu_in ? full + std::min<long long>(a.nseq, a.rows) * nhg * a.ntensor / 2 : full;
  const bool wide = ks == 1 && ctas > num_sms() && 20 * full >= 19LL * num_sms() && 3 * ctas <= 4LL * num_sms();
  const bool narrow = ks == 1 && D > 64 && 2 * busy(P0) <= num_sms();
  Maps m;
  const long long U = a.total_in / a.d, rem = a.total_in % a.d;
  const unsigned long long strides[4] = {(unsigned long long)D * 2, (unsigned long long)a.H * D * 2,
                                         (unsigned long long)a.d * a.H * D * 2, 128};
  const unsigned box[5] = {64, (unsigned)HB, 1, (unsigned)P0, 1};
  for (int t = 0; t < a.ntensor; ++t) {
    const unsigned long long d0[5] = {64, (unsigned long long)a.H, (unsigned long long)a.d, (unsigned long long)U, D / 64};
    const unsigned long long d1[5] = {64, (unsigned long long)a.H, (unsigned long long)(rem ? rem : a.d),
                                      (unsigned long long)(rem ? U + 1 : U), D / 64};
    int rc = make_tmap_generic(&m.x[t][0], a.x[t], 5, d0, strides, box);
    if (!rc) rc = make_tmap_generic(&m.x[t][1], a.x[t], 5, d1, strides, box);
    if (!rc) rc = make_tmap_rows2d(&m.w[t], a.w[t], D, (long long)a.l * D, 64);
    if (rc) return rc;
  }
  if (a.ntensor == 1) {
    m.x[1][0] = m.x[0][0];
    m.x[1][1] = m.x[0][1];
    m.w[1] = m.w[0];
  }
  if (wide) return launch_tile<D, 2, D>(m, a, P0, HB, ks, tiles(2 * P0) * nhg, s);
  if (narrow) return launch_tile<D, 1, 64>(m, a, P0, HB, ks, tiles(P0) * nhg, s);
  return launch_tile<D, 1, D>(m, a, P0, HB, ks, tiles(P0) * nhg, s);
}

}  // namespace

int compress_tile_positions(int H) { return H < 128 ? 128 / H : 1; }
int launch_compress_fwd_tc(const CompressFwdArgs& a, cudaStream_t s) {
  if ((a.cu_in ? a.rows : (long long)a.nseq * a.Tc) <= 0) return 0;
  if (a.D == 128) return launch<128>(a, s);
  if (a.D == 64) return launch<64>(a, s);
  set_error("head_dim %d not supported (64 or 128)", a.D);
  return -2;
}
int compress_tc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
