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
// Warps 0 and 1 stream the A and W tiles through an mbarrier ring (one TMA instruction each per stage: a warp's TMA
// instructions run one after another, ~850 cycles each, and three of them per 32 KB stage capped the kernel at 40 bytes
// per cycle), one thread of warp 2 issues tcgen05.mma into a [128 x D] fp32 accumulator in TMEM, warps 4-7 read it back
// with tcgen05.ld, add the bias and store bf16.
//
// A tile is a serial chain of l stages (32 at the default sizes, ~950 cycles of L2 traffic each), 16 us however few rows
// there are.  Where the caller allows it (`split`) the contraction is therefore split over a cluster of up to eight CTAs when
// that shortens the waves; the partial accumulators meet in distributed shared memory and are added in rank order.  The
// package does not allow it anywhere: a block selection turns last-bit differences of ck into other blocks, and with one
// order of summation (the same bits as a chain of mma.sync steps) a sequence selects the same blocks whatever batch it is
// in and however its cache was built.  What that costs: extending a cache by one position 8 us of 79 a generation step,
// the compression of eight packed sequences nothing that two runs do not differ by (176 and 181 us, 5 %).
#include "kernels.h"
#include "tc.cuh"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kThreads = 256;

template <int D>
constexpr int kRing = D == 128 ? 3 : 6;   // 64 KB (D = 128) or 24 KB stages

struct Maps {
  CUtensorMap x[2][2];   // [tensor][jj >= tok % d, jj < tok % d]
  CUtensorMap w[2];
};

__device__ __forceinline__ float4 cluster_ld4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
    compress_fwd_tc_kernel(const __grid_constant__ Maps maps, const CompressFwdArgs a, const int P, const int HB, const int ks) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  constexpr int NP = D / 64;                       // 64-channel panels
  constexpr uint32_t A_PANEL = 128 * 128;          // [128 rows][64 ch]
  constexpr uint32_t A_BYTES = NP * A_PANEL;
  constexpr uint32_t W_PANEL = D * 128;            // [D k][64 n]
  constexpr uint32_t W_BYTES = NP * W_PANEL;
  constexpr uint32_t STAGE = A_BYTES + W_BYTES;
  constexpr int RS = D + 4;                        // row stride of the partial tile in shared memory (floats)
  static_assert(128 * RS * 4 <= kRing<D> * STAGE, "the partial tile reuses the ring");
  constexpr int NR = kRing<D>;
  const uint32_t bar_base = sbase + NR * STAGE;
  auto full_bar = [&](int i) { return bar_base + 8u * i; };
  auto empty_bar = [&](int i) { return bar_base + 8u * (NR + i); };
  const uint32_t acc_bar = bar_base + 16u * NR;
  const uint32_t tmem_slot = acc_bar + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z, rank = blockIdx.y;
  const int nhg = (a.H + HB - 1) / HB;
  const int tile = blockIdx.x / nhg, h0 = (blockIdx.x % nhg) * HB;

  // ---- the tile's sequence, first position and limits -----------------------------------------------------------
  long long in0, out0;
  int i0, iend;
  if (!a.cu_in) {
    const int tps = (a.Tc + P - 1) / P;
    const int s = tile / tps;
    in0 = (long long)s * a.T;
    out0 = (long long)s * a.Tc;
    i0 = (tile % tps) * P;
    iend = a.Tc;
  } else {
    // sequence s owns the tile indices from cu_row[s] / P + s on (never fewer than it has tiles)
    int lo = 0, hi = a.nseq - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.cu_row[mid] / P + mid <= tile) lo = mid; else hi = mid - 1;
    }
    const int r0 = a.cu_row[lo], first = a.first ? a.first[lo] : 0;
    in0 = a.cu_in[lo];
    out0 = a.cu_out[lo];
    i0 = first + (tile - (r0 / P + lo)) * P;
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
  if (warp == 2) tmem_alloc(tmem_slot, D);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sgen + (tmem_slot - sbase));
  const int j_lo = a.l * rank / ks, j_hi = a.l * (rank + 1) / ks;   // this CTA's share of the contraction

  const int row = 32 * (warp & 3) + lane;
  const int pos = row / HB, h = h0 + row % HB;
  const bool live = row < P * HB && i0 + pos < iend && h < a.H;
  bool ok = true;
  if (warp < 2) {
    const int rem = (int)(a.total_in % a.d);
    for (int j = j_lo; j < j_hi; ++j) {
      const int stage = (j - j_lo) % NR;
      const uint32_t ph = ((j - j_lo) / NR) & 1;
      int good = 1;
      if (lane == 0) {
        good = mbar_wait(empty_bar(stage), ph ^ 1, DEV_ERR_EMPTY_WAIT) ? 1 : 0;
        if (good) mbar_expect_tx(full_bar(stage), warp == 0 ? (uint32_t)(P * HB) * 128 * NP : W_BYTES);
      }
      if (!__shfl_sync(0xffffffffu, good, 0)) break;
      const uint32_t a_s = sbase + stage * STAGE, w_s = a_s + A_BYTES;
      if (warp == 0) {
        const int jj = (int)((in0 + j) % a.d), u = (int)((in0 + j) / a.d) + i0;
        if (lane < NP) tma_load_5d(a_s + lane * A_PANEL, &maps.x[z][jj < rem ? 1 : 0], full_bar(stage), 0, h0, jj, u, lane);
      } else if (lane < NP) {
        tma_load_2d(w_s + lane * W_PANEL, &maps.w[z], full_bar(stage), lane * 64, j * D);
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, D, 0, 1);
      for (int j = j_lo; j < j_hi; ++j) {
        const int stage = (j - j_lo) % NR;
        const uint32_t ph = ((j - j_lo) / NR) & 1;
        if (!mbar_wait(full_bar(stage), ph, DEV_ERR_FULL_WAIT)) break;
        tc_fence_after();
        const uint32_t a_s = sbase + stage * STAGE, w_s = a_s + A_BYTES;
        const uint64_t ad = umma_smem_desc(a_s, 0, 1024), wd = umma_smem_desc(w_s, W_PANEL, 1024);
#pragma unroll
        for (int s = 0; s < D / 16; ++s)
          umma_ss(tmem, umma_desc_advance(ad, (s >> 2) * A_PANEL + (s & 3) * 32), umma_desc_advance(wd, s * 2048), idesc,
                  (j > j_lo || s) ? 1u : 0u);
        umma_commit(empty_bar(stage));
      }
      umma_commit(acc_bar);
    }
  } else if (warp >= 4) {
    ok = mbar_wait(acc_bar, 0, DEV_ERR_FULL_WAIT);
    tc_fence_after();
    bf16* dst = a.y[z] + ((out0 + i0 + pos) * a.H + h) * D;
    float* part = reinterpret_cast<float*>(sgen) + row * RS;
#pragma unroll
    for (int c = 0; c < D / 16; ++c) {
      float v[16];
      tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c * 16, v);
      tmem_ld_wait();
      if (ks > 1) {   // the ring is idle: every MMA that read it has completed
#pragma unroll
        for (int e = 0; e < 4; ++e)
          *reinterpret_cast<float4*>(part + c * 16 + 4 * e) = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
      } else if (ok && live) {
        uint4 o[2];
        __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float x0 = v[2 * e], x1 = v[2 * e + 1];
          if (a.bias[z]) {
            x0 += __bfloat162float(a.bias[z][c * 16 + 2 * e]);
            x1 += __bfloat162float(a.bias[z][c * 16 + 2 * e + 1]);
          }
          ho[e] = __floats2bfloat162_rn(x0, x1);
        }
        *reinterpret_cast<uint4*>(dst + c * 16) = o[0];
        *reinterpret_cast<uint4*>(dst + c * 16 + 8) = o[1];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, D);
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

template <int D>
int launch(const CompressFwdArgs& a, cudaStream_t s) {
  Maps m;
  const int HB = a.H < 128 ? a.H : 128, P = compress_tile_positions(a.H);
  const long long U = a.total_in / a.d, rem = a.total_in % a.d;
  const unsigned long long strides[4] = {(unsigned long long)D * 2, (unsigned long long)a.H * D * 2,
                                         (unsigned long long)a.d * a.H * D * 2, 128};
  const unsigned box[5] = {64, (unsigned)HB, 1, (unsigned)P, 1};
  for (int t = 0; t < a.ntensor; ++t) {
    const unsigned long long d0[5] = {64, (unsigned long long)a.H, (unsigned long long)a.d, (unsigned long long)U, D / 64};
    const unsigned long long d1[5] = {64, (unsigned long long)a.H, (unsigned long long)(rem ? rem : a.d),
                                      (unsigned long long)(rem ? U + 1 : U), D / 64};
    int rc = make_tmap_generic(&m.x[t][0], a.x[t], 5, d0, strides, box);
    if (!rc) rc = make_tmap_generic(&m.x[t][1], a.x[t], 5, d1, strides, box);
    if (!rc) rc = make_tmap_rows2d(&m.w[t], a.w[t], D, (long long)a.l * D, D);
    if (rc) return rc;
  }
  if (a.ntensor == 1) {
    m.x[1][0] = m.x[0][0];
    m.x[1][1] = m.x[0][1];
    m.w[1] = m.w[0];
  }
  const long long tiles = a.cu_in ? a.rows / P + a.nseq : (long long)a.nseq * ((a.Tc + P - 1) / P);
  const long long gx = tiles * ((a.H + HB - 1) / HB);
  if (gx > 0x7fffffffLL) {
    set_error("compression: grid too large");
    return -33;
  }
  // Split of the contraction: waves of CTAs times the stages of one, plus about six stages' worth of fixed cost (launch,
  // barrier set-up, epilogue, the cluster's reduction) per wave.
  // Ragged: of the nseq spare tile indices at most one per position has work (a generation step completes few positions).
  const long long used = a.cu_in && a.rows < a.nseq ? a.rows / P + a.rows : tiles;
  const long long busy = used * ((a.H + HB - 1) / HB) * a.ntensor;
  int ks = 1;
  long long best = -1;
  for (int k = 1; k <= (a.split ? 8 : 1) && k <= a.l; k *= 2) {
    const long long cost = (busy * k + num_sms() - 1) / num_sms() * ((a.l + k - 1) / k + 6);
    if (best < 0 || cost < best) {
      best = cost;
      ks = k;
    }
  }
  const int smem = kRing<D> * 2 * (128 + D) * (D / 64) * 64 + 1024 + 256;
  auto kern = compress_fwd_tc_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = next_config(dim3((unsigned)gx, (unsigned)ks, (unsigned)a.ntensor), dim3(kThreads), smem, s, at);
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
