// Key/value-major half of the backward of the selected branch (dK, dV), for head_dim 64 or selection blocks other than 64 keys.
//
// Reference behaviour: parallel_nsa_bwd_kernel_dkv (nsa/selection_attn.py:151-253) walks, for every 64-key block, ALL later
// query tokens and tests a dense boolean block mask built by parallel_nsa_kernel_mask (:256-273).  Here a per-block reverse
// index is walked instead (CSR lists of the tokens that selected the block, ascending; see build_rev in misc.cu), so the work is
// proportional to the number of (token, block) pairs and there is no global atomic: one CTA owns a key block, keeps dK and dV
// of its keys in registers over the whole list and stores them once.
//
// B200 design.  The key block [rows x D] of K and V is TMA-loaded once.  A producer warp then streams, per (token, 16-head
// group), the [16 x D] Q tile and dO tile (2-D TMA boxes, 128-byte swizzle) plus the 16 lse / delta / gate values (bulk copies)
// through an mbarrier ring.  Four consumer warps own 16 keys each; with keys on the mma M axis and the 16 heads on N:
//     S^T = K.Q^T      P^T = exp(S^T*scale - lse)      dV += (g.P^T).dO
//     dP^T = V.dO^T    dS^T = P^T.(g.dP^T - delta)     dK += dS^T.Q   (times scale at the end)
// When there are fewer blocks than SMs a block's list is cut into shares (a share walks its tokens one after the other at
// ~0.9 us each: 1.0 ms for the first block of a 1024-token sequence with one KV head in one piece, 0.07 ms in 16); they are fp32
// slabs, added in order by a second kernel.
#include "kernels.h"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kConsumerWarps = 4;
constexpr int kThreads = (kConsumerWarps + 1) * 32;

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
    kv_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                  const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const KvArgs a, const int nst) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int rows = a.BS;                                  // keys per CTA
  const uint32_t kv_panel = rows * 128;
  const uint32_t kv_tile = kv_panel * (D / 64);
  constexpr uint32_t q_panel = 16 * 128;
  constexpr uint32_t q_tile = q_panel * (D / 64);
  constexpr uint32_t stage_bytes = 2 * q_tile + 1024;
  const uint32_t k_s = sbase, v_s = sbase + kv_tile;
  const uint32_t ring = sbase + 2 * kv_tile;              // kv_tile is a multiple of 1024
  const uint32_t bar_base = ring + nst * stage_bytes;
  auto full_bar = [&](int i) { return bar_base + 8u * i; };
  auto empty_bar = [&](int i) { return bar_base + 8u * (nst + i); };
  const uint32_t kv_bar = bar_base + 16u * nst;

  if (threadIdx.x == 0) {
    for (int i = 0; i < nst; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(empty_bar(i), kConsumerWarps);
    }
    mbar_init(kv_bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  // ---- decode the work item -----------------------------------------------------------------------
  const int G16 = (a.Hq / a.Hk) / 16;
  const int BH = a.B * a.Hk, NB = (a.T + a.BS - 1) / a.BS;
  const int seg = blockIdx.x % a.nshare, item = blockIdx.x / a.nshare;
  const int blk = item / BH, bh = item % BH, b = bh / a.Hk, hk = bh % a.Hk;
  const int* rp = a.rev_ptr + (long long)bh * (NB + 1);
  const int* list = a.rev_tok + (long long)bh * a.rev_cap;
  int lo = rp[blk], n = rp[blk + 1] - lo;
  if (a.nshare > 1) {   // this CTA's share of the list
    const int a0 = (int)((long long)n * seg / a.nshare), a1 = (int)((long long)n * (seg + 1) / a.nshare);
    lo += a0;
    n = a1 - a0;
  }
  const int key0 = blk * rows;

  if (warp == kConsumerWarps) {
    // ------------------------------- producer ------------------------------------------------
    if (elect_one()) {
      mbar_expect_tx(kv_bar, 2 * kv_tile);
#pragma unroll
      for (int p = 0; p < D / 64; ++p) {
        tma_load_4d(k_s + p * kv_panel, &tmK, kv_bar, p * 64, hk, key0, b);
        tma_load_4d(v_s + p * kv_panel, &tmV, kv_bar, p * 64, hk, key0, b);
      }
    }
    uint32_t it = 0;
    for (int sub = 0; sub < G16; ++sub) {
      const int hg = hk * G16 + sub;
      const uint32_t tx = 2 * q_tile + 128 + (a.gate ? 32 : 0);
      for (int i0 = 0; i0 < n; i0 += 32) {
        const int tok = (i0 + lane < n) ? list[lo + i0 + lane] : 0;
        const int nn = min(32, n - i0);
        for (int j = 0; j < nn; ++j) {
          const int t = __shfl_sync(0xffffffffu, tok, j);
          bool okw = true;
          if (elect_one()) {
            const int stage = it % nst;
            const uint32_t ph = (it / nst) & 1;
            okw = mbar_wait(empty_bar(stage), ph ^ 1, DEV_ERR_EMPTY_WAIT);
            if (okw) {
              const long long qrow = ((long long)b * a.T + t) * a.Hq + hg * 16;
              const uint32_t dst = ring + stage * stage_bytes;
              mbar_expect_tx(full_bar(stage), tx);
#pragma unroll
              for (int p = 0; p < D / 64; ++p) {
                tma_load_2d(dst + p * q_panel, &tmQ, full_bar(stage), p * 64, (int)qrow);
                tma_load_2d(dst + q_tile + p * q_panel, &tmDO, full_bar(stage), p * 64, (int)qrow);
              }
              bulk_load(dst + 2 * q_tile, a.lse + qrow, 64, full_bar(stage));
              bulk_load(dst + 2 * q_tile + 64, a.delta + qrow, 64, full_bar(stage));
              if (a.gate) bulk_load(dst + 2 * q_tile + 128, a.gate + qrow, 32, full_bar(stage));
            }
          }
          if (!__all_sync(0xffffffffu, okw)) return;
          ++it;
        }
      }
    }
    return;
  }

  // --------------------------------- consumers -------------------------------------------------
  const int g = lane >> 2, tq = lane & 3;
  const bool active = warp * 16 < rows;
  const float sl2 = a.scale * kLog2e;
  float dk[D / 8][4], dv[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    dk[i][0] = dk[i][1] = dk[i][2] = dk[i][3] = 0.f;
    dv[i][0] = dv[i][1] = dv[i][2] = dv[i][3] = 0.f;
  }
  if (!mbar_wait(kv_bar, 0, DEV_ERR_FULL_WAIT)) return;
  const int kp0 = key0 + warp * 16 + g;  // key position of accumulator rows c<2; +8 for c>=2

  uint32_t it = 0;
  for (int sub = 0; sub < G16; ++sub) {
    const bool has_gate = a.gate != nullptr;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int tok = (i0 + lane < n) ? list[lo + i0 + lane] : 0;
      const int nn = min(32, n - i0);
      for (int j = 0; j < nn; ++j) {
        const int t = __shfl_sync(0xffffffffu, tok, j);
        const int stage = it % nst;
        const uint32_t ph = (it / nst) & 1;
        if (!mbar_wait(full_bar(stage), ph, DEV_ERR_FULL_WAIT)) return;
        if (active) {
          const uint32_t qs = ring + stage * stage_bytes;
          const uint32_t dos = qs + q_tile;
          const uint8_t* aux = sgen + (qs - sbase) + 2 * q_tile;
          const float* lse_s = reinterpret_cast<const float*>(aux);
          const float* del_s = reinterpret_cast<const float*>(aux + 64);
          const bf16* gate_s = reinterpret_cast<const bf16*>(aux + 128);
          float st[2][4], dpt[2][4];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            st[i][0] = st[i][1] = st[i][2] = st[i][3] = 0.f;
            dpt[i][0] = dpt[i][1] = dpt[i][2] = dpt[i][3] = 0.f;
          }
          {
            uint32_t af[D / 16][4];
            load_a_frags<D>(af, k_s, kv_panel, warp * 16, lane);
            mma_a_bt<D, 16>(st, af, qs, q_panel, 0, lane);
          }
          {
            uint32_t af[D / 16][4];
            load_a_frags<D>(af, v_s, kv_panel, warp * 16, lane);
            mma_a_bt<D, 16>(dpt, af, dos, q_panel, 0, lane);
          }
          float pg[2][4];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int h = 8 * nt + 2 * tq + (c & 1);
              const int kp = kp0 + (c >> 1) * 8;
              const bool ok = kp <= t;
              const float l2v = lse_s[h] * kLog2e;
              const float gv = has_gate ? __bfloat162float(gate_s[h]) : 1.f;
              const float p = (ok && l2v > -INFINITY) ? ex2(st[nt][c] * sl2 - l2v) : 0.f;
              pg[nt][c] = p * gv;
              st[nt][c] = p * (gv * dpt[nt][c] - del_s[h]);
            }
          uint32_t f[1][4];
          acc_to_a_frags<2>(f, pg);
          mma_a_b<D, 16>(dv, f, dos, q_panel, 0, lane);
          acc_to_a_frags<2>(f, st);
          mma_a_b<D, 16>(dk, f, qs, q_panel, 0, lane);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(stage));
        ++it;
      }
    }
  }

  // ---- store ----------------------------------------------------------------------------------------
  if (!active) return;
#pragma unroll
  for (int hrow = 0; hrow < 2; ++hrow) {
    const int kp = kp0 + hrow * 8;
    if (kp >= a.T) continue;
    const long long off = (((long long)b * a.T + kp) * a.Hk + hk) * D + 2 * tq;
    const long long N = (long long)a.B * a.T * a.Hk * D;
    if (a.nshare == 1) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        float2 xk = make_float2(dk[i][2 * hrow] * a.scale, dk[i][2 * hrow + 1] * a.scale);
        float2 xv = make_float2(dv[i][2 * hrow], dv[i][2 * hrow + 1]);
        for (int w = 0; w < a.nadd; ++w) {
          const float2 yk = *reinterpret_cast<const float2*>(a.part + w * N + off + i * 8);
          const float2 yv = *reinterpret_cast<const float2*>(a.part + (a.slabs + w) * N + off + i * 8);
          xk.x += yk.x; xk.y += yk.y; xv.x += yv.x; xv.y += yv.y;
        }
        *reinterpret_cast<__nv_bfloat162*>(a.dk + off + i * 8) = __floats2bfloat162_rn(xk.x, xk.y);
        *reinterpret_cast<__nv_bfloat162*>(a.dv + off + i * 8) = __floats2bfloat162_rn(xv.x, xv.y);
      }
    } else {
      float* pk = a.part + (long long)seg * N + off;
      float* pv = a.part + ((long long)a.slabs + seg) * N + off;
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        *reinterpret_cast<float2*>(pk + i * 8) = make_float2(dk[i][2 * hrow] * a.scale, dk[i][2 * hrow + 1] * a.scale);
        *reinterpret_cast<float2*>(pv + i * 8) = make_float2(dv[i][2 * hrow], dv[i][2 * hrow + 1]);
      }
    }
  }
}

template <int D>
int launch(const KvArgs& a, cudaStream_t s) {
  CUtensorMap tmQ, tmDO, tmK, tmV;
  const long long qrows = (long long)a.B * a.T * a.Hq;
  if (qrows > 0x7fffffffLL) {
    set_error("B*T*Hq exceeds the 2^31 rows a TMA coordinate can address");
    return -32;
  }
  // the bulk copies of 16 rows' lse, delta and gates
  if ((((uintptr_t)a.lse | (uintptr_t)a.delta | (uintptr_t)a.gate) & 15) != 0) {
    set_error("kv backward: lse, delta and gates must be 16-byte aligned");
    return -5;
  }
  int rc = make_tmap_rows2d(&tmQ, a.q, D, qrows, 16);
  if (!rc) rc = make_tmap_rows2d(&tmDO, a.dout, D, qrows, 16);
  if (!rc) rc = make_tmap_rows4d(&tmK, a.k, D, a.Hk, a.T, a.B, a.BS);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hk, a.T, a.B, a.BS);
  if (rc) return rc;
  int dev = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const int stage_bytes = 2 * 16 * D * 2 + 1024;
  const int fixed = 2 * a.BS * D * 2 + (2 * 16 + 1) * 8 + 1024;
  int nst = (max_smem / 2 - fixed) / stage_bytes;  // leave room for two CTAs per SM
  if (nst > 8) nst = 8;
  if (nst < 2) nst = 2;
  const int smem = fixed + nst * stage_bytes;
  auto kern = kv_bwd_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const long long grid = (long long)a.B * a.Hk * ((a.T + a.BS - 1) / a.BS) * a.nshare;
  if (grid <= 0) return 0;
  if (grid > 0x7fffffffLL) {
    set_error("kv backward: grid too large");
    return -33;
  }
  launch_next(kern, (unsigned)grid, kThreads, smem, s, tmQ, tmDO, tmK, tmV, a, nst);
  note_launches(1);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_kv_bwd(const KvArgs& a, int D, cudaStream_t s) {
  if (D == 128) return launch<128>(a, s);
  if (D == 64) return launch<64>(a, s);
  set_error("head_dim %d not supported (64 or 128)", D);
  return -2;
}
int kv_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
