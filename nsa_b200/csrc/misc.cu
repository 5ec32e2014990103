// Small memory-bound helpers: row dot products for the backward (delta and gate gradients), the gated
// combine of the three branches, the reverse index of the block selection, and the fixed-order reduction
// of the compressed branch's dCK/dCV partials.
#include "kernels.h"
#include "tmap.h"

namespace nsa {

int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

namespace {

// ---- gated combine ------------------------------------------------------------------------------------
// o = g0*a0 + g1*a1 + g2*a2  (nsa/selection_attn.py:808-811 and nsa/nsa.py:133, as one pass)
__global__ void combine_kernel(const bf16* __restrict__ a0, const bf16* __restrict__ g0, const bf16* __restrict__ a1,
                               const bf16* __restrict__ g1, const bf16* __restrict__ a2, const bf16* __restrict__ g2,
                               bf16* __restrict__ o, long long n8, int D8) {
  after_previous();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const long long row = i / D8;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  auto add = [&](const bf16* a, const bf16* gp) {
    if (!a) return;
    const float gv = gp ? __bfloat162float(gp[row]) : 1.f;
    const uint4 v = *reinterpret_cast<const uint4*>(a + i * 8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(h[k]);
      acc[2 * k] += gv * f.x;
      acc[2 * k + 1] += gv * f.y;
    }
  };
  add(a0, g0);
  add(a1, g1);
  add(a2, g2);
  uint4 out;
  __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
  for (int k = 0; k < 4; ++k) ho[k] = __floats2bfloat162_rn(acc[2 * k], acc[2 * k + 1]);
  *reinterpret_cast<uint4*>(o + i * 8) = out;
}

// ---- reverse index of the selection -----------------------------------------------------------------
// Replaces the dense boolean block mask of parallel_nsa_kernel_mask (nsa/selection_attn.py:256-273).
// A stable counting sort by block id in four launches; the order inside every list is ascending in t and
// independent of scheduling, so the backward is bit-reproducible.  All are latency: every serial chain (one warp
// walking the 64 tokens of a chunk, one thread walking the chunks of a block id) is cut into eight or 32 parts whose
// counts meet in shared memory.  Measured: T = 2080, 4 (batch, head) pairs 59 -> 17 us; T = 65536 650 -> 120 us.
constexpr int kRevWarps = 8;

// grid (NB chunks, B*H): histogram of the block ids selected by the BS tokens of one chunk
__global__ void rev_hist_kernel(const RevArgs a) {
  after_previous();
  extern __shared__ int sh[];
  const int chunk = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  for (int i = threadIdx.x; i < a.NB; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int n = a.BS * a.S;
#pragma unroll 4
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int tl = chunk * a.BS + e / a.S, s = e % a.S;
    if (tl >= a.Tq) continue;
    const int blk = rev_block(a, ((long long)b * a.Tq + tl) * a.H + h, s, a.q0 + tl);
    if (blk >= 0) atomicAdd(&sh[blk], 1);
  }
  __syncthreads();
  int* out = a.hist + ((long long)bh * gridDim.x + chunk) * a.NB;
  for (int i = threadIdx.x; i < a.NB; i += blockDim.x) out[i] = sh[i];
}

// grid (ceil(NB / 32), B*H), 1024 threads: exclusive prefix over the chunks of 32 block ids (in place), one lane per id,
// one warp per thirty-second of the chunks; the totals go to rev_ptr[blk] (the fill kernel turns them into offsets)
__global__ void __launch_bounds__(1024) rev_scan_kernel(const RevArgs a, const int nchunk) {
  after_previous();
  __shared__ int part[32][33];
  const int bh = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blk = blockIdx.x * 32 + lane;
  int* hist = a.hist + (long long)bh * nchunk * a.NB + blk;
  const int lo = (int)((long long)nchunk * warp / 32), hi = (int)((long long)nchunk * (warp + 1) / 32);
  int sum = 0;
  if (blk < a.NB) {
#pragma unroll 8
    for (int c = lo; c < hi; ++c) sum += hist[(long long)c * a.NB];
  }
  part[warp][lane] = sum;
  __syncthreads();
  int run = 0;
  for (int w = 0; w < warp; ++w) run += part[w][lane];
  if (blk >= a.NB) return;
  if (warp == 31) a.rev_ptr[(long long)bh * (a.NB + 1) + blk] = run + sum;
#pragma unroll 8
  for (int c = lo; c < hi; ++c) {
    const int v = hist[(long long)c * a.NB];
    hist[(long long)c * a.NB] = run;
    run += v;
  }
}

// grid (B*H), 1024 threads: totals per block id -> exclusive CSR offsets (in place)
__global__ void __launch_bounds__(1024) rev_offset_kernel(const RevArgs a) {
  after_previous();
  __shared__ int ws[32];
  int* rp = a.rev_ptr + (long long)blockIdx.x * (a.NB + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry = 0;
  for (int i0 = 0; i0 <= a.NB; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const int v = i < a.NB ? rp[i] : 0;
    int x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    int before = carry, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += ws[w];
      all += ws[w];
    }
    if (i <= a.NB) rp[i] = before + x - v;
    carry += all;
    __syncthreads();
  }
}

// grid (NB chunks, B*H), eight warps: write the tokens of the chunk, in order, behind each block's cursor.  A warp owns
// an eighth of the chunk's tokens; the cursors of a warp start behind the counts of the warps before it.
__global__ void __launch_bounds__(kRevWarps * 32) rev_fill_kernel(const RevArgs a) {
  after_previous();
  extern __shared__ int cur[];   // [warps][NB]
  const int nw = blockDim.x >> 5;
  const int chunk = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* rp = a.rev_ptr + (long long)bh * (a.NB + 1);
  const int* pre = a.hist + ((long long)bh * gridDim.x + chunk) * a.NB;
  for (int i = threadIdx.x; i < nw * a.NB; i += blockDim.x) cur[i] = 0;
  __syncthreads();
  int* mine = cur + warp * a.NB;
  const int per = (a.BS + nw - 1) / nw;
  const int t_lo = chunk * a.BS + warp * per, t_hi = min(min(t_lo + per, (chunk + 1) * a.BS), a.Tq);
  for (int e = lane; e < (t_hi - t_lo) * a.S; e += 32) {
    const int tl = t_lo + e / a.S;
    const int blk = rev_block(a, ((long long)b * a.Tq + tl) * a.H + h, e % a.S, a.q0 + tl);
    if (blk >= 0) atomicAdd(&mine[blk], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < a.NB; i += blockDim.x) {
    int run = rp[i] + pre[i];
    for (int w = 0; w < nw; ++w) {
      const int v = cur[w * a.NB + i];
      cur[w * a.NB + i] = run;
      run += v;
    }
  }
  __syncthreads();
  int* out = a.rev_tok + (long long)bh * a.cap;
  for (int tl = t_lo; tl < t_hi; ++tl) {
    const int t = a.q0 + tl;   // lists hold sequence positions
    const long long row = ((long long)b * a.Tq + tl) * a.H + h;
    for (int s0 = 0; s0 < a.S; s0 += 32) {
      const int s = s0 + lane;
      const int blk = (s < a.S) ? rev_block(a, row, s, t) : -1;
      const int key = blk >= 0 ? blk : -1 - lane;  // invalid lanes never match each other
      const unsigned same = __match_any_sync(0xffffffffu, key);
      if (blk >= 0) {
        const int rank = __popc(same & ((1u << lane) - 1));
        const int pos = mine[blk] + rank;
        if (pos < a.cap) {
          out[pos] = t;
          if (a.inv) a.inv[row * a.S + s] = pos;
        }
      } else if (a.inv && s < a.S) {
        a.inv[row * a.S + s] = -1;
      }
      __syncwarp();
      if (blk >= 0 && (lane == 31 || (same >> (lane + 1)) == 0)) mine[blk] += __popc(same);  // highest lane of the group
      __syncwarp();
    }
  }
}

// dk, dv = the sum of a key block's shares, in order
__global__ void __launch_bounds__(256) reduce_shares_kernel(const float* __restrict__ part, bf16* __restrict__ dk, bf16* __restrict__ dv,
                                                            int nshare, long long n) {
  after_previous();
  const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= n) return;
  const float* p = part + (blockIdx.y ? nshare * n : 0) + i;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < nshare; ++k) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p + k * n));
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  *reinterpret_cast<uint2*>((blockIdx.y ? dv : dk) + i) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
}

}  // namespace

int launch_reduce_shares(const float* part, bf16* dk, bf16* dv, int nshare, long long n, cudaStream_t s) {
  if (n <= 0) return 0;
  launch_next(reduce_shares_kernel, dim3((unsigned)((n / 4 + 255) / 256), 2), 256, 0, s, part, dk, dv, nshare, n);
  note_launches(1);
  return (int)cudaGetLastError();
}

int launch_rowdot(const bf16* o, const bf16* dout, const bf16* gate, float* delta, bf16* dgate, long long rows, int D,
                  cudaStream_t s) {
  const bf16* o3[3] = {o, nullptr, nullptr};
  const bf16* g3[3] = {gate, nullptr, nullptr};
  float* d3[3] = {delta, nullptr, nullptr};
  bf16* dg3[3] = {dgate, nullptr, nullptr};
  return launch_rowdot3(o3, dout, g3, d3, dg3, rows, D, s);
}

int launch_combine(const bf16* a0, const bf16* g0, const bf16* a1, const bf16* g1, const bf16* a2, const bf16* g2,
                   bf16* o, long long rows, int D, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (D % 8) {
    set_error("head_dim must be a multiple of 8");
    return -2;
  }
  const long long n8 = rows * (D / 8);
  launch_next(combine_kernel, (unsigned)((n8 + 255) / 256), 256, 0, s, a0, g0, a1, g1, a2, g2, o, n8, D / 8);
  note_launches(1);
  return (int)cudaGetLastError();
}

// Four warps per (batch, token, 16-head group), each four heads of the [16 x D] bf16 tile: the token's visits are added in slot
// order.  A load instruction of the warp covers 512 contiguous bytes; the list positions of all slots are fetched first so
// that the tiles of several slots are in flight at once (four heads instead of eight per warp: half the registers, twice the
// warps).  The gate projection's share of dq (sum_g dg_g W_g) can be added on the way: dq is in registers here, a pass of its
// own reads and writes it once more.
template <int D>
__global__ void __launch_bounds__(256) sel_dq_reduce_kernel(const RevArgs a, const bf16* __restrict__ part, bf16* __restrict__ dq,
                                                            const GateAdd gate, const int G16, const float scale, const int accumulate) {
  after_previous();
  constexpr int kHeads = 4, kWarps = 16 / kHeads;
  const long long w4 = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const long long total = (long long)a.B * a.Tq * a.H * G16;
  const long long w = w4 / kWarps;
  if (w >= total) return;
  const int hb = (int)(w4 % kWarps);                   // which heads of the tile
  const int lane = threadIdx.x & 31;
  const int sub = (int)(w % G16);
  const long long row = w / G16;                       // (b, tl, h) row of idx / counts
  const int h = (int)(row % a.H);
  const long long bt = row / a.H;
  const int tl = (int)(bt % a.Tq), b = (int)(bt / a.Tq);
  constexpr int NV = kHeads * D / 8 / 32;              // 16-byte vectors per lane: 2 at D = 128
  const long long bh = (long long)b * a.H + h;
  // lane s holds the list position of slot s (-1: the slot does not count)
  const int mypos = lane < a.S ? a.inv[row * a.S + lane] : -1;
  const int Hq = a.H * G16 * 16;
  const long long row0 = bt * Hq + (long long)(h * G16 + sub) * 16 + hb * kHeads;
  // the partial tiles keep the staging layout of the kernel that wrote them: within a 128-byte half row the 16-byte
  // chunk c sits at position c ^ (head & 7).  All tiles share it, so the sum is formed in place and undone at the end:
  // vector u = 32 i + lane of this part of the tile is its row u / 16, position u % 8.
  uint4* dst = reinterpret_cast<uint4*>(dq + row0 * D);
  int ud[NV];
  uint4 prev[NV];
  bf16 dg[NV][3];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int u = 32 * i + lane, r = u >> 4;
    ud[i] = (u & ~7) | ((u & 7) ^ ((hb * kHeads + r) & 7));
    prev[i] = make_uint4(0u, 0u, 0u, 0u);
    if (accumulate) prev[i] = __ldcs(dst + ud[i]);
#pragma unroll
    for (int g = 0; g < 3; ++g)
      if (gate.w) dg[i][g] = gate.dg[g][row0 + r];
  }
  unsigned live = __ballot_sync(0xffffffffu, mypos >= 0);
  const uint4* base = reinterpret_cast<const uint4*>(part) + hb * (kHeads * D / 8) + lane;
  auto tile = [&](int s) {
    const long long pos = __shfl_sync(0xffffffffu, mypos, s);
    return base + ((bh * a.cap + pos) * G16 + sub) * (16 * D / 8);
  };
  float acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[i][k] = 0.f;
  auto add = [&](const uint4 (&v)[NV]) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(hv[k]);
        acc[i][2 * k] += f.x;
        acc[i][2 * k + 1] += f.y;
      }
    }
  };
  while (live) {
    const int s0 = __ffs(live) - 1;
    live &= live - 1;
    const int s1 = live ? __ffs(live) - 1 : -1;
    if (s1 >= 0) live &= live - 1;
    const uint4* p0 = tile(s0);
    const uint4* p1 = tile(s1 >= 0 ? s1 : s0);
    uint4 v0[NV], v1[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v0[i] = __ldcs(p0 + 32 * i);
    if (s1 >= 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) v1[i] = __ldcs(p1 + 32 * i);
    }
    add(v0);
    if (s1 >= 0) add(v1);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[i][k] *= scale;
    auto add8 = [&](const uint4& v, float g) {
      const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(hv[k]);
        acc[i][2 * k] = fmaf(g, f.x, acc[i][2 * k]);
        acc[i][2 * k + 1] = fmaf(g, f.y, acc[i][2 * k + 1]);
      }
    };
    add8(prev[i], 1.f);
    if (gate.w) {
#pragma unroll
      for (int g = 0; g < 3; ++g)
        add8(__ldg(reinterpret_cast<const uint4*>(gate.w + g * D) + (ud[i] & 15)), __bfloat162float(dg[i][g]));
    }
    uint4 o;
    __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) ho[k] = __floats2bfloat162_rn(acc[i][2 * k], acc[i][2 * k + 1]);
    dst[ud[i]] = o;
  }
}

int launch_sel_dq_reduce(const RevArgs& a, const bf16* part, bf16* dq, int Hq, int D, const GateAdd& gate, float scale, int accumulate,
                         cudaStream_t s) {
  if (D != 128) {
    set_error("selected dQ reduction: head_dim 128 only");
    return -2;
  }
  const int G16 = Hq / a.H / 16;
  const long long total = (long long)a.B * a.Tq * a.H * G16;
  if (total <= 0) return 0;
  if (a.S > 32) {
    set_error("selected dQ reduction: at most 32 selected blocks per token");
    return -2;
  }
  launch_next(sel_dq_reduce_kernel<128>, (unsigned)((4 * total + 7) / 8), 256, 0, s, a, part, dq, gate, G16, scale, accumulate);
  note_launches(1);
  return (int)cudaGetLastError();
}

int launch_build_rev(const RevArgs& a, cudaStream_t s) {
  if (a.B <= 0 || a.T <= 0) return 0;
  const size_t sm = (size_t)a.NB * 4;
  if (sm > 200 * 1024) {
    set_error("reverse index: too many selection blocks (%d)", a.NB);
    return -34;
  }
  // a private set of cursors per warp: eight warps up to 6400 blocks, fewer beyond
  const int nw = (int)(200 * 1024 / sm < kRevWarps ? 200 * 1024 / sm : kRevWarps);
  const int nchunk = (a.Tq + a.BS - 1) / a.BS;   // chunks of BS local tokens
  const dim3 grid(nchunk, a.B * a.H);
  if (sm > 48 * 1024) cudaFuncSetAttribute(rev_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (nw * sm > 48 * 1024)
    cudaFuncSetAttribute(rev_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(nw * sm));
  launch_next(rev_hist_kernel, grid, 256, sm, s, a);
  launch_next(rev_scan_kernel, dim3((a.NB + 31) / 32, a.B * a.H), 1024, 0, s, a, nchunk);
  launch_next(rev_offset_kernel, a.B * a.H, 1024, 0, s, a);
  launch_next(rev_fill_kernel, grid, nw * 32, nw * sm, s, a);
  note_launches(4);
  return (int)cudaGetLastError();
}

int misc_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
