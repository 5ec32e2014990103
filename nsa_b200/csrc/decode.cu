// Batched decode step: the whole NSA forward (nsa/nsa.py:94-135) for ONE new query token per sequence, every sequence
// of a packed, ragged K/V cache in a single launch.  The reference has no decode entry point (its module assumes
// len(q) == len(k), nsa/nsa.py:97); the arithmetic is that of its forward evaluated for the row t = L-1:
// compressed attention over the compressed cache with the mask t >= 16 j + 32 (nsa/triton_attention.py:87-181), the
// block scores softmax(q.ck) summed over the 16 heads of the group, 5/4 average-pooled and top-n'd
// (nsa/torch_attention.py:51-62,121-125), attention over the selected 64-key blocks and over the last `window` keys
// (nsa/selection_attn.py:401-517), and the gated sum (nsa/nsa.py:133).
//
// The step is HBM-bound: a sequence contributes its compressed cache (1/16 of its K/V), 16 selected blocks and the
// window, each read once.  One CTA works on one (sequence, kv head): the 16 query heads of the group are the M = 16
// rows of mma.sync.m16n8k16.  Where there are fewer items than SMs, a cluster of 2, 4 or 8 CTAs shares one: the tile pairs of
// every phase behind the statistics are dealt out to its CTAs, which exchange the scores through each other's shared
// memory and then select the blocks each for itself (one CTA alone draws at most 1/148 of the bandwidth: 4 items of 4096 keys
// took 25 us).  Where there are more, a CTA takes one after another, and two CTAs of half the size share an SM unless lengths or
// their evenness speak against it (the rule at decode_spread).  The sums of a phase are six chains of tile pairs: a warp of six has
// one of them, a warp of three two, one after the other, and their partials are merged in one order, so that either form gives
// the same bits.  The statistics (pass 1) are the same six chains in a cluster too, where every CTA makes them for itself.  In another
// order near ties of two blocks' scores come out otherwise, and a sequence's blocks would depend on how many others it is decoded with:
// with pass 1 dealt out like the rest up to one in 16 items chose others (1 x 32768 keys 28.7 us so, 34.8 now; 4 x 16384
// 30.7 and 32.8; 1 x 9000, where an exchange is saved, 26.6 and 25.5).  Three chains of a CTA of three warps instead of six gave outputs
// that differed by 0.2 % with the form that a batch took (P is rounded against the maximum of its chain).  Producer warps stream [64 rows x 128] tiles by TMA
// through a ring (192 KB in flight per SM); each consumer warp owns two slots, so every slot is filled and drained by the same
// pair of warps in order.  The tile stream of an item:
//   1. ck tiles:           raw scores -> per-row maxima and sums of the unscaled soft-max over ALL compressed keys and
//                          of the scaled, masked attention soft-max (merged over the warps in shared memory);
//   2. (ck, cv) pairs:     scores again (ck comes from L2 this time) -> attention P.cv with the final statistics, and
//                          p_sel summed over the heads into a per-position vector in shared memory;
//                          then pooling and a warp top-n while the other warps go on;
//   3. window (k, v) pairs and 4. selected (k, v) pairs: online soft-max per warp.
// Every chain leaves its partial (maximum, sum, unnormalised output) of each branch in a caller-provided workspace (the split-KV
// scheme of decode attention).  The CTAs of an item then merge its rows, in a fixed order: without clusters each warp a row (of three warps
// two rows) at a time, from a scratch that the CTA's next item uses again while the ring fills with that item's tiles; with
// clusters each CTA its share of the rows, a row and branch per warp.  The scratch is to stay in L2 beside the caches that stream
// through it: CTAs that share an SM fetch what they read for the last time under an evict-first policy, the partials
// themselves when they merge them (the rows of the compressed cache then stay for the next step: 128 sequences of 1024 to 4000 keys,
// cache extended and decoded, 138 -> 135 us).
// Measured, 128 sequences of 4096 to 32768 keys, 4 KV heads, one CTA per SM / two: 164 / 140 to 144 us (4.7 to 4.9 TB/s); two without the policies
// 163, and with one row per warp at a time 165; a second kernel that merges (77 MB of partials written and read) 179; one
// sequence of 4096 keys 18.9 us with the second kernel and 17.5 without.  Also tried, with the same bits: two accumulators per warp of
// three, the chains' pairs in turn (185 us: twice the code); six warps in a CTA that shares its SM, on a ring of three pairs
// (196: too few tiles under way for a warp to wait as little).  Merging through shared memory, warp after warp, cost seven
// named barriers and six serialised rounds per branch.  No atomics; every wait is bounded.
#include <algorithm>
#include <array>

#include "kernels.h"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int D = 128;
constexpr int kCons = 6;                       // consumer warps of a CTA that has an SM to itself; chains of a phase
constexpr int kHalfCons = 3;                   // ... of one that shares it with another
// Producer warps of a CTA.
__host__ __device__ constexpr int decode_producers(int cons) { return cons == kCons ? 2 : 1; }
__host__ __device__ constexpr int decode_threads(int cons) { return (cons + decode_producers(cons)) * 32; }
static_assert(kCons == 2 * kHalfCons, "one chain per warp, or two");
constexpr uint32_t PANEL = 64 * 128;           // [64 rows][64 columns] bf16
constexpr uint32_t TILE = 2 * PANEL;           // 16 KB
constexpr int kMaxTc = 2048;                   // compressed positions of one sequence held in shared memory
constexpr int kMaxPoolD = 512;
constexpr int kMaxSel = 32;
constexpr int kPartFloats = 16 * D + 32;        // one warp's partial of one branch: O[16][D], m[16], l[16]
constexpr int kMaxCluster = 8;

struct Plan {   // tile pairs of one item's phases; CTA `rank` of a cluster takes all of pass 1, of the others rank, rank + cl, ...
  int L, Tc, nvis, row_k, row_c;
  int n1p;     // pairs of ck tiles of pass 1
  int n2p;     // (ck, cv) pairs of pass 2: covers all of Tc
  int nw;      // window pairs
  int cs;      // CTAs that share pass 2
  int w0;      // first window key
};

__device__ __forceinline__ Plan make_plan(const DecodeArgs& a, int seq, int cl) {
  Plan p;
  p.row_k = a.cu_k[seq];
  p.row_c = a.cu_c[seq];
  p.L = a.cu_k[seq + 1] - p.row_k;
  p.Tc = a.cu_c[seq + 1] - p.row_c;
  if (p.Tc > kMaxTc) p.Tc = kMaxTc;            // rejected on the host; keeps the indexing inside shared memory
  const int t = p.L - 1;
  p.nvis = (t < a.cblock) ? 0 : min(p.Tc, (t - a.cblock) / a.cstride + 1);
  const int nck = (p.Tc + 63) / 64;
  p.n1p = (nck + 1) / 2;
  p.n2p = nck;
  // An exchange costs about as much as one pair (3500 cycles): with no more than a pair for each warp the scores are not shared,
  // every CTA makes its own.
  p.cs = p.n2p > kCons ? cl : 1;
  p.w0 = max(0, p.L - a.window);
  p.nw = a.window > 0 ? (p.L - p.w0 + 63) / 64 : 0;
  return p;
}

// Items are dealt to the CTAs in boustrophedon order (left to right in even rounds, right to left in odd ones): with
// the sequences sorted longest first, every CTA then gets a long and a short item in turn (maximum / mean load 1.09
// for lengths uniform in [4096, 32768], against 1.23 for a plain round robin).
__device__ __forceinline__ int snake_item(int round, int cta, int ncta) {
  return round * ncta + ((round & 1) ? ncta - 1 - cta : cta);
}

// ---- the CTAs of a cluster -----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {   // releases what this thread has seen, to the cluster
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// bounded wait for a barrier that other CTAs arrive at
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, int code, volatile int* abort_flag) {
  const uint64_t t0 = global_timer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i) {
      uint32_t ok;
      asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                   : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
      if (ok) return true;
    }
    if (*abort_flag) return false;
    if (global_timer_ns() - t0 > 2000000000ull) {
      atomicCAS(&g_dev_error, 0, code);
      *abort_flag = 1;
      return false;
    }
  }
}

// avg_pool1d(kernel k, stride s, no padding, ceil_mode) output length, as nsa_pool_out_len computes it
__device__ __forceinline__ int pool_len(int n, int k, int s) {
  if (n <= 0) return 0;
  const int num = n - k;
  int out = (num >= 0 ? (num + s - 1) / s : -((-num) / s)) + 1;
  if ((out - 1) * s >= n) --out;
  return out < 0 ? 0 : out;
}

// How many tile pairs a CTA that has one of the GPU's `sms` SMs to itself has behind it when it comes to `item` (by one warp).
// Counts every block that can be selected: NaN among the scores takes some out, which then changes the order of a sum and no more.
__device__ __forceinline__ uint32_t pairs_before(const DecodeArgs& a, int item, int sms, int lane) {
  const int rounds = item / sms, x = item % sms, cta = rounds & 1 ? sms - 1 - x : x;
  uint32_t n = 0;
  for (int r = lane; r < rounds; r += 32) {
    const int sq = snake_item(r, cta, sms) / a.Hkv;
    const Plan p = make_plan(a, a.order ? a.order[sq] : sq, 1);
    n += p.n1p + p.n2p + p.nw + min(a.n_sel, min(kMaxPoolD, pool_len(p.Tc, a.sel_block / a.cstride + 1, a.sel_block / a.cstride)));
  }
  return __reduce_add_sync(0xffffffffu, n);
}

// acc (16 x 128) += P (16 x 64, in sc as mma C layout) . V tile
__device__ __forceinline__ void pv_tile(float (&acc)[D / 8][4], const float (&sc)[8][4], uint32_t vbase, int lane) {
  uint32_t pf[4][4];
  acc_to_a_frags<8>(pf, sc);
  mma_a_b<D, 64>(acc, pf, vbase, PANEL, 0, lane);
}

// The n blocks with the highest pooled score (ties to the lower index), in order, by one warp: lane l holds the blocks l + 32
// e as
// integers that order like the scores.  The n-th highest is found bit by bit, from the first bit in which the scores differ: a
// lane counts its own and one warp reduction adds.  The n survivors are ranked among themselves.  (A chain, on which the loads of
// the selected blocks wait; 16 of 512 blocks.  Counting by ballots from the highest bit 8800 cycles, n rounds of a shared-memory
// scan and a butterfly 6400 with the other warps' help, n rounds of two integer warp reductions 18000, every block's rank by all
// warps 38000.)
template <int E>
__device__ __forceinline__ int top_blocks(const float* pooled, int2* tmp, int n_pool, int n_sel, int lane) {   // lane r: the r-th, or -1
  unsigned v[E], hi = 0u, lo = 0xffffffffu;
  int valid = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int blk = lane + 32 * e;
    const float x = blk < n_pool ? pooled[blk] : -1.f;
    v[e] = x >= 0.f ? __float_as_uint(x) + 1u : 0u;   // 0: none
    valid += v[e] != 0u ? 1 : 0;
    hi = max(hi, v[e]);
    lo = min(lo, v[e] - 1u);   // (none: the highest)
  }
  valid = __reduce_add_sync(0xffffffffu, valid);
  hi = __reduce_max_sync(0xffffffffu, hi);
  lo = __reduce_min_sync(0xffffffffu, lo) + 1u;
  const int n = min(n_sel, valid);
  if (n == 0) return -1;
  // the highest value that at least n blocks reach, and how many do: all of them reach the bits that all have in common
  const unsigned differ = hi ^ lo;
  unsigned bit = differ ? 0x80000000u >> __clz(differ) : 0u;
  unsigned thr = bit ? hi & ~(2u * bit - 1u) : hi;
  int cnt = valid;
  for (; bit && cnt != n; bit >>= 1) {
    int c = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) c += v[e] >= (thr | bit) ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (c >= n) {
      thr |= bit;
      cnt = c;
    }
  }
  const unsigned below = (1u << lane) - 1u;
  if (cnt == n) {   // exactly these
    int own = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) own += v[e] >= thr && v[e] != 0u ? 1 : 0;
    int k = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, k, off);
      if (lane >= off) k += y;
    }
    k -= own;
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (v[e] >= thr && v[e] != 0u) tmp[k++] = make_int2((int)v[e], lane + 32 * e);
  } else {          // those above the threshold, and the first of those at it
    int above = 0, k = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) above += v[e] > thr ? 1 : 0;
    int ties = n - __reduce_add_sync(0xffffffffu, above);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const unsigned eq = __ballot_sync(0xffffffffu, v[e] == thr);
      const bool take = v[e] > thr || (v[e] == thr && __popc(eq & below) < ties);
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) tmp[k + __popc(m & below)] = make_int2((int)v[e], lane + 32 * e);
      k += __popc(m);
      ties -= min(ties, __popc(eq));
    }
  }
  __syncwarp();
  const int2 own = lane < n ? tmp[lane] : make_int2(0, 0);
  int rank = 0;
  for (int i = 0; i < n; ++i) {
    const int2 x = tmp[i];
    rank += (x.x > own.x || (x.x == own.x && x.y < own.y)) ? 1 : 0;
  }
  __syncwarp();
  if (lane < n) tmp[rank].x = own.y;
  __syncwarp();
  return lane < n ? tmp[lane].x : -1;
}

// A maximum passes over NaN scores, the sum of their exponentials is NaN.  Partials are merged by their maxima, and those of -inf
// left out: where the sum is NaN the maximum is made so too, and the NaN reaches the output.
__device__ __forceinline__ float nan_or(float sum, float m) { return sum == sum ? m : sum; }

// One (K, V) pair of an online soft-max: keys key0 .. key0+63 of the tile are valid iff kmin <= key < kmax.
__device__ __forceinline__ void online_pair(float (&acc)[D / 8][4], float (&m_run)[2], float (&l_run)[2],
                                            const uint32_t (&qf)[D / 16][4], uint32_t kbase, uint32_t vbase, uint32_t k_empty,
                                            uint32_t v_full, uint32_t v_par, uint32_t v_empty, int key0, int kmin, int kmax,
                                            float sl2, int lane, bool& ok, volatile int* abort_flag) {
  const int tq = lane & 3;
  float sc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
  if (ok) mma_a_bt<D, 64>(sc, qf, kbase, PANEL, 0, lane);
  __syncwarp();
  if (lane == 0) mbar_arrive(k_empty);
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int key = key0 + nt * 8 + 2 * tq + (c & 1);
      if (key < kmin || key >= kmax) sc[nt][c] = -INFINITY;
      mx[c >> 1] = fmaxf(mx[c >> 1], sc[nt][c]);
    }
  float alpha[2];
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    const float mnew = fmaxf(m_run[rr], quad_max(mx[rr]) * sl2);
    const float muse = (mnew == -INFINITY) ? 0.f : mnew;
    alpha[rr] = ex2(m_run[rr] - muse);
    m_run[rr] = mnew;
    float rs = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const float e0 = ex2(fmaf(sc[nt][2 * rr], sl2, -muse)), e1 = ex2(fmaf(sc[nt][2 * rr + 1], sl2, -muse));
      sc[nt][2 * rr] = e0;
      sc[nt][2 * rr + 1] = e1;
      rs += e0 + e1;
    }
    l_run[rr] = l_run[rr] * alpha[rr] + rs;
  }
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    acc[i][0] *= alpha[0];
    acc[i][1] *= alpha[0];
    acc[i][2] *= alpha[1];
    acc[i][3] *= alpha[1];
  }
  ok = ok && mbar_wait_abortable(v_full, v_par, DEV_ERR_FULL_WAIT, abort_flag);
  if (ok) pv_tile(acc, sc, vbase, lane);
  __syncwarp();
  if (lane == 0) mbar_arrive(v_empty);
}

// One row and branch of an item that a cluster shared: the partials of all its warps merged in a fixed order (CTA by CTA, warp by
// warp), by one warp, a lane holding four channels.  Branch order in the workspace: 0 compressed, 1 selected, 2 window.
// Warps that
// had no tile are left out.  The first loads are under way while the weights are formed.  Returns the output as rounded.
static_assert(kMaxCluster * kCons <= 64, "two partials per lane below");
__device__ __forceinline__ float4 merge_row(const DecodeArgs& a, int item, long long qrow, int r, int br, int nw, int lane) {
  constexpr int kFirst = 6;   // (no cluster has fewer warps)
  const float* part = a.part + ((long long)item * 3 + br) * nw * kPartFloats;
  const float* hd = part + 16 * D + r;
  float m[2], l[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    m[k] = -INFINITY;
    l[k] = 0.f;
    const int w = lane + 32 * k;
    if (w < nw) {
      m[k] = __ldcg(hd + w * kPartFloats);
      l[k] = __ldcg(hd + w * kPartFloats + 16);
    }
  }
  const float4* base = reinterpret_cast<const float4*>(part + r * D) + lane;
  float4 first[kFirst];
#pragma unroll
  for (int w = 0; w < kFirst; ++w) first[w] = __ldcg(base + w * (kPartFloats / 4));
  float M = fmaxf(m[0], m[1]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
  float e[2], L = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    e[k] = m[k] != -INFINITY ? ex2(m[k] - M) : 0.f;
    if (m[k] != -INFINITY) L += l[k] * e[k];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
  const float inv = L > 0.f ? 1.f / L : 0.f;
  e[0] *= inv;
  e[1] *= inv;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](const float4& x, float w) {
    v.x += x.x * w; v.y += x.y * w; v.z += x.z * w; v.w += x.w * w;
  };
#pragma unroll
  for (int w = 0; w < kFirst; ++w) {
    const float wt = __shfl_sync(0xffffffffu, e[0], w);
    if (wt != 0.f) add(first[w], wt);   // (a warp without a tile has left no output)
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    unsigned rest = __ballot_sync(0xffffffffu, e[k] != 0.f && (k || lane >= kFirst));
    while (rest) {   // eight at a time
      float4 x[8];
      float wt[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int w = rest ? __ffs(rest) - 1 : 0;
        wt[u] = rest ? __shfl_sync(0xffffffffu, e[k], w) : 0.f;
        if (rest) x[u] = __ldcg(base + (w + 32 * k) * (kPartFloats / 4));
        rest &= rest - 1;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (wt[u] != 0.f) add(x[u], wt[u]);
    }
  }
  const __nv_bfloat162 b0 = __floats2bfloat162_rn(v.x, v.y), b1 = __floats2bfloat162_rn(v.z, v.w);
  bf16* out = br == 0 ? a.o_cmp : br == 1 ? a.o_slc : a.o_swa;
  if (out) *reinterpret_cast<uint2*>(out + qrow * D + lane * 4) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  if (a.lse && lane == 0) a.lse[(long long)br * a.nseq * a.Hq + qrow] = L > 0.f ? (M + log2f(L)) * kLn2 : -INFINITY;
  const float2 f0 = __bfloat1622float2(b0), f1 = __bfloat1622float2(b1);
  return make_float4(f0.x, f0.y, f1.x, f1.y);
}

// CONS consumer warps with a pair of slots each; CL: the CTAs of a cluster share an item.
template <int CONS, bool CL>
__global__ void __launch_bounds__(decode_threads(CONS), CONS == kCons ? 1 : 2)
    decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                  const __grid_constant__ CUtensorMap tmCK, const __grid_constant__ CUtensorMap tmCV, const DecodeArgs a, const int ncl,
                  const int sms) {
  after_previous();
  constexpr int kSlots = 2 * CONS, kProdW = decode_producers(CONS);
  constexpr int kOwn = kCons / CONS;   // chains of a warp
  constexpr int kRows = kOwn, kLanes = 32 / kRows;   // rows that a warp merges at a time, lanes of one
  const int cl = CL ? ncl : 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ring = sbase;
  uint8_t* after = sgen + kSlots * TILE;
  float* ps = reinterpret_cast<float*>(after);                    // [kMaxTc + 64] head-summed p_sel per compressed position
  float* pooled = ps + kMaxTc + 64;                               // [kMaxPoolD]
  float* stat = pooled + kMaxPoolD;                               // [kCons][4][16] the chains' statistics
  float* fin = stat + kCons * 64;                                 // [4][16] merged: M_raw, 1/L_raw, M_att (log2), L_att
  float2* ml = reinterpret_cast<float2*>(fin + 64);               // [3][kCons][16] (m, l) of the chains' partials, without clusters
  float* gates = reinterpret_cast<float*>(ml + 3 * kCons * 16);      // [3][16], branch order as ml's
  int* sel = reinterpret_cast<int*>(gates + 48);                  // [kMaxSel] selected blocks of the item, [kMaxSel] = count
  volatile int* abort_flag = sel + kMaxSel + 2;
  const uint32_t bar_base = sbase + kSlots * TILE + (uint32_t)((uint8_t*)(sel + kMaxSel + 4) - after);
  const uint32_t bar0 = (bar_base + 7u) & ~7u;
  auto full_bar = [&](uint32_t s) { return bar0 + 8u * s; };
  auto empty_bar = [&](uint32_t s) { return bar0 + 8u * (kSlots + s); };
  const uint32_t sel_ready = bar0 + 8u * (2 * kSlots);
  const uint32_t ps_bar = sel_ready + 8;   // every CTA's scores have arrived here
  const int rank = cl > 1 ? (int)cluster_rank() : 0, group = blockIdx.x / cl, ngroup = gridDim.x / cl;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(sel_ready, 1);
    mbar_init(ps_bar, cl);
    fence_mbar_init();
  }
  __syncthreads();
  if (cl > 1) cluster_sync_all();   // no CTA writes into another's shared memory before it runs, or after it ended (below)

  const int nitem = a.nseq * a.Hkv;
  // of the pairs of a phase that cs CTAs share: how many are this CTA's, and which is its i-th
  auto share = [&](int n, int cs) { return !CL || cs == 1 ? n : (n - rank + cs - 1) / cs; };
  auto deal = [&](int i, int cs) { return !CL || cs == 1 ? i : rank + i * cs; };
  const int pool_k = a.sel_block / a.cstride + 1, pool_s = a.sel_block / a.cstride;

  if (warp >= CONS) {
    // ------------------------------- producers --------------------------------------------------------
    // Tiles go out in pairs (both tiles of a (K, V) pair, or two consecutive ck tiles of pass 1: the two slots of a consumer
    // warp), and the producer warps (one in a CTA that shares its SM) take alternate pairs.
    const int pw = warp - CONS;
    uint32_t np = 0, it = 0;     // tile pairs issued so far by both producers together; items so far
    // what an item reads for the last time goes first from L2, before the partials of 2 x 148 CTAs (44 MB)
    const uint64_t once = l2_evict_first();
    bool last = false;
    auto issue2 = [&](const CUtensorMap* tmA, int rowA, const CUtensorMap* tmB, int rowB, int h) -> bool {
      const uint32_t mine = np % kProdW == (uint32_t)pw;
      const uint32_t n = 2 * np;
      ++np;
      if (!mine) return true;
      const uint32_t s0 = n % kSlots, ph = (n / kSlots) & 1;     // the pair's slots s0, s0+1 belong to one consumer warp
      const bool good = mbar_wait_abortable(empty_bar(s0), ph ^ 1, DEV_ERR_EMPTY_WAIT, abort_flag) &&
                        mbar_wait_abortable(empty_bar(s0 + 1), ph ^ 1, DEV_ERR_EMPTY_WAIT, abort_flag);
      if (!__all_sync(0xffffffffu, good)) return false;
      if (elect_one()) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          mbar_expect_tx(full_bar(s0 + w), TILE);
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            const uint32_t dst = ring + (s0 + w) * TILE + p * PANEL;
            if (kOwn > 1 && last)
              tma_load_4d(dst, w ? tmB : tmA, full_bar(s0 + w), p * 64, h, w ? rowB : rowA, 0, once);
            else
              tma_load_4d(dst, w ? tmB : tmA, full_bar(s0 + w), p * 64, h, w ? rowB : rowA, 0);
          }
        }
      }
      return true;
    };
    // the n pairs of a phase as the warps take them: those of the first CONS chains, then (CONS < kCons) of the others
    auto each_pair = [&](int n, bool& ok, auto&& issue) {
      if constexpr (kOwn == 1) {
        for (int i = 0; ok && i < n; ++i) ok = issue(i);
      } else {
        for (int e = 0; e < kCons; e += CONS)
          for (int c = e; c < n; c += kCons)
            for (int i = c; ok && i < min(c + CONS, n); ++i) ok = issue(i);
      }
    };
    for (int r = 0; r * ngroup < nitem; ++r) {
      const int item = snake_item(r, group, ngroup);
      if (item >= nitem) continue;
      const int sq = item / a.Hkv, h = item % a.Hkv;
      const int seq = a.order ? a.order[sq] : sq;
      const Plan p = make_plan(a, seq, cl);
      bool ok = true;
      last = false;
      each_pair(p.n1p, ok, [&](int j) { return issue2(&tmCK, p.row_c + j * 128, &tmCK, p.row_c + j * 128 + 64, h); });
      last = true;
      each_pair(share(p.n2p, p.cs), ok, [&](int i) {
        const int j = deal(i, p.cs);
        return issue2(&tmCK, p.row_c + j * 64, &tmCV, p.row_c + j * 64, h);
      });
      each_pair(share(p.nw, cl), ok, [&](int i) {
        const int j = deal(i, cl);
        return issue2(&tmK, p.row_k + p.w0 + j * 64, &tmV, p.row_k + p.w0 + j * 64, h);
      });
      // the selected blocks are known once the consumers have pooled the scores
      if (ok && lane == 0) ok = mbar_wait_abortable(sel_ready, it & 1, DEV_ERR_FULL_WAIT, abort_flag);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      const int nsel = *reinterpret_cast<volatile int*>(sel + kMaxSel);
      each_pair(share(nsel, cl), ok, [&](int i) {
        const int blk = *reinterpret_cast<volatile int*>(sel + deal(i, cl));
        return issue2(&tmK, p.row_k + blk * 64, &tmV, p.row_k + blk * 64, h);
      });
      if (!ok) break;
      ++it;
    }
  } else {
  // --------------------------------- consumers ----------------------------------------------------------
  const int g = lane >> 2, tq = lane & 3;
  const float sl2 = a.scale * kLog2e;
  const int cthreads = CONS * 32;
  const int ct = threadIdx.x;               // 0 .. cthreads-1
  // Six chains in every phase: chain c has the pairs c, c + 6, ...  A warp of six has one of them.  A warp of three has two, one after
  // the other: the same terms in the same order, so that outputs have the same bits, with one accumulator.
  // tile pair i of the CTA, over all phases and items, is warp i % CONS's, in that warp's own two slots
  uint32_t np0 = 0, it = 0;                 // pairs of the CTA so far (before the current phase's current chains); items so far
  uint32_t own0 = 0;                        // pairs before the current phase of the CTA of six warps that would have the item
  uint32_t use = 0;                         // pairs of this warp so far
  const uint32_t sk = 2 * warp, sv = sk + 1;
  // this warp's chain of a phase: of the first CONS ones (e = 0) or of the others
  auto chain_of = [&](int e) { return (int)((warp + CONS - np0 % CONS) % CONS) + e * CONS; };
  auto pairs_of = [&](int n, int e) { return kOwn == 1 ? n : n / kCons * CONS + max(0, min(n % kCons - e * CONS, CONS)); };   // of all warps
  // where its partial goes: to the warp that has the chain in a CTA of six
  auto part_of = [&](int chain) { return kOwn == 1 ? warp : (int)((own0 + chain) % kCons); };
  bool ok = true;
  for (int r = 0; r * ngroup < nitem; ++r) {
    const int item = snake_item(r, group, ngroup);
    if (item >= nitem) continue;
    const int sq = item / a.Hkv, h = item % a.Hkv;
    const int seq = a.order ? a.order[sq] : sq;
    const Plan p = make_plan(a, seq, cl);
    const int t = p.L - 1;
    const long long qrow = (long long)seq * a.Hq + h * 16;     // first of the 16 (head) rows of this item
    uint32_t qf[D / 16][4];
    load_a_frags_global<D>(qf, a.q + qrow * D, lane);
    if (kOwn > 1) own0 = pairs_before(a, item, sms, lane);

    // ---- pass 1: statistics over all compressed keys ---------------------------------------------------
#pragma unroll 1
    for (int e = 0; e < kOwn; ++e) {
      float mr[2] = {-INFINITY, -INFINITY}, lr[2] = {0.f, 0.f};   // raw scores, all keys (natural-log domain kept in log2)
      float ma[2] = {-INFINITY, -INFINITY}, la[2] = {0.f, 0.f};   // scaled scores, visible keys
      const int chain = chain_of(e);
      for (int u = chain; u < p.n1p; u += kCons, ++use) {
#pragma unroll 1
        for (int t2 = 0; t2 < 2; ++t2) {
          const uint32_t s = sk + t2;
          const int j0 = (2 * u + t2) * 64;
          ok = ok && mbar_wait_abortable(full_bar(s), use & 1, DEV_ERR_FULL_WAIT, abort_flag);
          float sc[8][4];
#pragma unroll
          for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
          if (ok) mma_a_bt<D, 64>(sc, qf, ring + s * TILE, PANEL, 0, lane);
          __syncwarp();
          if (lane == 0) mbar_arrive(empty_bar(s));
          float mxr[2] = {-INFINITY, -INFINITY}, mxa[2] = {-INFINITY, -INFINITY};
#pragma unroll
          for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int j = j0 + nt * 8 + 2 * tq + (c & 1);
              if (j < p.Tc) mxr[c >> 1] = fmaxf(mxr[c >> 1], sc[nt][c]);
              if (j < p.nvis) mxa[c >> 1] = fmaxf(mxa[c >> 1], sc[nt][c]);
            }
#pragma unroll
          for (int rr = 0; rr < 2; ++rr) {
            const float nr = fmaxf(mr[rr], quad_max(mxr[rr]) * kLog2e), na = fmaxf(ma[rr], quad_max(mxa[rr]) * sl2);
            const float ur = (nr == -INFINITY) ? 0.f : nr, ua = (na == -INFINITY) ? 0.f : na;
            float sr = 0.f, sa = 0.f;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
              for (int c2 = 0; c2 < 2; ++c2) {
                const int j = j0 + nt * 8 + 2 * tq + c2;
                const float x = sc[nt][2 * rr + c2];
                if (j < p.Tc) sr += ex2(fmaf(x, kLog2e, -ur));
                if (j < p.nvis) sa += ex2(fmaf(x, sl2, -ua));
              }
            lr[rr] = lr[rr] * ex2(mr[rr] - ur) + sr;
            la[rr] = la[rr] * ex2(ma[rr] - ua) + sa;
            mr[rr] = nr;
            ma[rr] = na;
          }
        }
      }
      // the statistics of the chains are merged in their order whichever warps had them, so that an item's scores do not depend on
      // the items before it (each value lives in the four lanes of a quad: sum the partial sums)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const float l_r = quad_sum(lr[rr]), l_a = quad_sum(la[rr]);
        if (tq == 0) {
          float* st = stat + chain * 64;
          st[0 * 16 + g + 8 * rr] = mr[rr];
          st[1 * 16 + g + 8 * rr] = l_r;
          st[2 * 16 + g + 8 * rr] = nan_or(l_a, ma[rr]);
          st[3 * 16 + g + 8 * rr] = l_a;
        }
      }
      np0 += pairs_of(p.n1p, e);
    }
    own0 += p.n1p;
    named_bar_sync(1, cthreads);
    if (ct < 16) {
      float Mr = -INFINITY, Ma = -INFINITY;
      for (int w = 0; w < kCons; ++w) {
        Mr = fmaxf(Mr, stat[w * 64 + ct]);
        Ma = fmaxf(Ma, stat[w * 64 + 32 + ct]);
      }
      float Lr = 0.f, La = 0.f;
      for (int w = 0; w < kCons; ++w) {
        const float m1 = stat[w * 64 + ct], m2 = stat[w * 64 + 32 + ct];
        if (m1 > -INFINITY) Lr += stat[w * 64 + 16 + ct] * ex2(m1 - Mr);
        if (m2 != -INFINITY) La += stat[w * 64 + 48 + ct] * ex2(m2 - Ma);
      }
      fin[ct] = Mr;
      fin[16 + ct] = Lr > 0.f ? 1.f / Lr : 0.f;
      fin[32 + ct] = Ma;
      fin[48 + ct] = La;
    }
    named_bar_sync(1, cthreads);
    float Mr[2], iLr[2], Ma[2], La[2];
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      Mr[rr] = fin[g + 8 * rr];
      iLr[rr] = fin[16 + g + 8 * rr];
      Ma[rr] = fin[32 + g + 8 * rr];
      La[rr] = fin[48 + g + 8 * rr];
      if (Mr[rr] == -INFINITY) Mr[rr] = 0.f;
      if (Ma[rr] == -INFINITY) Ma[rr] = 0.f;
    }

    // a chain's partial of a branch -> workspace: [item][branch][chain of the cluster]{ O[16][D], m[16], l[16] } fp32; a chain
    // that had no tile leaves m = -inf and no O
    auto put_partial = [&](int branch, int w, const float (&x)[D / 8][4], const float (&mm)[2], const float (&ll)[2], bool has) {
      float* dst = a.part + (((long long)(cl > 1 ? item : (int)blockIdx.x) * 3 + branch) * (cl * kCons) + rank * kCons + w) * kPartFloats;
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        if (!has) break;
        *reinterpret_cast<float2*>(dst + g * D + i * 8 + 2 * tq) = make_float2(x[i][0], x[i][1]);
        *reinterpret_cast<float2*>(dst + (g + 8) * D + i * 8 + 2 * tq) = make_float2(x[i][2], x[i][3]);
      }
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const float l = quad_sum(ll[rr]);
        if (tq == 0) {
          const float m = has ? nan_or(l, mm[rr]) : -INFINITY;
          if (cl > 1) {
            dst[16 * D + g + 8 * rr] = m;
            dst[16 * D + 16 + g + 8 * rr] = l;
          } else {
            ml[(branch * kCons + w) * 16 + g + 8 * rr] = make_float2(m, l);
          }
        }
      }
    };
    // compressed branch: every chain used the final maximum; the row sum is known to the CTA and rides with the first partial
    auto put_compressed = [&](int w, const float (&x)[D / 8][4], bool has) {
      float mm[2], ll[2];
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        mm[rr] = fin[32 + g + 8 * rr];
        ll[rr] = (rank == 0 && w == 0 && tq == 0) ? La[rr] : 0.f;
      }
      put_partial(0, w, x, mm, ll, has);
    };

    // ---- pass 2: attention over the visible compressed keys and the block scores -------------------------
    float acc[D / 8][4];
    bool full = false;   // the chain's partial has an output
#pragma unroll 1
    for (int e = 0; e < kOwn; ++e) {
      const int n = share(p.n2p, p.cs), chain = chain_of(e), part = part_of(chain);
#pragma unroll
      for (int i = 0; i < D / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      full = rank == 0 && part == 0;   // (the first always: the row sums ride with it)
      for (int i = chain; i < n; i += kCons, ++use) {
        const int u = deal(i, p.cs);
        full = p.cs > 1 || rank == 0;
        const int j0 = u * 64;
        ok = ok && mbar_wait_abortable(full_bar(sk), use & 1, DEV_ERR_FULL_WAIT, abort_flag);
        float sc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
        if (ok) mma_a_bt<D, 64>(sc, qf, ring + sk * TILE, PANEL, 0, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(sk));
        // p_sel summed over the 16 heads: rows live in the eight quads of the warp
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          float c0 = 0.f, c1 = 0.f;   // columns nt*8 + 2 tq and + 1, rows g and g+8 of this thread
#pragma unroll
          for (int rr = 0; rr < 2; ++rr) {
            c0 += ex2(fmaf(sc[nt][2 * rr], kLog2e, -Mr[rr])) * iLr[rr];
            c1 += ex2(fmaf(sc[nt][2 * rr + 1], kLog2e, -Mr[rr])) * iLr[rr];
          }
#pragma unroll
          for (int off = 4; off < 32; off <<= 1) {
            c0 += __shfl_xor_sync(0xffffffffu, c0, off);
            c1 += __shfl_xor_sync(0xffffffffu, c1, off);
          }
          if (g == 0) {
            const int j = j0 + nt * 8 + 2 * tq;
            if (j < p.Tc) ps[j] = c0;
            if (j + 1 < p.Tc) ps[j + 1] = c1;
          }
        }
        if (p.cs > 1) {   // the tile's 64 scores to the other CTAs (positions past Tc are there, and not read)
          __syncwarp();
          const float* src = ps + j0 + 2 * lane;
          const float2 v = *reinterpret_cast<const float2*>(src);
          for (int c = 0; c < cl; ++c)
            if (c != rank) st_cluster(map_cta(smem_u32(src), c), v);
        }
        // attention weights with the final maximum (unnormalised; the sum divides at the end)
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int j = j0 + nt * 8 + 2 * tq + (c & 1);
            sc[nt][c] = (j < p.nvis) ? ex2(fmaf(sc[nt][c], sl2, -Ma[c >> 1])) : 0.f;
          }
        ok = ok && mbar_wait_abortable(full_bar(sv), use & 1, DEV_ERR_FULL_WAIT, abort_flag);
        if (ok && j0 < p.nvis && (p.cs > 1 || rank == 0)) pv_tile(acc, sc, ring + sv * TILE, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(sv));
      }
      np0 += pairs_of(n, e);
      if (kOwn > 1) put_compressed(part, acc, full);
    }
    own0 += p.n2p;
    // ---- pooled scores and the top-n (warp 0), the compressed-branch output (all warps, fixed order) ------------
    named_bar_sync(1, cthreads);            // ps complete
    if (p.cs > 1) {   // in every CTA
      if (ct < cl) arrive_cluster(map_cta(ps_bar, ct));
      ok = ok && wait_cluster(ps_bar, 0, 321, abort_flag);   // (a cluster has one item)
    }
    const int n_pool = min(kMaxPoolD, pool_len(p.Tc, pool_k, pool_s));
    for (int blk = ct; blk < n_pool; blk += cthreads) {
      const int lo = blk * pool_s, hi = min(lo + pool_k, p.Tc);
      float sum = 0.f;
      for (int j = lo; j < hi; ++j) sum += ps[j];
      pooled[blk] = sum / (float)(hi - lo);
    }
    named_bar_sync(1, cthreads);
    if (warp == 0) {
      const int blk = n_pool <= 128 ? top_blocks<4>(pooled, reinterpret_cast<int2*>(stat), n_pool, a.n_sel, lane) : top_blocks<kMaxPoolD / 32>(pooled, reinterpret_cast<int2*>(stat), n_pool, a.n_sel, lane);
      if (rank == 0 && lane < a.n_sel) a.idx[((long long)seq * a.Hkv + h) * a.n_sel + lane] = blk;   // n_sel <= kMaxSel = 32
      const bool use = blk >= 0 && (long long)blk * 64 <= t;   // blocks that start after t are skipped
      const unsigned m = __ballot_sync(0xffffffffu, use);
      __syncwarp();
      if (use) sel[__popc(m & ((1u << lane) - 1))] = blk;
      __syncwarp();
      if (lane == 0) {
        sel[kMaxSel] = __popc(m);
        __threadfence_block();
        mbar_arrive(sel_ready);
      }
    }
    if (kOwn == 1) put_compressed(warp, acc, full);

    // ---- gates, by the last warp (the first one is still choosing blocks) --------------------------------
    // (what the item before left in gates, ml and the scratch has been read: its rows are merged before anything of this one)
    if (warp == CONS - 1) {
      if (a.gate_w) {
        // g_x[row] = q[row,:] . W[x,:] + b[x] (nn.Linear(head_dim, 3), rows of W: selected, window, compressed) as one 16 x 8
        // tile of mma.sync, rounded to bf16 as the module's gate tensors are
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t wf[D / 16][2];
        auto two = [](const bf16* x) {   // (a parameter may lie at any address)
          const unsigned short* p = reinterpret_cast<const unsigned short*>(x);
          return (uint32_t)p[0] | (uint32_t)p[1] << 16;
        };
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const bf16* w = a.gate_w + g * D + ks * 16 + 2 * tq;
          wf[ks][0] = g < 3 ? two(w) : 0u;
          wf[ks][1] = g < 3 ? two(w + 8) : 0u;
        }
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) mma_bf16(c, qf[ks], wf[ks][0], wf[ks][1]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int x = 2 * tq + (i & 1);
          if (x < 3) gates[(x == 2 ? 0 : x + 1) * 16 + g + 8 * (i >> 1)] = __bfloat162float(__float2bfloat16(c[i] + (a.gate_b ? __bfloat162float(a.gate_b[x]) : 0.f)));
        }
      } else if (lane < 16) {
#pragma unroll
        for (int br = 0; br < 3; ++br) {
          const bf16* gin = br == 0 ? a.g_cmp : br == 1 ? a.g_slc : a.g_swa;
          gates[br * 16 + lane] = gin ? __bfloat162float(gin[qrow + lane]) : 1.f;
        }
      }
    }

    // ---- window ---------------------------------------------------------------------------------------
#pragma unroll 1
    for (int e = 0; e < kOwn; ++e) {
      const int n = share(p.nw, cl), chain = chain_of(e), part = part_of(chain);
      float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
      for (int i = 0; i < D / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      full = false;
      for (int i = chain; i < n; i += kCons, ++use) {
        const int u = deal(i, cl);
        full = true;
        ok = ok && mbar_wait_abortable(full_bar(sk), use & 1, DEV_ERR_FULL_WAIT, abort_flag);
        online_pair(acc, m_run, l_run, qf, ring + sk * TILE, ring + sv * TILE, empty_bar(sk), full_bar(sv), use & 1,
                    empty_bar(sv), p.w0 + u * 64, p.w0, p.L, sl2, lane, ok, abort_flag);
      }
      np0 += pairs_of(n, e);
      // l_run holds this lane's share of the row sums (four lanes per row): put_partial adds the quad
      put_partial(2, part, acc, m_run, l_run, full);
    }
    own0 += p.nw;

    // ---- selected blocks ---------------------------------------------------------------------------------
    ok = ok && mbar_wait_abortable(sel_ready, it & 1, DEV_ERR_FULL_WAIT, abort_flag);
    const int nsel = *reinterpret_cast<volatile int*>(sel + kMaxSel);
#pragma unroll 1
    for (int e = 0; e < kOwn; ++e) {
      const int n = share(nsel, cl), chain = chain_of(e), part = part_of(chain);
      float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
      for (int i = 0; i < D / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      full = false;
      for (int i = chain; i < n; i += kCons, ++use) {
        const int u = deal(i, cl);
        full = true;
        const int blk = *reinterpret_cast<volatile int*>(sel + u);
        ok = ok && mbar_wait_abortable(full_bar(sk), use & 1, DEV_ERR_FULL_WAIT, abort_flag);
        online_pair(acc, m_run, l_run, qf, ring + sk * TILE, ring + sv * TILE, empty_bar(sk), full_bar(sv), use & 1,
                    empty_bar(sv), blk * 64, 0, p.L, sl2, lane, ok, abort_flag);
      }
      np0 += pairs_of(n, e);
      put_partial(1, part, acc, m_run, l_run, full);
    }
    named_bar_sync(1, cthreads);   // ps, pooled, fin and sel are reused by the next item
    ++it;
    // ---- this item's rows: partials merged chain by chain, gated sum of the branches (a lane holds four channels of every kRows-th of a
    // row; two rows at a time where three warps share them) -----------------------------------------------------------------
    const uint64_t once = l2_evict_first();
    for (int r0 = warp; cl == 1 && r0 < 16 / kRows; r0 += CONS) {
      const int row = kRows * r0 + lane / kLanes, c0 = 4 * (lane % kLanes);
      const float4* base = reinterpret_cast<const float4*>(a.part + (long long)blockIdx.x * 3 * kCons * kPartFloats + row * D + c0);
      float4 x[3][kCons][kRows];
      float e[3][kCons], inv[3], lse[3];
#pragma unroll
      for (int br = 0; br < 3; ++br)
#pragma unroll
        for (int w = 0; w < kCons; ++w) {
          e[br][w] = ml[(br * kCons + w) * 16 + row].x;
#pragma unroll
          for (int k = 0; k < kRows; ++k) {
            x[br][w][k] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4* src = base + (br * kCons + w) * (kPartFloats / 4) + kLanes * k;
            if (e[br][w] != -INFINITY) x[br][w][k] = kOwn > 1 ? ld_l2(src, once) : __ldcg(src);
          }
        }
#pragma unroll
      for (int br = 0; br < 3; ++br) {
        float M = e[br][0], L = 0.f;
#pragma unroll
        for (int w = 1; w < kCons; ++w) M = fmaxf(M, e[br][w]);
#pragma unroll
        for (int w = 0; w < kCons; ++w) {
          e[br][w] = e[br][w] != -INFINITY ? ex2(e[br][w] - M) : 0.f;
          L += ml[(br * kCons + w) * 16 + row].y * e[br][w];
        }
        inv[br] = L > 0.f ? 1.f / L : 0.f;
        lse[br] = L > 0.f ? (M + log2f(L)) * kLn2 : -INFINITY;
      }
      float4 tot[kRows];
#pragma unroll
      for (int k = 0; k < kRows; ++k) tot[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int br = 0; br < 3; ++br) {
        if (br == 2 && a.window <= 0) continue;
        bf16* out = br == 0 ? a.o_cmp : br == 1 ? a.o_slc : a.o_swa;
        const float gt = gates[br * 16 + row];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int w = 0; w < kCons; ++w) {
            const float wt = e[br][w] * inv[br];
            v.x = fmaf(x[br][w][k].x, wt, v.x);
            v.y = fmaf(x[br][w][k].y, wt, v.y);
            v.z = fmaf(x[br][w][k].z, wt, v.z);
            v.w = fmaf(x[br][w][k].w, wt, v.w);
          }
          const __nv_bfloat162 b0 = __floats2bfloat162_rn(v.x, v.y), b1 = __floats2bfloat162_rn(v.z, v.w);
          if (out) *reinterpret_cast<uint2*>(out + (qrow + row) * D + c0 + 4 * kLanes * k) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
          const float2 f0 = __bfloat1622float2(b0), f1 = __bfloat1622float2(b1);
          tot[k].x += gt * f0.x; tot[k].y += gt * f0.y; tot[k].z += gt * f1.x; tot[k].w += gt * f1.y;
        }
        if (a.lse && lane % kLanes == 0) a.lse[(long long)br * a.nseq * a.Hq + qrow + row] = lse[br];
      }
#pragma unroll
      for (int k = 0; k < kRows; ++k)
        *reinterpret_cast<uint2*>(a.o + (qrow + row) * D + c0 + 4 * kLanes * k) = make_uint2(pack_bf16(tot[k].x, tot[k].y), pack_bf16(tot[k].z, tot[k].w));
    }
  }
  }
  if (CL) {
    __syncwarp();
    cluster_sync_all();   // every CTA's partials are written (a cluster has one item), and no CTA writes into another's memory any more
    if (warp >= CONS) return;
    const int item = group, sq = item / a.Hkv, h = item % a.Hkv, rows = 16 / cl, nb = a.window > 0 ? 3 : 2;
    const long long qrow = (long long)(a.order ? a.order[sq] : sq) * a.Hq + h * 16 + rank * rows;   // first of this CTA's rows
    float4* out = reinterpret_cast<float4*>(ps);   // [row][branch][lane], over what the item no longer needs
    for (int u = warp; u < rows * nb; u += CONS) out[u * 32 + lane] = merge_row(a, item, qrow + u / nb, rank * rows + u / nb, u % nb, cl * kCons, lane);
    named_bar_sync(1, CONS * 32);
    for (int row = warp; row < rows; row += CONS) {
      float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int br = 0; br < nb; ++br) {
        const float gt = gates[br * 16 + rank * rows + row];
        const float4 f = out[(row * nb + br) * 32 + lane];
        tot.x += gt * f.x; tot.y += gt * f.y; tot.z += gt * f.z; tot.w += gt * f.w;
      }
      *reinterpret_cast<uint2*>(a.o + (qrow + row) * D + lane * 4) = make_uint2(pack_bf16(tot.x, tot.y), pack_bf16(tot.z, tot.w));
    }
  }
}

constexpr int decode_smem(int cons) {
  return 2 * cons * (int)TILE + (kMaxTc + 64 + kMaxPoolD + kCons * 64 + 64 + 3 * kCons * 32 + 48) * 4 + (kMaxSel + 4) * 4 +
         (4 * cons + 2) * 8 + 16 + 1024;
}
static_assert(2 * (decode_smem(kHalfCons) + 1024) <= 228 * 1024, "two CTAs per SM");

// A launch of `ncta` CTAs in clusters of `cl`; at: two attributes.
cudaLaunchConfig_t decode_config(int ncta, int cons, int cl, cudaLaunchAttribute* at, cudaStream_t s) {
  cudaLaunchConfig_t cfg = next_config(dim3((unsigned)ncta), dim3(decode_threads(cons)), decode_smem(cons), s, at);
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cl;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  if (cl > 1) cfg.numAttrs = 2;
  return cfg;
}
// Clusters of cl CTAs that the GPU holds at a time (fewer than SMs / cl: a cluster lies within one GPC; 16 of 8 would be 128
// of 148 SMs, but they do not all fit and the rest would run as a second wave).
int ask_resident(int cl) {
  int c = 0;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = decode_config(num_sms() / cl * cl, kCons, cl, at, nullptr);
  cfg.attrs = at + 1;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(decode_kernel<kCons, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem(kCons)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&c, decode_kernel<kCons, true>, &cfg) != cudaSuccess)
    c = num_sms() / cl;
  cudaGetLastError();   // (no device: workspace sizes can be asked for all the same)
  return c;
}
// How `nitem` items are spread: up to the number of SMs as many CTAs per item as keep every item in the first wave, with an SM to
// itself each; with more items two CTAs of half the warps and slots share an SM, so that one streams tiles while the other chooses
// its blocks or merges its rows.  Below two items per SM such a CTA has one item and takes 32 us + 1.2 us per 1000 keys for the
// longest, against two items, a long and a short one, behind each other.  One CTA per SM -> two, 4 KV heads, lengths from 1024 up to the
// given one: 152 items of 4000 keys 44.2 -> 36.9 us, 192 of 9000 51.2 -> 45.4, 272 of 16000 68.4 -> 58.9; but 152 of 20000 46.6 -> 56.5, 168 of
// 26000 54.9 -> 63.8, 248 of 32000 75.7 -> 77.6, so not there.  512 items of 4096 to 32768 keys 164 -> 140, 512 of 1500 99 -> 85.
// Three rounds of equal items are no more than two of pairs, the second half empty: 300 to 444 items of 32000 keys 160 to 179 us, as
// pairs 169 to 184 (of 12000 100 to 114, 103 to 114); four are: 452 of 32000 218 -> 185.
struct Spread {
  int cons, cl, ncta;
};
const std::array<int, 4>& clusters_held() {
  static const std::array<int, 4> held = {num_sms(), ask_resident(2), ask_resident(4), ask_resident(8)};
  return held;
}
Spread decode_spread(int nitem, int max_Tc, bool even) {   // even: the longest sequence is within 1.3 of the mean
  const std::array<int, 4>& held = clusters_held();
  for (int i = 3; i >= 0; --i)
    if (nitem <= held[i]) return {kCons, 1 << i, nitem << i};
  const int sms = num_sms();
  if (nitem < 2 * sms && max_Tc > 768 + (int)(640LL * (nitem - sms) / sms)) return {kCons, 1, sms};   // (12 K keys, 22 K with two items per SM)
  if (even && nitem > 2 * sms && nitem <= 3 * sms) return {kCons, 1, sms};
  return {kHalfCons, 1, std::min(nitem, 2 * sms)};
}

}  // namespace

// A set of partials for every CTA (of a cluster: one item each): as many as any number of items up to this one needs, so that a
// workspace made for a batch serves the smaller ones too.
size_t decode_workspace_bytes(int nseq, int Hkv) {
  const std::array<int, 4>& held = clusters_held();
  int ncta = nseq * Hkv > held[0] ? std::min(nseq * Hkv, 2 * num_sms()) : 0;
  for (int i = 0; i < 4; ++i) ncta = std::max(ncta, std::min(nseq * Hkv, held[i]) << i);
  return (size_t)ncta * 3 * kCons * kPartFloats * sizeof(float);
}

int launch_decode(const DecodeArgs& a, cudaStream_t s) {
  if (a.D != D) {
    set_error("decode: head_dim %d not supported (128)", a.D);
    return -2;
  }
  if (a.Hq != 16 * a.Hkv) {
    set_error("decode: needs exactly 16 query heads per KV head (got %d / %d)", a.Hq, a.Hkv);
    return -7;
  }
  if (a.sel_block != 64 || a.cstride != 16 || a.cblock != 32 || a.n_sel < 1 || a.n_sel > kMaxSel || a.window < 0) {
    set_error("decode: needs 64-key selection blocks, compression 32/16 and 1..%d selected blocks", kMaxSel);
    return -9;
  }
  if (a.max_Tc > kMaxTc) {
    set_error("decode: a sequence has %d compressed positions, the kernel holds %d (cache length <= %d)", a.max_Tc, kMaxTc,
              (kMaxTc - 1) * a.cstride + a.cblock + a.cstride - 1);
    return -14;
  }
  CUtensorMap tmK, tmV, tmCK, tmCV;
  int rc = make_tmap_rows4d(&tmK, a.k, D, a.Hkv, a.total_k, 1, 64);
  if (!rc) rc = make_tmap_rows4d(&tmV, a.v, D, a.Hkv, a.total_k, 1, 64);
  if (!rc) rc = make_tmap_rows4d(&tmCK, a.ck, D, a.Hkv, a.total_c, 1, 64);
  if (!rc) rc = make_tmap_rows4d(&tmCV, a.cv, D, a.Hkv, a.total_c, 1, 64);
  if (rc) return rc;
  if (!a.part || a.part_bytes < decode_workspace_bytes(a.nseq, a.Hkv)) {
    set_error("decode: workspace too small (%lld bytes needed)", (long long)decode_workspace_bytes(a.nseq, a.Hkv));
    return -6;
  }
  const int nitem = a.nseq * a.Hkv;
  if (nitem <= 0) return 0;
  const Spread p = decode_spread(nitem, a.max_Tc, 10LL * a.max_Tc * a.nseq <= 13 * a.total_c);
  const int cl = p.cl;
  const auto kernel = p.cons == kHalfCons ? decode_kernel<kHalfCons, false> : cl > 1 ? decode_kernel<kCons, true> : decode_kernel<kCons, false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem(p.cons));
  if (e != cudaSuccess) return (int)e;
  {
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = decode_config(p.ncta, p.cons, cl, at, s);
    e = cudaLaunchKernelEx(&cfg, kernel, tmK, tmV, tmCK, tmCV, a, cl, num_sms());
    if (e != cudaSuccess) return (int)e;
  }
  note_launches(1);
  return (int)cudaGetLastError();
}
int decode_status(int* out) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(out, g_dev_error, sizeof(int));
  if (e == cudaSuccess && *out) e = cudaMemcpyToSymbol(g_dev_error, &zero, sizeof(int));
  return (int)e;
}

}  // namespace nsa
