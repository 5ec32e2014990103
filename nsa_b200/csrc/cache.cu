// The compressed cache of a generation loop and the weight layout of the compression kernels.
//
// Extending a packed cache by the tokens of one step moves every sequence's compressed rows to their new offset and
// appends the few positions that the new tokens complete.  All length arithmetic is done here on the host from the
// caller's length tables; the device tables travel as kernel parameters (no pinned staging, no pageable copy, so no
// stream synchronisation), the moved rows are one kernel over both tensors, and the new rows are one launch of the
// compression GEMM with a first position per sequence.
#include <algorithm>
#include <vector>

#include "kernels.h"
#include "tmap.h"

namespace nsa {

namespace {

constexpr int kTabInts = 896;   // 3.5 KB of the 4 KB of kernel parameters
struct TabChunk {
  int v[kTabInts];
};

__global__ void upload_table_kernel(const __grid_constant__ TabChunk c, int* __restrict__ dst, const int n) {
  after_previous();
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = c.v[i];
}

// One 16-byte vector of ck and of cv per thread: compressed row r of the old cache belongs to the sequence whose
// cu_old covers it and keeps its distance from the sequence's first row.  Bound by HBM: 2 x (read + write) of the cache.
__global__ void __launch_bounds__(256) move_rows_kernel(const uint4* __restrict__ ck0, const uint4* __restrict__ cv0,
                                                        uint4* __restrict__ ck1, uint4* __restrict__ cv1,
                                                        const int* __restrict__ cu_old, const int* __restrict__ cu_new,
                                                        const int nseq, const int vec_per_row, const long long nvec) {
  after_previous();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= nvec) return;
  const uint4 a = __ldcs(ck0 + i), b = __ldcs(cv0 + i);
  const int r = (int)(i / vec_per_row);
  int lo = 0, hi = nseq - 1;   // the last sequence with cu_old[s] <= r (empty ones before it share that value)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_old[mid] <= r) lo = mid; else hi = mid - 1;
  }
  const long long j = i + (long long)(cu_new[lo] - cu_old[lo]) * vec_per_row;
  ck1[j] = a;
  cv1[j] = b;
}

// Conv1d weight [o][c][j] -> [j*D + c][o], both tensors.  Block = one input channel c: D x 32 tile through shared memory.
__global__ void __launch_bounds__(256) conv_weight_kernel(const bf16* __restrict__ w0, const bf16* __restrict__ w1,
                                                          bf16* __restrict__ o0, bf16* __restrict__ o1, const int D, const int l) {
  after_previous();
  __shared__ bf16 t[32][130];
  const bf16* w = blockIdx.y ? w1 : w0;
  bf16* out = blockIdx.y ? o1 : o0;
  const int c = blockIdx.x;
  for (int j0 = 0; j0 < l; j0 += 32) {
    const int nj = min(32, l - j0);
    for (int e = threadIdx.x; e < D * 32; e += 256) {
      const int o = e >> 5, j = e & 31;
      if (j < nj) t[j][o] = w[((long long)o * D + c) * l + j0 + j];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nj * (D / 2); e += 256) {
      const int j = e / (D / 2), o = (e % (D / 2)) * 2;
      *reinterpret_cast<__nv_bfloat162*>(out + ((long long)(j0 + j) * D + c) * D + o) =
          *reinterpret_cast<const __nv_bfloat162*>(&t[j][o]);
    }
    __syncthreads();
  }
}

}  // namespace

int launch_upload_table(const int* host, int n, int* dst, cudaStream_t s) {
  for (int i = 0; i < n; i += kTabInts) {
    TabChunk c;
    const int m = std::min(kTabInts, n - i);
    std::copy(host + i, host + i + m, c.v);
    launch_next(upload_table_kernel, 1, 256, 0, s, c, dst + i, m);
    note_launches(1);
  }
  return (int)cudaGetLastError();
}

int launch_move_rows(const bf16* ck0, const bf16* cv0, bf16* ck1, bf16* cv1, const int* cu_old, const int* cu_new, int nseq,
                     long long rows, int row_elems, cudaStream_t s) {
  if (rows <= 0) return 0;
  const int vpr = row_elems / 8;
  const long long nvec = rows * vpr;
  launch_next(move_rows_kernel, (unsigned)((nvec + 255) / 256), 256, 0, s, (const uint4*)ck0, (const uint4*)cv0, (uint4*)ck1, (uint4*)cv1,
                                                                 cu_old, cu_new, nseq, vpr, nvec);
  note_launches(1);
  return (int)cudaGetLastError();
}

int launch_conv_weight(const bf16* w0, const bf16* w1, bf16* o0, bf16* o1, int D, int l, cudaStream_t s) {
  if (D > 128 || (D & 1)) {
    set_error("head_dim %d not supported (64 or 128)", D);
    return -2;
  }
  launch_next(conv_weight_kernel, dim3((unsigned)D, w1 ? 2 : 1), 256, 0, s, w0, w1, o0, o1, D, l);
  note_launches(1);
  return (int)cudaGetLastError();
}

// Length tables of a cache that grows from (cu_old, cuc_old) to cu_new, all [nseq+1] host tables of cumulative lengths:
//   table = [ cu_new (n+1) | new compressed offsets (n+1) | old compressed offsets (n+1) | offsets of the rows to compute
//             (n+1) | first position to compute (n) | sequences, longest first (n) ]
//   info  = { compressed rows in all, longest compressed sequence, rows to compute }
// With cu_old = null everything is new.  Returns 0, s + 1 if sequence s became shorter, or -(s + 1) if more of its positions
// are in
// the old cache than it has (that cache was built with another block or stride).
int cache_plan(const int* cu_new, const int* cu_old, const int* cuc_old, int nseq, int block, int stride, int* table, int* info) {
  const int n = nseq;
  int* t_cu = table;
  int* t_cc = t_cu + n + 1;
  int* t_old = t_cc + n + 1;
  int* t_row = t_old + n + 1;
  int* t_first = t_row + n + 1;
  int* t_order = t_first + n;
  int max_tc = 0;
  t_cu[0] = cu_new[0];
  t_cc[0] = t_old[0] = t_row[0] = 0;
  for (int i = 0; i < n; ++i) {
    const int len = cu_new[i + 1] - cu_new[i];
    if (cu_old && len < cu_old[i + 1] - cu_old[i]) return i + 1;
    const int tc = len >= block ? (len - block) / stride + 1 : 0;
    const int old = cuc_old ? cuc_old[i + 1] - cuc_old[i] : 0;
    if (old < 0 || old > tc) return -(i + 1);
    t_cu[i + 1] = cu_new[i + 1];
    t_cc[i + 1] = t_cc[i] + tc;
    t_old[i + 1] = t_old[i] + old;
    t_row[i + 1] = t_row[i] + tc - old;
    t_first[i] = old;
    t_order[i] = i;
    max_tc = std::max(max_tc, tc);
  }
  std::stable_sort(t_order, t_order + n, [&](int a, int b) { return cu_new[a + 1] - cu_new[a] > cu_new[b + 1] - cu_new[b]; });
  info[0] = t_cc[n];
  info[1] = max_tc;
  info[2] = t_row[n];
  return 0;
}

}  // namespace nsa
