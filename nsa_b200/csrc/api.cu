// The C ABI of libnsa_b200.so (declared in include/nsa_b200.h): argument checks, workspace carving and kernel
// launches.  No torch types, no allocation, no synchronisation except nsa_device_status().
#include <stdarg.h>
#include <stdio.h>

#include <algorithm>

#include "../../include/nsa_b200.h"
#include "kernels.h"
#include "tmap.h"

namespace nsa {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

static int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static int check_attn_shape(const char* who, int B, int T, int Hq, int Hk, int D) {
  if (B <= 0 || T <= 0 || Hq <= 0 || Hk <= 0) return fail(-1, "%s: empty or negative shape", who);
  if (D != 64 && D != 128) return fail(-2, "%s: head_dim %d not supported (64 or 128)", who, D);
  if (Hq % Hk != 0 || (Hq / Hk) % 16 != 0)
    return fail(-3, "%s: query heads per KV head must be a multiple of 16 (Hq=%d, Hkv=%d)", who, Hq, Hk);
  return 0;
}

static int check_bs(const char* who, int BS) {
  if (BS != 16 && BS != 32 && BS != 64) return fail(-9, "%s: selection block size %d not supported (16, 32, 64)", who, BS);
  return 0;
}

// Shares of a key block's token stream in the key-major backward of the selected branch.  The first blocks are visited
// most: one CTA per block is enough only when there are six blocks per SM; with fewer a list is shared by two CTAs, or by as
// many as
// give every SM two (at most 16; a share then still has some dozens of tokens).  The CTAs of a shared list leave fp32
// partials that a
// second kernel adds in order.  kv_bwd_tc_kernel with 4 KV heads, one CTA a block -> two: 5008 tokens (316 blocks) 498 -> 282
// us + 24
// for the sums, 9008 tokens (564) 711 -> 531 + 23, 14000 tokens (876) 1049 -> 848 + 34, 17008 tokens (1064) 1050 -> 1031 +
// 41, so not
// there; 2 x 2080 tokens, 2 KV heads (132) three shares 126 us, two 144, four 130, five 135.
static int kv_shares(long long blocks) {
  if (blocks <= 0 || blocks >= 6LL * num_sms()) return 1;
  return (int)std::min(16LL, std::max(2LL, (2LL * num_sms() + blocks - 1) / blocks));
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace nsa

using namespace nsa;

extern "C" {

int nsa_abi_version(void) { return 1; }

long long nsa_kernel_launch_count(void) { return launch_count(); }

const char* nsa_last_error(void) { return g_err; }

int nsa_device_status(void) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return fail(1000 + (int)e, "cudaDeviceSynchronize: %s", cudaGetErrorString(e));
  int worst = 0, v = 0;
  int (*fns[])(int*) = {sel_status, sel_block_status, dense_status, kv_status, compress_status, misc_status, compress_tc_status, compress_bwd_tc_status, kv_tc_status, dense_kv_tc_status, dense_dq_tc_status, gather_probe_status, dense_tc2_status, score_tc_status, decode_status, sel_fwd_kv_status};
  for (auto f : fns) {
    v = 0;
    const int rc = f(&v);
    if (rc) return fail(1000 + rc, "reading the device status failed: %s", cudaGetErrorString((cudaError_t)rc));
    if (v && !worst) worst = v;
  }
  if (worst) fail(worst, "a kernel gave up waiting on its pipeline (code %d)", worst);
  return worst;
}

int nsa_pool_out_len(int n, int k, int s, int p) {
  if (n <= 0 || k <= 0 || s <= 0) return 0;
  const int num = n + 2 * p - k;
  int out = (num >= 0 ? (num + s - 1) / s : -((-num) / s)) + 1;
  if ((out - 1) * s >= n + p) --out;
  return out < 0 ? 0 : out;
}

// ---- compression ------------------------------------------------------------------------------------
int nsa_compress_fwd(const void* x, const void* w, const void* bias, void* y, const int32_t* cu_in,
                     const int32_t* cu_out, int nseq, int H, int D, int block, int stride, int max_out,
                     void* stream) {
  if (!x || !w || !y || !cu_in || !cu_out) return fail(-1, "nsa_compress_fwd: null pointer");
  if (nseq <= 0 || H <= 0) return fail(-1, "nsa_compress_fwd: empty shape");
  if (stride <= 0 || block <= 0 || block % stride) return fail(-4, "nsa_compress_fwd: block must be a multiple of stride");
  if (!aligned16(x) || !aligned16(w) || !aligned16(y)) return fail(-5, "nsa_compress_fwd: pointers must be 16-byte aligned");
  CompressArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.bias = (const bf16*)bias; a.y = (bf16*)y;
  a.cu_in = cu_in; a.cu_out = cu_out; a.nseq = nseq; a.H = H; a.D = D; a.l = block; a.d = stride; a.max_out = max_out;
  return launch_compress_fwd(a, (cudaStream_t)stream);
}

int nsa_compress_fwd_uniform(const void* x, const void* w, const void* bias, void* y, int B, int T, int H, int D,
                             int block, int stride, void* stream) {
  if (!x || !w || !y) return fail(-1, "nsa_compress_fwd_uniform: null pointer");
  if (B <= 0 || H <= 0) return fail(-1, "nsa_compress_fwd_uniform: empty shape");
  if (stride <= 0 || block <= 0 || block % stride) return fail(-4, "nsa_compress_fwd_uniform: block must be a multiple of stride");
  if (T < block || T % stride) return fail(-10, "nsa_compress_fwd_uniform: T must be a multiple of stride and at least block");
  if (!aligned16(x) || !aligned16(w) || !aligned16(y)) return fail(-5, "nsa_compress_fwd_uniform: pointers must be 16-byte aligned");
  CompressFwdArgs a = {};
  a.x[0] = (const bf16*)x; a.w[0] = (const bf16*)w; a.bias[0] = (const bf16*)bias; a.y[0] = (bf16*)y; a.ntensor = 1;
  a.nseq = B; a.T = T; a.Tc = (T - block) / stride + 1; a.total_in = (long long)B * T;
  a.H = H; a.D = D; a.l = block; a.d = stride;
  return launch_compress_fwd_tc(a, (cudaStream_t)stream);
}

int nsa_compress_fwd_kv(const void* k, const void* v, const void* w_k, const void* w_v, const void* bias_k,
                        const void* bias_v, void* ck, void* cv, const int32_t* cu_in, const int32_t* cu_out, int nseq, int T,
                        int Tc, long long total_in, long long total_out, int H, int D, int block, int stride, int split,
                        void* stream) {
  if (!k || !v || !w_k || !w_v || !ck || !cv) return fail(-1, "nsa_compress_fwd_kv: null pointer");
  if (nseq <= 0 || H <= 0 || total_in < 0) return fail(-1, "nsa_compress_fwd_kv: empty shape");
  if (stride <= 0 || block <= 0 || block % stride) return fail(-4, "nsa_compress_fwd_kv: block must be a multiple of stride");
  if (!aligned16(k) || !aligned16(v) || !aligned16(w_k) || !aligned16(w_v) || !aligned16(ck) || !aligned16(cv))
    return fail(-5, "nsa_compress_fwd_kv: pointers must be 16-byte aligned");
  if (!cu_in != !cu_out) return fail(-1, "nsa_compress_fwd_kv: cu_in and cu_out must be given together");
  if (!cu_in && (total_in != (long long)nseq * T || (Tc > 0 && T < block + (Tc - 1) * stride)))
    return fail(-10, "nsa_compress_fwd_kv: %d sequences of %d tokens do not hold %d positions each", nseq, T, Tc);
  if (cu_in && total_out > 0 && total_in < block) return fail(-10, "nsa_compress_fwd_kv: fewer tokens than one block");
  CompressFwdArgs a = {};
  a.x[0] = (const bf16*)k; a.w[0] = (const bf16*)w_k; a.bias[0] = (const bf16*)bias_k; a.y[0] = (bf16*)ck;
  a.x[1] = (const bf16*)v; a.w[1] = (const bf16*)w_v; a.bias[1] = (const bf16*)bias_v; a.y[1] = (bf16*)cv;
  a.ntensor = 2; a.cu_in = cu_in; a.cu_out = cu_out; a.cu_row = cu_out; a.rows = total_out; a.split = split;
  a.nseq = nseq; a.T = T; a.Tc = Tc; a.total_in = total_in; a.H = H; a.D = D; a.l = block; a.d = stride;
  return launch_compress_fwd_tc(a, (cudaStream_t)stream);
}

int nsa_upload_table(const int32_t* host, int n, int32_t* dev, void* stream) {
  if (n > 0 && (!host || !dev)) return fail(-1, "nsa_upload_table: null pointer");
  return launch_upload_table(host, n, dev, (cudaStream_t)stream);
}

int nsa_conv_weight_layout(const void* w_k, const void* w_v, void* out_k, void* out_v, int D, int block, void* stream) {
  if (!w_k || !out_k || (!w_v != !out_v)) return fail(-1, "nsa_conv_weight_layout: null pointer");
  if (D != 64 && D != 128) return fail(-2, "nsa_conv_weight_layout: head_dim %d not supported (64 or 128)", D);
  if (block <= 0) return fail(-1, "nsa_conv_weight_layout: empty shape");
  return launch_conv_weight((const bf16*)w_k, (const bf16*)w_v, (bf16*)out_k, (bf16*)out_v, D, block, (cudaStream_t)stream);
}

int nsa_cache_plan(const int32_t* cu_new, const int32_t* cu_old, const int32_t* cuc_old, int nseq, int block, int stride,
                   int32_t* table, int32_t* info) {
  if (!cu_new || !table || !info || (!cu_old != !cuc_old)) return fail(-1, "nsa_cache_plan: null pointer");
  if (nseq < 0 || block <= 0 || stride <= 0) return fail(-1, "nsa_cache_plan: empty or negative shape");
  const int rc = cache_plan(cu_new, cu_old, cuc_old, nseq, block, stride, table, info);
  if (rc < 0) return fail(-18, "the old cache holds more positions of sequence %d than it has now: another block or stride", -rc - 1);
  return rc ? fail(-17, "sequence %d became shorter", rc - 1) : 0;
}

int nsa_cache_build(const void* k, const void* v, const void* conv_k, const void* conv_v, const void* bias_k,
                    const void* bias_v, void* w_ws, const void* ck_old, const void* cv_old, void* ck, void* cv,
                    const int32_t* table, int32_t* table_dev, int nseq, long long total_in, int H, int D, int block, int stride,
                    void* stream) {
  if (!table || !table_dev) return fail(-1, "nsa_cache_build: null pointer");
  if (nseq < 0 || H <= 0) return fail(-1, "nsa_cache_build: empty shape");
  if (D != 64 && D != 128) return fail(-2, "nsa_cache_build: head_dim %d not supported (64 or 128)", D);
  if (block % stride) return fail(-4, "nsa_cache_build: block must be a multiple of stride");
  if (!aligned16(k) || !aligned16(v) || !aligned16(w_ws) || !aligned16(ck) || !aligned16(cv) || !aligned16(ck_old) || !aligned16(cv_old))
    return fail(-5, "nsa_cache_build: pointers must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int n = nseq;
  const int32_t* cu = table_dev;
  const int32_t* cc = cu + n + 1;
  const int32_t* old = cc + n + 1;
  const int32_t* row = old + n + 1;
  const int32_t* first = row + n + 1;
  const long long nold = table[2 * (n + 1) + n], nnew = table[3 * (n + 1) + n];
  if (table[n] > total_in) return fail(-10, "nsa_cache_build: the sequences end at token %d of %lld", table[n], total_in);
  // (an empty tensor has no address: the caches before a sequence has reached its first block, and what no position is made from)
  if ((nold > 0 && (!ck_old || !cv_old)) || (nold + nnew > 0 && (!ck || !cv)) ||
      (nnew > 0 && (!k || !v || !conv_k || !conv_v || !w_ws)))
    return fail(-1, "nsa_cache_build: null pointer");
  int rc = launch_upload_table(table, 6 * n + 4, table_dev, s);
  if (!rc) rc = launch_move_rows((const bf16*)ck_old, (const bf16*)cv_old, (bf16*)ck, (bf16*)cv, old, cc, n, nold, H * D, s);
  if (rc || nnew <= 0) return rc;
  bf16* wk = (bf16*)w_ws;
  bf16* wv = wk + (size_t)block * D * D;
  rc = launch_conv_weight((const bf16*)conv_k, (const bf16*)conv_v, wk, wv, D, block, s);
  if (rc) return rc;
  CompressFwdArgs a = {};
  a.x[0] = (const bf16*)k; a.w[0] = wk; a.bias[0] = (const bf16*)bias_k; a.y[0] = (bf16*)ck;
  a.x[1] = (const bf16*)v; a.w[1] = wv; a.bias[1] = (const bf16*)bias_v; a.y[1] = (bf16*)cv;
  a.ntensor = 2; a.cu_in = cu; a.cu_out = cc; a.cu_row = row; a.first = first; a.rows = nnew; a.split = 0;
  a.nseq = n; a.total_in = total_in; a.H = H; a.D = D; a.l = block; a.d = stride;
  return launch_compress_fwd_tc(a, s);
}

size_t nsa_compress_bwd_workspace_bytes(int nseq, int H, int D, int block) {
  long long split = (long long)nseq * H;
  if (split > 32) split = 32;
  return (size_t)split * block * D * D * sizeof(float);
}

int nsa_compress_bwd(const void* x, const void* w, const void* dy, void* dx, float* dw, float* dbias, void* ws,
                     size_t ws_bytes, const int32_t* cu_in, const int32_t* cu_out, int nseq, int H, int D, int block,
                     int stride, int max_in, int total_out, void* stream) {
  if (!x || !w || !dy || !cu_in || !cu_out) return fail(-1, "nsa_compress_bwd: null pointer");
  if (nseq <= 0 || H <= 0) return fail(-1, "nsa_compress_bwd: empty shape");
  if (D != 64 && D != 128) return fail(-2, "nsa_compress_bwd: head_dim %d not supported (64 or 128)", D);
  if (stride <= 0 || block <= 0 || block % stride) return fail(-4, "nsa_compress_bwd: block must be a multiple of stride");
  if (dw && (!ws || ws_bytes < nsa_compress_bwd_workspace_bytes(nseq, H, D, block)))
    return fail(-6, "nsa_compress_bwd: workspace too small");
  CompressArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.dy = (const bf16*)dy; a.dx = (bf16*)dx; a.dw = dw; a.dbias = dbias;
  a.ws = (float*)ws; a.cu_in = cu_in; a.cu_out = cu_out; a.nseq = nseq; a.H = H; a.D = D; a.l = block; a.d = stride;
  a.max_in = max_in; a.total_out = total_out;
  return launch_compress_bwd(a, (cudaStream_t)stream);
}

size_t nsa_compress_bwd_kv_workspace_bytes(int nseq, int Tc, long long total_out, int ragged, int H, int D, int block,
                                           int stride) {
  if (block <= 0 || stride <= 0 || H <= 0 || !compress_bwd_tc_supported(D, block, stride)) return 0;
  return compress_bwd_tc_workspace_bytes(nseq, Tc, total_out, ragged != 0, H, D, block);
}

int nsa_compress_bwd_kv(const void* k, const void* v, const void* w_k, const void* w_v, const void* dck, const void* dcv,
                        void* dk, void* dv, int accumulate, void* dw_k, void* dw_v, void* dbias_k, void* dbias_v, int dw_mode,
                        void* ws, size_t ws_bytes, const int32_t* cu_in, const int32_t* cu_out, int nseq, int T, int Tc,
                        long long total_in, long long total_out, int H, int D, int block, int stride, void* stream) {
  if (!k || !v || !w_k || !w_v || !dck || !dcv) return fail(-1, "nsa_compress_bwd_kv: null pointer");
  if (nseq <= 0 || H <= 0 || total_in <= 0 || total_out <= 0) return fail(-1, "nsa_compress_bwd_kv: empty shape");
  if (D != 64 && D != 128) return fail(-2, "nsa_compress_bwd_kv: head_dim %d not supported (64 or 128)", D);
  if (stride <= 0 || block <= 0 || !compress_bwd_tc_supported(D, block, stride))
    return fail(-4, "nsa_compress_bwd_kv: block must be stride or 2 * stride (got %d, %d); use nsa_compress_bwd", block, stride);
  if (dw_mode < 0 || dw_mode > 2) return fail(-16, "nsa_compress_bwd_kv: dw_mode must be 0, 1 or 2");
  if (!cu_in != !cu_out) return fail(-1, "nsa_compress_bwd_kv: cu_in and cu_out must be given together");
  if (!cu_in && (total_in != (long long)nseq * T || total_out != (long long)nseq * Tc || T < block + (Tc - 1) * stride))
    return fail(-10, "nsa_compress_bwd_kv: %d sequences of %d tokens do not hold %d positions each", nseq, T, Tc);
  if ((dw_k || dw_v || dbias_k || dbias_v) &&
      (!ws || ws_bytes < nsa_compress_bwd_kv_workspace_bytes(nseq, Tc, total_out, cu_in != nullptr, H, D, block, stride)))
    return fail(-6, "nsa_compress_bwd_kv: workspace too small");
  CompressBwdArgs a = {};
  a.x[0] = (const bf16*)k; a.w[0] = (const bf16*)w_k; a.dy[0] = (const bf16*)dck; a.dx[0] = (bf16*)dk; a.dw[0] = dw_k; a.dbias[0] = dbias_k;
  a.x[1] = (const bf16*)v; a.w[1] = (const bf16*)w_v; a.dy[1] = (const bf16*)dcv; a.dx[1] = (bf16*)dv; a.dw[1] = dw_v; a.dbias[1] = dbias_v;
  a.accumulate = accumulate; a.mode = dw_mode; a.ws = (float*)ws; a.cu_in = cu_in; a.cu_out = cu_out;
  a.nseq = nseq; a.T = T; a.Tc = Tc; a.total_in = total_in; a.total_out = total_out; a.H = H; a.D = D; a.l = block; a.d = stride;
  return launch_compress_bwd_tc(a, (cudaStream_t)stream);
}

int nsa_compress_bwd_noalloc(const void* x, const void* w, const void* dy, void* dx, float* dw, float* dbias,
                             const int32_t* cu_in, const int32_t* cu_out, int nseq, int H, int D, int block, int stride,
                             int max_in, int total_out, void* stream) {
  if (!x || !w || !dy || !cu_in || !cu_out) return fail(-1, "nsa_compress_bwd_noalloc: null pointer");
  if (nseq <= 0 || H <= 0) return fail(-1, "nsa_compress_bwd_noalloc: empty shape");
  if (D != 64 && D != 128) return fail(-2, "nsa_compress_bwd_noalloc: head_dim %d not supported (64 or 128)", D);
  if (stride <= 0 || block <= 0 || block % stride)
    return fail(-4, "nsa_compress_bwd_noalloc: block must be a multiple of stride");
  if (dw && (long long)block * D * D > compress_static_scratch_floats())
    return fail(-41, "nsa_compress_bwd_noalloc: block*D*D = %lld floats exceeds the built-in scratch of %lld floats; "
                     "use nsa_compress_bwd with a caller workspace", (long long)block * D * D,
                compress_static_scratch_floats());
  CompressArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.dy = (const bf16*)dy; a.dx = (bf16*)dx; a.dw = dw; a.dbias = dbias;
  a.cu_in = cu_in; a.cu_out = cu_out; a.nseq = nseq; a.H = H; a.D = D; a.l = block; a.d = stride;
  a.max_in = max_in; a.total_out = total_out;
  return launch_compress_bwd_static(a, (cudaStream_t)stream);
}

// ---- compressed attention ---------------------------------------------------------------------------
struct GateArgs {   // optional gate projection fused into the compressed-attention forward
  const void *w, *b;
  void* g[3];
};

static int cmp_attn_fwd_impl(const void* q, const void* ck, const void* cv, void* o, float* lse, int32_t* sel_idx,
                     float* sel_scores, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, int n_sel, int pool_k, int pool_s, int pool_p, int Tq, int q0, void* stream,
                     const GateArgs* gate = nullptr, int score_mode = 0) {
  const bool sharded = (Tq != T) || (q0 != 0);
  if (Tq <= 0 || q0 < 0 || q0 + Tq > T) return fail(-12, "%s: query shard [%d, %d) is outside the sequence of %d tokens", "nsa_cmp_attn_fwd", q0, q0 + Tq, T);
  (void)sharded;
  if (!q || !ck || !cv || !o || !lse) return fail(-1, "nsa_cmp_attn_fwd: null pointer");
  int rc = check_attn_shape("nsa_cmp_attn_fwd", B, T, Hq, Hk, D);
  if (rc) return rc;
  if (Tc <= 0) return fail(-1, "nsa_cmp_attn_fwd: no compressed positions (sequence shorter than one block)");
  DenseArgs a = {};
  a.mode = 1; a.q = (const bf16*)q; a.k = (const bf16*)ck; a.v = (const bf16*)cv; a.o = (bf16*)o; a.lse = lse;
  a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Lk = Tc; a.Hq = Hq; a.Hk = Hk; a.cblock = block; a.cstride = stride; a.causal = causal;
  a.scale = scale; a.n_sel = n_sel; a.score_mode = score_mode;
  if (score_mode != 0 && score_mode != 1) return fail(-16, "nsa_cmp_attn_fwd: score_mode must be 0 (reference) or 1 (causal)");
  if (score_mode == 1 && !causal) return fail(-16, "nsa_cmp_attn_fwd: causal selection scores need causal = 1");
  if (n_sel > 0) {
    if (!sel_idx) return fail(-1, "nsa_cmp_attn_fwd: sel_idx is null");
    if (Hq / Hk != 16)
      return fail(-7, "nsa_cmp_attn_fwd: block selection needs exactly 16 query heads per KV head (got %d)", Hq / Hk);
    if (pool_k <= 0 || pool_s <= 0 || pool_p < 0) return fail(-8, "nsa_cmp_attn_fwd: bad pooling parameters");
    a.pool_k = pool_k; a.pool_s = pool_s; a.pool_p = pool_p;
    a.n_pool = nsa_pool_out_len(Tc, pool_k, pool_s, pool_p);
    a.sel_idx = sel_idx; a.sel_scores = sel_scores;
  }
  if (dense_fwd_tc_supported(a, D)) {
    if (n_sel > 0) {   // the selection has its own kernel
      ScoreArgs c = {};
      c.q = a.q; c.ck = a.k; c.sel_idx = sel_idx; c.sel_scores = sel_scores;
      c.seq.B = B; c.seq.Tq = Tq; c.seq.q0 = q0; c.seq.Tc = Tc;
      c.Hq = Hq; c.Hk = Hk; c.n_sel = n_sel; c.Tc_max = Tc; c.score_mode = score_mode; c.cblock = block;
      c.cstride = stride; c.scale = scale;
      rc = launch_score_tc(c, (cudaStream_t)stream);
      if (rc) return rc;
      a.n_sel = 0;
    }
    if (gate) {
      a.gate_w = (const bf16*)gate->w; a.gate_b = (const bf16*)gate->b;
      for (int i = 0; i < 3; ++i) a.g_out[i] = (bf16*)gate->g[i];
    }
    return launch_dense_fwd2_tc(a, D, (cudaStream_t)stream);
  }
  if (sharded) return fail(-11, "query shards need head_dim 128 and the default pooling geometry");
  if (score_mode == 1 && n_sel > 0) return fail(-16, "causal selection scores need head_dim 128 and the default pooling geometry");
  rc = launch_dense_fwd(a, D, (cudaStream_t)stream);
  if (rc || !gate) return rc;
  return launch_gate_fwd((const bf16*)q, (const bf16*)gate->w, (const bf16*)gate->b, (bf16*)gate->g[0], (bf16*)gate->g[1],
                         (bf16*)gate->g[2], (long long)B * Tq * Hq, D, (cudaStream_t)stream);
}

int nsa_cmp_attn_fwd(const void* q, const void* ck, const void* cv, void* o, float* lse, int32_t* sel_idx,
                     float* sel_scores, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, int n_sel, int pool_k, int pool_s, int pool_p, void* stream) {
  return cmp_attn_fwd_impl(q, ck, cv, o, lse, sel_idx, sel_scores, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, n_sel, pool_k, pool_s, pool_p, T, 0, stream);
}

int nsa_cmp_attn_fwd_sharded(const void* q, const void* ck, const void* cv, void* o, float* lse, int32_t* sel_idx,
                     float* sel_scores, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, int n_sel, int pool_k, int pool_s, int pool_p, int Tq, int q0, void* stream) {
  return cmp_attn_fwd_impl(q, ck, cv, o, lse, sel_idx, sel_scores, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, n_sel, pool_k, pool_s, pool_p, Tq, q0, stream);
}

int nsa_cmp_attn_fwd_gated(const void* q, const void* ck, const void* cv, void* o, float* lse, int32_t* sel_idx,
                           float* sel_scores, const void* gate_w, const void* gate_b, void* g_slc, void* g_swa, void* g_cmp,
                           int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal, float scale,
                           int n_sel, int pool_k, int pool_s, int pool_p, int score_mode, int Tq, int q0, void* stream) {
  if (gate_w && (!g_slc || !g_swa || !g_cmp)) return fail(-1, "nsa_cmp_attn_fwd_gated: null gate output");
  const GateArgs g = {gate_w, gate_b, {g_slc, g_swa, g_cmp}};
  return cmp_attn_fwd_impl(q, ck, cv, o, lse, sel_idx, sel_scores, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, n_sel, pool_k, pool_s, pool_p, Tq, q0, stream, gate_w ? &g : nullptr, score_mode);
}

size_t nsa_cmp_attn_bwd_workspace_bytes(int B, int T, int Tc, int Hk, int D) {
  if (T <= 0) return 0;
  const int rows = dense_kv_segment_rows(B, T, Tc, Hk);
  return (size_t)2 * ((T + rows - 1) / rows) * B * Tc * Hk * D * sizeof(float);
}

// dCK, dCV: one launch over segments of the queries and the sum of their fp32 slabs (the workspace), or straight to bf16 when
// one segment does.
static int cmp_dkv(const void* q, const void* ck, const void* cv, const float* lse, const void* dout, const float* delta,
                   const void* gate, void* dck, void* dcv, void* ws, int B, int T, int Tc, int Hq, int Hk, int D, int block,
                   int stride, int causal, float scale, int Tq, int q0, cudaStream_t s) {
  DenseKvArgs a = {};
  a.mode = 1; a.q = (const bf16*)q; a.k = (const bf16*)ck; a.v = (const bf16*)cv; a.dout = (const bf16*)dout;
  a.lse = lse; a.delta = delta; a.gate = (const bf16*)gate; a.dk = (bf16*)dck; a.dv = (bf16*)dcv;
  a.seg_len = dense_kv_segment_rows(B, T, Tc, Hk);
  a.nslab = a.slabs = (Tq + a.seg_len - 1) / a.seg_len;
  a.part = a.nslab > 1 ? (float*)ws : nullptr;
  a.Hq = Hq; a.Hk = Hk; a.Lk = Tc; a.cblock = block; a.cstride = stride; a.causal = causal; a.scale = scale;
  a.seq.B = B; a.seq.Tq = Tq; a.seq.q0 = q0; a.seq.Tc = Tc;
  return launch_dense_kv_tc(a, D, s);
}

struct PreCmp {   // row pre-pass folded into the compressed branch's dQ kernel
  const void* o_cmp;
  void* dg_cmp;
};

static int cmp_attn_bwd_impl(const void* q, const void* ck, const void* cv, const float* lse, const void* dout,
                     const float* delta, const void* gate, void* dq, int accumulate_dq, void* dck, void* dcv, void* ws,
                     size_t ws_bytes, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, int Tq, int q0, void* stream, const PreCmp* pre = nullptr) {
  const bool sharded = (Tq != T) || (q0 != 0);
  if (Tq <= 0 || q0 < 0 || q0 + Tq > T) return fail(-12, "%s: query shard [%d, %d) is outside the sequence of %d tokens", "nsa_cmp_attn_bwd", q0, q0 + Tq, T);
  (void)sharded;
  if (!q || !ck || !cv || !lse || !dout || !delta) return fail(-1, "nsa_cmp_attn_bwd: null pointer");
  int rc = check_attn_shape("nsa_cmp_attn_bwd", B, T, Hq, Hk, D);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  bool fold = false;
  if (pre) {
    if (!pre->o_cmp) return fail(-1, "nsa_cmp_attn_bwd_fused: o_cmp is null");
    fold = dq && D == 128;
    if (!fold) {   // no tcgen05 dQ kernel to carry the pre-pass: run it on its own
      rc = launch_rowdot((const bf16*)pre->o_cmp, (const bf16*)dout, (const bf16*)gate, const_cast<float*>(delta),
                         (bf16*)pre->dg_cmp, (long long)B * Tq * Hq, D, s);
      if (rc) return rc;
    }
  }
  if (dq) {
    DenseArgs a = {};
    if (fold) {
      a.pre_o[0] = (const bf16*)pre->o_cmp; a.pre_gate[0] = (const bf16*)gate; a.pre_delta[0] = const_cast<float*>(delta);
      a.pre_dgate[0] = (bf16*)pre->dg_cmp;
    }
    a.mode = 1; a.q = (const bf16*)q; a.k = (const bf16*)ck; a.v = (const bf16*)cv; a.lse = const_cast<float*>(lse);
    a.dout = (const bf16*)dout; a.delta = delta; a.gate = (const bf16*)gate; a.dq = (bf16*)dq;
    a.accumulate = accumulate_dq; a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Lk = Tc; a.Hq = Hq; a.Hk = Hk; a.cblock = block;
    a.cstride = stride; a.causal = causal; a.scale = scale;
    if (D != 128 && sharded) return fail(-11, "query shards need head_dim 128");
    rc = launch_dense_dq_tc(a, D, s);
    if (rc) return rc;
  }
  if (dck || dcv) {
    if (!dck || !dcv) return fail(-1, "nsa_cmp_attn_bwd: dck and dcv must be given together");
    if (!ws || ws_bytes < nsa_cmp_attn_bwd_workspace_bytes(B, T, Tc, Hk, D))
      return fail(-6, "nsa_cmp_attn_bwd: workspace too small");
    if (D != 128 && sharded) return fail(-11, "query shards need head_dim 128");
    rc = cmp_dkv(q, ck, cv, lse, dout, delta, gate, dck, dcv, ws, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, Tq, q0, s);
    if (rc) return rc;
  }
  return 0;
}

int nsa_cmp_attn_bwd(const void* q, const void* ck, const void* cv, const float* lse, const void* dout,
                     const float* delta, const void* gate, void* dq, int accumulate_dq, void* dck, void* dcv, void* ws,
                     size_t ws_bytes, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, void* stream) {
  return cmp_attn_bwd_impl(q, ck, cv, lse, dout, delta, gate, dq, accumulate_dq, dck, dcv, ws, ws_bytes, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, T, 0, stream);
}

int nsa_cmp_attn_bwd_sharded(const void* q, const void* ck, const void* cv, const float* lse, const void* dout,
                     const float* delta, const void* gate, void* dq, int accumulate_dq, void* dck, void* dcv, void* ws,
                     size_t ws_bytes, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride, int causal,
                     float scale, int Tq, int q0, void* stream) {
  return cmp_attn_bwd_impl(q, ck, cv, lse, dout, delta, gate, dq, accumulate_dq, dck, dcv, ws, ws_bytes, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, Tq, q0, stream);
}

// ---- selected + sliding window ----------------------------------------------------------------------

// The reverse index of a selection in one buffer: histogram, CSR offsets, token lists, and its inverse.  Returns the bytes.
static size_t rev_layout(void* base, const void* idx, int idx64, const int32_t* counts, int B, int T, int Tq, int q0, int Hkv,
                         int S, int BS, RevArgs* r) {
  const size_t NB = (size_t)(T + BS - 1) / BS, bh = (size_t)B * Hkv;
  size_t n[4] = {align_up(bh * NB * NB * 4, 256), align_up(bh * (NB + 1) * 4, 256), align_up(bh * (size_t)T * S * 4, 256),
                 align_up((size_t)B * Tq * Hkv * S * 4, 256)};
  if (r) {
    *r = {};
    r->idx = idx; r->idx64 = idx64; r->counts = counts; r->B = B; r->T = T; r->Tq = Tq; r->q0 = q0; r->H = Hkv; r->S = S;
    r->BS = BS; r->NB = (int)NB; r->cap = (long long)Tq * S;
    char* p = (char*)base;
    r->hist = (int*)p;
    r->rev_ptr = (int*)(p + n[0]);
    r->rev_tok = (int*)(p + n[0] + n[1]);
    r->inv = (int*)(p + n[0] + n[1] + n[2]);
  }
  return n[0] + n[1] + n[2] + n[3];
}

size_t nsa_sel_index_bytes(int B, int T, int Tq, int Hkv, int S, int BS) {
  return BS <= 0 ? 0 : rev_layout(nullptr, nullptr, 0, nullptr, B, T, Tq, 0, Hkv, S, BS, nullptr);
}

int nsa_sel_index(const void* idx, int idx64, const int32_t* counts, void* index, size_t index_bytes, int B, int T, int Tq,
                  int q0, int Hkv, int S, int BS, void* stream) {
  if (!idx || !index) return fail(-1, "nsa_sel_index: null pointer");
  if (B <= 0 || T <= 0 || Hkv <= 0 || S <= 0) return fail(-1, "nsa_sel_index: empty or negative shape");
  if (Tq <= 0 || q0 < 0 || q0 + Tq > T) return fail(-12, "nsa_sel_index: query shard [%d, %d) is outside the sequence of %d tokens", q0, q0 + Tq, T);
  const int rc = check_bs("nsa_sel_index", BS);
  if (rc) return rc;
  if (index_bytes < nsa_sel_index_bytes(B, T, Tq, Hkv, S, BS)) return fail(-6, "nsa_sel_index: buffer too small");
  RevArgs r;
  rev_layout(index, idx, idx64, counts, B, T, Tq, q0, Hkv, S, BS, &r);
  return launch_build_rev(r, (cudaStream_t)stream);
}

// Workspace of the key-major selected forward: the reverse index, one [16 x D] bf16 tile and 16 (max, sum) pairs per
// (list position, 16-head sub-group).
size_t nsa_sel_swa_fwd_ix_workspace_bytes(int B, int T, int Tq, int Hq, int Hkv, int D, int S, int BS) {
  if (BS <= 0 || Hkv <= 0) return 0;
  const size_t ent = (size_t)B * Tq * S * Hq;   // (list position, head) pairs
  return align_up(ent * D * 2, 256) + align_up(ent * 8, 256);
}

size_t nsa_sel_swa_fwd_workspace_bytes(int B, int T, int Tq, int Hq, int Hkv, int D, int S, int BS) {
  if (BS <= 0 || Hkv <= 0) return 0;
  return nsa_sel_index_bytes(B, T, Tq, Hkv, S, BS) + nsa_sel_swa_fwd_ix_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS);
}

static int sel_swa_fwd_impl(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    void* o_slc, float* lse_slc, void* o_swa, float* lse_swa, const void* g_slc, const void* g_swa,
                    const void* o_cmp, const void* g_cmp, void* o, int B, int T, int Hq, int Hkv, int D, int S, int BS,
                    int window, float scale, int Tq, int q0, void* stream, void* ws = nullptr, size_t ws_bytes = 0,
                    const void* index = nullptr) {
  const bool sharded = (Tq != T) || (q0 != 0);
  if (Tq <= 0 || q0 < 0 || q0 + Tq > T) return fail(-12, "%s: query shard [%d, %d) is outside the sequence of %d tokens", "nsa_sel_swa_fwd", q0, q0 + Tq, T);
  (void)sharded;
  if (!q || !k || !v) return fail(-1, "nsa_sel_swa_fwd: null pointer");
  int rc = check_attn_shape("nsa_sel_swa_fwd", B, T, Hq, Hkv, D);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if (window > 0) {   // first: the selected branch's merge adds it
    if (!o_swa || !lse_swa) return fail(-1, "nsa_sel_swa_fwd: o_swa / lse_swa is null");
    DenseArgs a = {};
    a.mode = 0; a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.o = (bf16*)o_swa; a.lse = lse_swa;
    a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Lk = T; a.Hq = Hq; a.Hk = Hkv; a.window = window; a.scale = scale;
    rc = launch_dense_fwd2_tc(a, D, s);
    if (rc) return rc;
  }
  const bf16* swa = window > 0 ? (const bf16*)o_swa : nullptr;
  if (o_slc || (o && index)) {   // (with an index of its own and a workspace a caller may leave out o_slc)
    if (!idx) return fail(-1, "nsa_sel_swa_fwd: idx is null");
    rc = check_bs("nsa_sel_swa_fwd", BS);
    if (rc) return rc;
    if (S <= 0) return fail(-1, "nsa_sel_swa_fwd: no selected blocks");
    SelKvArgs ka = {};
    ka.q = (const bf16*)q; ka.k = (const bf16*)k; ka.v = (const bf16*)v; ka.merge.o = (bf16*)o_slc; ka.merge.lse = lse_slc;
    ka.B = B; ka.T = T; ka.Tq = Tq; ka.q0 = q0; ka.Hq = Hq; ka.Hk = Hkv; ka.S = S; ka.BS = BS; ka.scale = scale;
    if (ws && sel_fwd_kv_supported(ka, D) &&
        ws_bytes >= (index ? nsa_sel_swa_fwd_ix_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS)
                           : nsa_sel_swa_fwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS))) {
      // key-major: reverse index, then one CTA per key block over the queries that selected it, then the per-token merge
      RevArgs r;
      const size_t nrev = rev_layout(index ? const_cast<void*>(index) : ws, idx, idx64, counts, B, T, Tq, q0, Hkv, S, BS, &r);
      char* p = (char*)ws + (index ? 0 : nrev);
      ka.part = (bf16*)p;
      ka.stats = (float*)(p + align_up((size_t)B * Tq * S * Hq * D * 2, 256));
      if (!index) {
        rc = launch_build_rev(r, s);
        if (rc) return rc;
      }
      ka.rev_ptr = r.rev_ptr; ka.rev_tok = r.rev_tok; ka.rev_cap = r.cap;
      ka.merge.g0 = (const bf16*)g_slc; ka.merge.a1 = swa; ka.merge.g1 = (const bf16*)g_swa; ka.merge.a2 = (const bf16*)o_cmp;
      ka.merge.g2 = (const bf16*)g_cmp; ka.merge.out = (bf16*)o;
      return launch_sel_fwd_kv(ka, r, s);
    }
    if (!o_slc || !lse_slc) return fail(-1, "nsa_sel_swa_fwd: o_slc / lse_slc is null");
    SelArgs a = {};
    a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.idx = idx; a.idx64 = idx64; a.counts = counts;
    a.o = (bf16*)o_slc; a.lse = lse_slc; a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Hq = Hq; a.Hkv = Hkv; a.S = S; a.BS = BS; a.scale = scale;
    rc = launch_sel_fwd(a, D, s);
    if (rc) return rc;
  }
  if (o) {
    rc = launch_combine((const bf16*)o_slc, (const bf16*)g_slc, swa, (const bf16*)g_swa, (const bf16*)o_cmp, (const bf16*)g_cmp,
                        (bf16*)o, (long long)B * Tq * Hq, D, s);
    if (rc) return rc;
  }
  return 0;
}

int nsa_sel_swa_fwd(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    void* o_slc, float* lse_slc, void* o_swa, float* lse_swa, const void* g_slc, const void* g_swa,
                    const void* o_cmp, const void* g_cmp, void* o, int B, int T, int Hq, int Hkv, int D, int S, int BS,
                    int window, float scale, void* stream) {
  return sel_swa_fwd_impl(q, k, v, idx, idx64, counts, o_slc, lse_slc, o_swa, lse_swa, g_slc, g_swa, o_cmp, g_cmp, o, B, T, Hq, Hkv, D, S, BS, window, scale, T, 0, stream);
}

int nsa_sel_swa_fwd_sharded(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    void* o_slc, float* lse_slc, void* o_swa, float* lse_swa, const void* g_slc, const void* g_swa,
                    const void* o_cmp, const void* g_cmp, void* o, int B, int T, int Hq, int Hkv, int D, int S, int BS,
                    int window, float scale, int Tq, int q0, void* stream) {
  return sel_swa_fwd_impl(q, k, v, idx, idx64, counts, o_slc, lse_slc, o_swa, lse_swa, g_slc, g_swa, o_cmp, g_cmp, o, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream);
}

int nsa_sel_swa_fwd_ws(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    void* o_slc, float* lse_slc, void* o_swa, float* lse_swa, const void* g_slc, const void* g_swa,
                    const void* o_cmp, const void* g_cmp, void* o, void* ws, size_t ws_bytes, int B, int T, int Hq, int Hkv,
                    int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream) {
  return sel_swa_fwd_impl(q, k, v, idx, idx64, counts, o_slc, lse_slc, o_swa, lse_swa, g_slc, g_swa, o_cmp, g_cmp, o, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream, ws, ws_bytes);
}

int nsa_sel_swa_fwd_ix(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                       const void* index, void* o_slc, float* lse_slc, void* o_swa, float* lse_swa, const void* g_slc,
                       const void* g_swa, const void* o_cmp, const void* g_cmp, void* o, void* ws, size_t ws_bytes, int B, int T,
                       int Hq, int Hkv, int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream) {
  return sel_swa_fwd_impl(q, k, v, idx, idx64, counts, o_slc, lse_slc, o_swa, lse_swa, g_slc, g_swa, o_cmp, g_cmp, o, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream, ws, ws_bytes, index);
}

int nsa_cmp_attn_bwd_fused(const void* q, const void* ck, const void* cv, const void* o_cmp, const float* lse, const void* dout,
                           float* delta, const void* gate, void* dgate, void* dq, int accumulate_dq, void* dck, void* dcv,
                           void* ws, size_t ws_bytes, int B, int T, int Tc, int Hq, int Hk, int D, int block, int stride,
                           int causal, float scale, int Tq, int q0, void* stream) {
  const PreCmp pre = {o_cmp, dgate};
  return cmp_attn_bwd_impl(q, ck, cv, lse, dout, delta, gate, dq, accumulate_dq, dck, dcv, ws, ws_bytes, B, T, Tc, Hq, Hk, D, block, stride, causal, scale, Tq, q0, stream, &pre);
}

// fp32 dK, dV of `slabs` slabs
static size_t kv_slab_bytes(int slabs, int B, int T, int Hkv, int D) { return (size_t)2 * slabs * B * T * Hkv * D * sizeof(float); }
static size_t rev_base_bytes(int B, int T, int Hkv, int S, int BS) {
  const size_t NB = (size_t)(T + BS - 1) / BS, bh = (size_t)B * Hkv;
  return align_up(bh * NB * NB * 4, 256) + align_up(bh * (NB + 1) * 4, 256) + align_up(bh * (size_t)T * S * 4, 256);
}

// The reverse index, then the window's dK, dV (fp32, sized for the larger head_dim).
size_t nsa_sel_swa_bwd_workspace_bytes(int B, int T, int Hkv, int S, int BS) {
  return BS <= 0 ? 0 : rev_base_bytes(B, T, Hkv, S, BS) + kv_slab_bytes(1, B, T, Hkv, 128);
}

// Behind the reverse index: one [16 x D] bf16 tile per (list position, 16-head sub-group) for the selected branch's dQ as
// per-visit partials (tcgen05 kernel only), then the fp32 dK, dV slabs of the shares and of the window.
static bool dq_from_kv_covers(int D, int S, int BS) { return D == 128 && BS == 64 && S <= 32; }
static size_t sel_dq_tile_bytes(int B, int Tq, int Hq, int D, int S, int BS) {
  return dq_from_kv_covers(D, S, BS) ? align_up((size_t)B * Tq * Hq * S * D * 2, 256) : 0;
}
struct KvSlabs {
  int nshare, nwin;                                             // shares of the selected lists, parts of the window
  int slabs() const { return (nshare > 1 ? nshare : 0) + nwin; }
};
static KvSlabs kv_slabs(int B, int T, int Hkv, int BS, int window) {
  return {kv_shares((long long)B * Hkv * ((T + BS - 1) / BS)), window > 0 ? dense_kv_window_slabs(B, T, Hkv, window) : 0};
}

size_t nsa_sel_swa_bwd_workspace_bytes_dq(int B, int T, int Tq, int Hq, int Hkv, int D, int S, int BS) {
  if (BS <= 0 || Hkv <= 0) return 0;
  return nsa_sel_index_bytes(B, T, Tq, Hkv, S, BS) + align_up((size_t)B * Tq * Hq * S * D * 2, 256) + kv_slab_bytes(1, B, T, Hkv, 128);
}

size_t nsa_sel_swa_bwd_ix_workspace_bytes(int B, int T, int Tq, int Hq, int Hkv, int D, int S, int BS, int window) {
  if (BS <= 0 || Hkv <= 0) return 0;
  return sel_dq_tile_bytes(B, Tq, Hq, D, S, BS) + kv_slab_bytes(kv_slabs(B, T, Hkv, BS, window).slabs(), B, T, Hkv, D);
}

size_t nsa_attn_bwd_ix_workspace_bytes(int B, int T, int Tc, int Hq, int Hkv, int D, int S, int BS, int window) {
  return std::max(nsa_sel_swa_bwd_ix_workspace_bytes(B, T, T, Hq, Hkv, D, S, BS, window),
                  nsa_cmp_attn_bwd_workspace_bytes(B, T, Tc, Hkv, D));
}

struct PreSel {   // row pre-pass of the selected and window branches folded into the window's dQ kernel
  const void *o_slc, *o_swa;
  void *dg_slc, *dg_swa;
};

struct CmpBwd {   // the compressed branch in the same call: its dQ shares the window's pass
  const void *ck, *cv;
  const float *lse, *delta;
  const void* gate;
  int Tc, block, stride, causal;
  GateAdd add;   // the gate projection's share of dq (where dQ comes from the key-major kernel)
};

static int sel_swa_bwd_impl(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    const void* dout_slc, const float* lse_slc, const float* delta_slc, const void* gate_slc,
                    const void* dout_swa, const float* lse_swa, const float* delta_swa, const void* gate_swa, void* dq,
                    int accumulate_dq, void* dk, void* dv, void* ws, size_t ws_bytes, int B, int T, int Hq, int Hkv,
                    int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream,
                    const PreSel* pre = nullptr, const void* index = nullptr, const CmpBwd* cmp = nullptr) {
  const bool sharded = (Tq != T) || (q0 != 0);
  if (Tq <= 0 || q0 < 0 || q0 + Tq > T) return fail(-12, "%s: query shard [%d, %d) is outside the sequence of %d tokens", "nsa_sel_swa_bwd", q0, q0 + Tq, T);
  (void)sharded;
  if (!q || !k || !v) return fail(-1, "nsa_sel_swa_bwd: null pointer");
  int rc = check_attn_shape("nsa_sel_swa_bwd", B, T, Hq, Hkv, D);
  if (rc) return rc;
  rc = check_bs("nsa_sel_swa_bwd", BS);
  if (rc) return rc;
  const bool has_slc = dout_slc != nullptr, has_swa = window > 0 && dout_swa != nullptr;
  if (!has_slc && !has_swa) return fail(-1, "nsa_sel_swa_bwd: neither branch has an upstream gradient");
  if (has_slc && (!idx || !lse_slc || !delta_slc)) return fail(-1, "nsa_sel_swa_bwd: selected branch inputs missing");
  if (has_swa && (!lse_swa || !delta_swa)) return fail(-1, "nsa_sel_swa_bwd: window branch inputs missing");
  cudaStream_t s = (cudaStream_t)stream;
  const long long rows = (long long)B * Tq * Hq;
  // With the larger workspace of nsa_sel_swa_bwd_workspace_bytes_dq the selected branch's dQ is produced by the
  // kv-major backward (per-visit partial tiles + a slot-order reduction) instead of the query-major dQ kernel.
  // (A caller that hands over a reverse index gives the workspace behind it alone, with room for the shares.)
  if (index && ws_bytes < nsa_sel_swa_bwd_ix_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS, has_swa ? window : 0))
    return fail(-6, "nsa_sel_swa_bwd_ix: workspace too small");
  const bool large_ws = index || (ws && ws_bytes >= nsa_sel_swa_bwd_workspace_bytes_dq(B, T, Tq, Hq, Hkv, D, S, BS));
  const bool dq_from_kv = dq && dk && has_slc && dq_from_kv_covers(D, S, BS) && large_ws;
  int dq_acc_for_reduce = accumulate_dq;
  bool fold = false;
  if (pre) {
    if ((has_slc && !pre->o_slc) || (has_swa && !pre->o_swa)) return fail(-1, "nsa_sel_swa_bwd_fused: a branch output is null");
    if (has_slc && has_swa && dout_slc != dout_swa)
      return fail(-15, "nsa_sel_swa_bwd_fused: both branches must share one upstream gradient (the module's dO)");
    // the window's tcgen05 dQ kernel carries the pre-pass of both branches and therefore runs first
    fold = dq && has_swa && D == 128;
    if (!fold) {
      const bf16* o3[3] = {has_slc ? (const bf16*)pre->o_slc : nullptr, has_swa ? (const bf16*)pre->o_swa : nullptr, nullptr};
      const bf16* g3[3] = {(const bf16*)gate_slc, (const bf16*)gate_swa, nullptr};
      float* d3[3] = {const_cast<float*>(delta_slc), const_cast<float*>(delta_swa), nullptr};
      bf16* dg3[3] = {(bf16*)pre->dg_slc, (bf16*)pre->dg_swa, nullptr};
      rc = launch_rowdot3(o3, (const bf16*)(has_slc ? dout_slc : dout_swa), g3, d3, dg3, rows, D, s);
      if (rc) return rc;
    }
  }
  if (dq) {
    int acc = accumulate_dq;
    // The selected branch's dQ from its own query-major kernel (else the reduction behind the key-major kernel adds it).  dq is
    // rounded to bf16 behind every kernel, so with the compressed branch in the dense pass the selected one, the smaller, goes
    // first (head_dim 64, 1024 tokens, error of dq against fp64: 3.12 to 3.16e-3 with the dense pass first, 3.04e-3 so).
    auto selected = [&]() {
      SelArgs a = {};
      a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.idx = idx; a.idx64 = idx64; a.counts = counts;
      a.lse = const_cast<float*>(lse_slc); a.dout = (const bf16*)dout_slc; a.delta = delta_slc;
      a.gate = (const bf16*)gate_slc; a.dq = (bf16*)dq; a.accumulate = acc;
      a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Hq = Hq; a.Hkv = Hkv; a.S = S; a.BS = BS; a.scale = scale;
      acc = 1;
      return launch_sel_dq(a, D, s);
    };
    const bool own_dq = has_slc && !dq_from_kv, sel_first = own_dq && cmp && !fold;
    if (sel_first) {
      rc = selected();
      if (rc) return rc;
    }
    if (has_swa || cmp) {   // with `fold` it also forms the deltas of both branches
      if (D != 128 && sharded) return fail(-11, "query shards need head_dim 128");
      DenseArgs a = {};
      a.q = (const bf16*)q; a.dout = (const bf16*)(has_swa ? dout_swa : dout_slc); a.dq = (bf16*)dq; a.accumulate = acc;
      a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Lk = T; a.Hq = Hq; a.Hk = Hkv; a.scale = scale;
      if (has_swa) {
        a.mode = 0; a.k = (const bf16*)k; a.v = (const bf16*)v; a.lse = const_cast<float*>(lse_swa); a.delta = delta_swa;
        a.gate = (const bf16*)gate_swa; a.window = window;
      }
      if (cmp) {
        a.cblock = cmp->block; a.cstride = cmp->stride; a.causal = cmp->causal; a.seq.Tc = cmp->Tc;
        if (has_swa) {
          a.ck = (const bf16*)cmp->ck; a.cv = (const bf16*)cmp->cv; a.lse_c = cmp->lse; a.delta_c = cmp->delta;
          a.gate_c = (const bf16*)cmp->gate;
        } else {
          a.mode = 1; a.k = (const bf16*)cmp->ck; a.v = (const bf16*)cmp->cv; a.lse = const_cast<float*>(cmp->lse);
          a.delta = cmp->delta; a.gate = (const bf16*)cmp->gate; a.Lk = cmp->Tc;
        }
      }
      if (fold) {
        a.pre_o[0] = (const bf16*)pre->o_swa; a.pre_gate[0] = (const bf16*)gate_swa;
        a.pre_delta[0] = const_cast<float*>(delta_swa); a.pre_dgate[0] = (bf16*)pre->dg_swa;
        if (has_slc) {
          a.pre_o[1] = (const bf16*)pre->o_slc; a.pre_gate[1] = (const bf16*)gate_slc;
          a.pre_delta[1] = const_cast<float*>(delta_slc); a.pre_dgate[1] = (bf16*)pre->dg_slc;
        }
      }
      rc = launch_dense_dq_tc(a, D, s);
      if (rc) return rc;
      acc = 1;
    }
    dq_acc_for_reduce = acc;
    if (own_dq && !sel_first) {
      rc = selected();
      if (rc) return rc;
    }
  }
  if (dk || dv) {
    if (!dk || !dv) return fail(-1, "nsa_sel_swa_bwd: dk and dv must be given together");
    if (sharded && (D != 128 || (has_slc && BS != 64))) return fail(-11, "query shards need head_dim 128 and 64-key selection blocks");
    // fp32 slabs behind everything else in the workspace (none for the window alone: it is rounded straight away).  Only a
    // caller with a reverse index of its own has room for shares and for parts of the window.
    KvSlabs n = {1, has_swa ? 1 : 0};
    bf16* tiles = nullptr;
    if (index) n = kv_slabs(B, T, Hkv, BS, has_swa ? window : 0);
    RevArgs r = {};
    float* part = nullptr;
    if (has_slc) {
      if (!index && (!ws || ws_bytes < nsa_sel_swa_bwd_workspace_bytes(B, T, Hkv, S, BS)))
        return fail(-6, "nsa_sel_swa_bwd: workspace too small");
      const size_t nrev = rev_layout(index ? const_cast<void*>(index) : ws, idx, idx64, counts, B, T, Tq, q0, Hkv, S, BS, &r);
      if (!index && !large_ws) r.inv = nullptr;   // the small workspace has the token lists only
      char* p = (char*)ws + (index ? 0 : nrev);
      if (dq_from_kv) tiles = (bf16*)p;
      if (index)
        part = (float*)(p + sel_dq_tile_bytes(B, Tq, Hq, D, S, BS));
      else if (large_ws)
        part = (float*)(p + align_up((size_t)B * Tq * Hq * S * D * 2, 256));
      else
        part = (float*)((char*)ws + rev_base_bytes(B, T, Hkv, S, BS));
      if (!index) {
        rc = launch_build_rev(r, s);
        if (rc) return rc;
      }
    }
    if (has_swa) {
      DenseKvArgs a = {};
      a.mode = 0; a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.dout = (const bf16*)dout_swa;
      a.lse = lse_swa; a.delta = delta_swa; a.gate = (const bf16*)gate_swa; a.dk = (bf16*)dk; a.dv = (bf16*)dv;
      a.part = part; a.nslab = part ? n.nwin : 1; a.slab0 = n.nshare > 1 ? n.nshare : 0; a.slabs = n.slabs();
      a.Hq = Hq; a.Hk = Hkv; a.Lk = T; a.window = window; a.scale = scale;
      a.seq.B = B; a.seq.Tq = Tq; a.seq.q0 = q0;
      rc = launch_dense_kv_tc(a, D, s);
      if (rc) return rc;
    }
    if (has_slc) {
      KvArgs a = {};
      a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.dout = (const bf16*)dout_slc; a.lse = lse_slc;
      a.delta = delta_slc; a.gate = (const bf16*)gate_slc;
      a.B = B; a.T = T; a.Tq = Tq; a.q0 = q0; a.Hq = Hq; a.Hk = Hkv; a.BS = BS; a.scale = scale; a.dk = (bf16*)dk; a.dv = (bf16*)dv;
      a.rev_ptr = r.rev_ptr; a.rev_tok = r.rev_tok; a.rev_cap = r.cap; a.dq_part = tiles;
      a.nshare = n.nshare; a.part = part; a.slabs = n.slabs(); a.nadd = n.nwin;
      rc = (D == 128 && BS == 64) ? launch_kv_bwd_tc(a, s) : launch_kv_bwd(a, D, s);
      if (rc) return rc;
      if (n.nshare > 1) {
        rc = launch_reduce_shares(part, a.dk, a.dv, n.slabs(), (long long)B * T * Hkv * D, s);
        if (rc) return rc;
      }
    }
    if (dq_from_kv) {   // every token's partial tiles, in slot order, onto dq (after the window's dQ if that ran first)
      rc = launch_sel_dq_reduce(r, tiles, (bf16*)dq, Hq, D, cmp ? cmp->add : GateAdd{}, scale, dq_acc_for_reduce, s);
      if (rc) return rc;
    }
  }
  return 0;
}

int nsa_sel_swa_bwd(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    const void* dout_slc, const float* lse_slc, const float* delta_slc, const void* gate_slc,
                    const void* dout_swa, const float* lse_swa, const float* delta_swa, const void* gate_swa, void* dq,
                    int accumulate_dq, void* dk, void* dv, void* ws, size_t ws_bytes, int B, int T, int Hq, int Hkv,
                    int D, int S, int BS, int window, float scale, void* stream) {
  return sel_swa_bwd_impl(q, k, v, idx, idx64, counts, dout_slc, lse_slc, delta_slc, gate_slc, dout_swa, lse_swa, delta_swa, gate_swa, dq, accumulate_dq, dk, dv, ws, ws_bytes, B, T, Hq, Hkv, D, S, BS, window, scale, T, 0, stream);
}

int nsa_sel_swa_bwd_sharded(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                    const void* dout_slc, const float* lse_slc, const float* delta_slc, const void* gate_slc,
                    const void* dout_swa, const float* lse_swa, const float* delta_swa, const void* gate_swa, void* dq,
                    int accumulate_dq, void* dk, void* dv, void* ws, size_t ws_bytes, int B, int T, int Hq, int Hkv,
                    int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream) {
  return sel_swa_bwd_impl(q, k, v, idx, idx64, counts, dout_slc, lse_slc, delta_slc, gate_slc, dout_swa, lse_swa, delta_swa, gate_swa, dq, accumulate_dq, dk, dv, ws, ws_bytes, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream);
}

int nsa_sel_swa_bwd_ix(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                       const void* index, const void* dout_slc, const float* lse_slc, const float* delta_slc,
                       const void* gate_slc, const void* dout_swa, const float* lse_swa, const float* delta_swa,
                       const void* gate_swa, void* dq, int accumulate_dq, void* dk, void* dv, void* ws, size_t ws_bytes, int B,
                       int T, int Hq, int Hkv, int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream) {
  return sel_swa_bwd_impl(q, k, v, idx, idx64, counts, dout_slc, lse_slc, delta_slc, gate_slc, dout_swa, lse_swa, delta_swa, gate_swa, dq, accumulate_dq, dk, dv, ws, ws_bytes, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream, nullptr, index);
}

int nsa_attn_bwd_ix(const void* q, const void* k, const void* v, const void* ck, const void* cv, const void* idx, int idx64,
                    const int32_t* counts, const void* index, const void* dout, const float* lse_slc, const float* lse_swa,
                    const float* lse_cmp, const float* delta_slc, const float* delta_swa, const float* delta_cmp,
                    const void* g_slc, const void* g_swa, const void* g_cmp, const void* dg_slc, const void* dg_swa,
                    const void* dg_cmp, const void* w_gate, void* dq, void* dk, void* dv, void* dck, void* dcv,
                    void* ws, size_t ws_bytes, int B, int T, int Tc, int Hq, int Hkv, int D, int S, int BS, int window, int block,
                    int stride, int causal, float scale, void* stream) {
  if (!ck || !cv || !lse_cmp || !dout || !delta_cmp || !dq || !dk || !dv || !dck || !dcv || !idx || !index || !ws)
    return fail(-1, "nsa_attn_bwd_ix: null pointer");
  if (Tc <= 0) return fail(-1, "nsa_attn_bwd_ix: no compressed position");
  if (ws_bytes < nsa_attn_bwd_ix_workspace_bytes(B, T, Tc, Hq, Hkv, D, S, BS, window))
    return fail(-6, "nsa_attn_bwd_ix: workspace too small");
  if (!aligned16(w_gate)) return fail(-5, "nsa_attn_bwd_ix: w_gate must be 16-byte aligned");
  if (w_gate && (!dq_from_kv_covers(D, S, BS) || !dg_slc || !dg_swa || !dg_cmp))
    return fail(-1, "nsa_attn_bwd_ix: the gate projection's share needs its gradients, head_dim 128 and 64-key blocks");
  const CmpBwd c = {ck, cv, lse_cmp, delta_cmp, g_cmp, Tc, block, stride, causal,
                    {{(const bf16*)dg_slc, (const bf16*)dg_swa, (const bf16*)dg_cmp}, (const bf16*)w_gate}};
  int rc = sel_swa_bwd_impl(q, k, v, idx, idx64, counts, dout, lse_slc, delta_slc, g_slc, window > 0 ? dout : nullptr, lse_swa, delta_swa, g_swa, dq, 0, dk, dv, ws, ws_bytes, B, T, Hq, Hkv, D, S, BS, window, scale, T, 0, stream, nullptr, index, &c);
  if (rc) return rc;
  return cmp_dkv(q, ck, cv, lse_cmp, dout, delta_cmp, g_cmp, dck, dcv, ws, B, T, Tc, Hq, Hkv, D, block, stride, causal, scale, T, 0, (cudaStream_t)stream);
}

int nsa_gather_probe(const void* k, const void* v, const void* idx, int idx64, int B, int T, int Hq, int Hkv, int D, int S,
                     int BS, void* stream) {
  if (!k || !v || !idx) return fail(-1, "nsa_gather_probe: null pointer");
  int rc = check_attn_shape("nsa_gather_probe", B, T, Hq, Hkv, D);
  if (rc) return rc;
  SelArgs a = {};
  a.k = (const bf16*)k; a.v = (const bf16*)v; a.idx = idx; a.idx64 = idx64;
  a.B = B; a.T = T; a.Tq = T; a.q0 = 0; a.Hq = Hq; a.Hkv = Hkv; a.S = S; a.BS = BS;
  return launch_gather_probe(a, D, (cudaStream_t)stream);
}

int nsa_sel_swa_bwd_fused(const void* q, const void* k, const void* v, const void* idx, int idx64, const int32_t* counts,
                          const void* o_slc, const void* o_swa, const void* dout, const float* lse_slc, float* delta_slc,
                          const void* gate_slc, void* dgate_slc, const float* lse_swa, float* delta_swa, const void* gate_swa,
                          void* dgate_swa, void* dq, int accumulate_dq, void* dk, void* dv, void* ws, size_t ws_bytes, int B,
                          int T, int Hq, int Hkv, int D, int S, int BS, int window, float scale, int Tq, int q0, void* stream) {
  if (!dout || !delta_slc) return fail(-1, "nsa_sel_swa_bwd_fused: null pointer");
  if (window > 0 && !delta_swa) return fail(-1, "nsa_sel_swa_bwd_fused: delta_swa is null");
  const PreSel pre = {o_slc, o_swa, dgate_slc, dgate_swa};
  return sel_swa_bwd_impl(q, k, v, idx, idx64, counts, dout, lse_slc, delta_slc, gate_slc, window > 0 ? dout : nullptr, lse_swa, delta_swa, gate_swa, dq, accumulate_dq, dk, dv, ws, ws_bytes, B, T, Hq, Hkv, D, S, BS, window, scale, Tq, q0, stream, &pre);
}

// ---- decode ---------------------------------------------------------------------------------------------
int nsa_decode_fwd(const void* q, const void* k, const void* v, const void* ck, const void* cv, const int32_t* cu_k,
                   const int32_t* cu_c, const int32_t* order, const void* gate_w, const void* gate_b, const void* g_slc,
                   const void* g_swa, const void* g_cmp, void* o, void* o_cmp, void* o_slc, void* o_swa, float* lse,
                   int32_t* idx, void* ws, size_t ws_bytes, int nseq,
                   long long total_k, long long total_c, int max_Tc, int Hq, int Hkv, int D, int block, int stride,
                   int sel_block, int n_sel, int window, float scale, void* stream) {
  if (!q || !k || !v || !ck || !cv || !cu_k || !cu_c || !o || !idx || !ws) return fail(-1, "nsa_decode_fwd: null pointer");
  if (nseq <= 0) return 0;
  if (total_k <= 0 || total_c <= 0 || Hq <= 0 || Hkv <= 0) return fail(-1, "nsa_decode_fwd: empty shape");
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(ck) || !aligned16(cv) || !aligned16(o))
    return fail(-5, "nsa_decode_fwd: pointers must be 16-byte aligned");
  DecodeArgs a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.ck = (const bf16*)ck; a.cv = (const bf16*)cv;
  a.cu_k = cu_k; a.cu_c = cu_c; a.order = order; a.gate_w = (const bf16*)gate_w; a.gate_b = (const bf16*)gate_b;
  a.g_slc = (const bf16*)g_slc; a.g_swa = (const bf16*)g_swa; a.g_cmp = (const bf16*)g_cmp;
  a.o = (bf16*)o; a.o_cmp = (bf16*)o_cmp; a.o_slc = (bf16*)o_slc; a.o_swa = (bf16*)o_swa; a.lse = lse; a.idx = idx;
  a.nseq = nseq; a.Hq = Hq; a.Hkv = Hkv; a.D = D; a.n_sel = n_sel; a.window = window; a.cblock = block; a.cstride = stride;
  a.sel_block = sel_block; a.total_k = total_k; a.total_c = total_c; a.max_Tc = max_Tc; a.scale = scale;
  a.part = (float*)ws; a.part_bytes = ws_bytes;
  return launch_decode(a, (cudaStream_t)stream);
}

size_t nsa_decode_workspace_bytes(int nseq, int Hkv) { return decode_workspace_bytes(nseq, Hkv); }

// ---- helpers ------------------------------------------------------------------------------------------
int nsa_rowdot(const void* o, const void* dout, const void* gate, float* delta, void* dgate, long long rows, int D,
               void* stream) {
  if (!o || !dout) return fail(-1, "nsa_rowdot: null pointer");
  return launch_rowdot((const bf16*)o, (const bf16*)dout, (const bf16*)gate, delta, (bf16*)dgate, rows, D,
                       (cudaStream_t)stream);
}

int nsa_gate_fwd(const void* q, const void* w, const void* bias, void* g_slc, void* g_swa, void* g_cmp, long long rows,
                 int D, void* stream) {
  if (!q || !w || !g_slc || !g_swa || !g_cmp) return fail(-1, "nsa_gate_fwd: null pointer");
  if (!aligned16(q) || !aligned16(w)) return fail(-5, "nsa_gate_fwd: pointers must be 16-byte aligned");
  return launch_gate_fwd((const bf16*)q, (const bf16*)w, (const bf16*)bias, (bf16*)g_slc, (bf16*)g_swa, (bf16*)g_cmp, rows,
                         D, (cudaStream_t)stream);
}

int nsa_rowdot3(const void* o_slc, const void* o_swa, const void* o_cmp, const void* dout, const void* g_slc,
                const void* g_swa, const void* g_cmp, float* delta_slc, float* delta_swa, float* delta_cmp, void* dg_slc,
                void* dg_swa, void* dg_cmp, long long rows, int D, void* stream) {
  if (!dout) return fail(-1, "nsa_rowdot3: null upstream gradient");
  const bf16* o[3] = {(const bf16*)o_slc, (const bf16*)o_swa, (const bf16*)o_cmp};
  const bf16* g[3] = {(const bf16*)g_slc, (const bf16*)g_swa, (const bf16*)g_cmp};
  float* dl[3] = {delta_slc, delta_swa, delta_cmp};
  bf16* dg[3] = {(bf16*)dg_slc, (bf16*)dg_swa, (bf16*)dg_cmp};
  return launch_rowdot3(o, (const bf16*)dout, g, dl, dg, rows, D, (cudaStream_t)stream);
}

long long nsa_gate_bwd_workspace_bytes(long long rows, int D) { return gate_bwd_workspace_bytes(rows, D); }

int nsa_gate_bwd(const void* q, const void* dg_slc, const void* dg_swa, const void* dg_cmp, const void* w, void* dq,
                 void* dw, void* dbias, void* workspace, long long workspace_bytes, long long rows, int D, void* stream) {
  if (!q || !dg_slc || !dg_swa || !dg_cmp || !w || !dw || !workspace) return fail(-1, "nsa_gate_bwd: null pointer");
  if (!aligned16(q) || !aligned16(w) || !aligned16(dq)) return fail(-5, "nsa_gate_bwd: pointers must be 16-byte aligned");
  if (workspace_bytes < gate_bwd_workspace_bytes(rows, D)) return fail(-3, "nsa_gate_bwd: workspace too small");
  return launch_gate_bwd((const bf16*)q, (const bf16*)dg_slc, (const bf16*)dg_swa, (const bf16*)dg_cmp, (const bf16*)w,
                         (bf16*)dq, (bf16*)dw, (bf16*)dbias, (float*)workspace, rows, D, (cudaStream_t)stream);
}

int nsa_combine(const void* a0, const void* g0, const void* a1, const void* g1, const void* a2, const void* g2, void* o,
                long long rows, int D, void* stream) {
  if (!o) return fail(-1, "nsa_combine: null output");
  return launch_combine((const bf16*)a0, (const bf16*)g0, (const bf16*)a1, (const bf16*)g1, (const bf16*)a2,
                        (const bf16*)g2, (bf16*)o, rows, D, (cudaStream_t)stream);
}

}  // extern "C"
