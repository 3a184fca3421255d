// Forward pass of a whole GPT model without a graph (scoring, prompts, decoding steps): one library
// call queues every kernel of the model. Called op by op from Python a decoding step of a 12-block
// model is about 100 calls and 1.9 ms of host time around 0.37 ms on the device (124 M parameters, fp16, 8 sequences; queueing
// its 62 launches from here takes 0.35 ms).
//
// Two schedules. A step with one new token per sequence (and few sequences) runs five kernels per
// block: {norm + q/k/v}, {rotary + QK-norm + cache append + attention}, {output projection +
// residual}, {norm + up-projection + activation}, {down-projection + residual}, all launched with
// programmatic serialisation so that a kernel's weights travel while its predecessor finishes.
// Everything else runs the training kernels: norm, GEMM with its epilogues, flash attention.
#include "attention.cuh"
#include "common.cuh"
#include "decode.cuh"
#include "gemm.cuh"
#include "skinny.cuh"
#include "tempbuf.cuh"

namespace mt {

enum { BP_LN1_W, BP_LN1_B, BP_LN2_W, BP_LN2_B, BP_Q, BP_K, BP_V, BP_O, BP_UP, BP_DOWN, BP_BQ, BP_BK, BP_BV, BP_BO, BP_BUP, BP_BDOWN,
       BP_COUNT };

constexpr int64_t kStepRows = 32;        // sequences up to which a step takes the five-kernel schedule
constexpr int64_t kFusedNormRows = 32;   // rows up to which a norm is folded into the product behind it

struct Infer {
  const mt_gpt_model& g;
  const mt_gpt_pass& s;
  cudaStream_t st;
  int64_t M, E, D, nq, nkv, nqkv, es;

  int norm_kind() const { return g.kind == MT_GPT_LEARNED ? 1 : 2; }
  int norm(const void* x, const void* w, const void* b, void* y, int64_t rows) const {
    return g.kind == MT_GPT_LEARNED ? mt_layernorm_fwd(x, w, b, y, nullptr, nullptr, rows, E, g.eps, g.dtype, (void*)st)
                                    : mt_rmsnorm_fwd(x, w, y, nullptr, rows, E, g.eps, g.dtype, (void*)st);
  }
  // out = act(norm(x) @ w^T + bias) for up to three weights side by side
  int norm_linear(const void* x, int64_t rows, const void* nw, const void* nb, void* h, int nseg, const void* const* w,
                  const void* const* bias, const int64_t* n, void* out, int64_t ldo, int act, float softcap) const {
    SkinnyArgs a;
    a.x = x; a.ldx = E; a.M = (int)rows; a.K = (int)E; a.dtype = g.dtype;
    a.nseg = nseg; a.ldw = E;
    for (int i = 0; i < nseg; ++i) { a.w[i] = w[i]; a.bias[i] = bias[i]; a.n[i] = (int)n[i]; }
    a.out = out; a.ldo = ldo; a.act = act; a.softcap = softcap;
    a.norm = norm_kind(); a.gamma = nw; a.beta = nb; a.eps = g.eps;
    a.early_weights = 1;
    SkinnyShape shape;
    if (gemm_automatic() && rows <= kFusedNormRows && skinny_fits(a, shape)) return skinny_gemm(a, shape, st);
    int rc = norm(x, nw, nb, h, rows);
    int64_t col = 0;
    for (int i = 0; i < nseg && !rc; ++i) {
      rc = mt_gemm(h, w[i], (char*)out + col * es, nullptr, bias[i], rows, n[i], E, E, E, ldo, 0, 1, g.dtype, g.dtype, act, 1.f, 0,
                   (void*)st);
      col += n[i];
    }
    if (!rc && softcap > 0.f) rc = mt_softcap(out, out, rows * ldo, softcap, g.dtype, (void*)st);
    return rc;
  }
  // x += a @ w^T + bias
  int linear_residual(const void* a_, const void* w, const void* bias, void* x, int64_t rows, int64_t K) const {
    SkinnyArgs a;
    a.x = a_; a.ldx = K; a.M = (int)rows; a.K = (int)K; a.dtype = g.dtype;
    a.w[0] = w; a.bias[0] = bias; a.n[0] = (int)E; a.ldw = K;
    a.out = x; a.ldo = E; a.residual = x; a.early_weights = 1;
    SkinnyShape shape;
    if (gemm_automatic() && skinny_fits(a, shape)) return skinny_gemm(a, shape, st);
    return mt_gemm_ex(a_, w, x, nullptr, bias, x, 1, rows, E, K, K, K, E, 0, 1, g.dtype, g.dtype, 0, 1.f, 0, (void*)st);
  }
  mt_strides3 rows_of(int64_t ld, int64_t d) const { return mt_strides3{s.new_tokens * ld, d, ld}; }

  // q, k, v of head 0, token 0 inside one row of the projection, and their head strides
  void split_qkv(void* qkv, char*& q, char*& k, char*& v, mt_strides3& sq, mt_strides3& skv) const {
    if (g.kind == MT_GPT_LEARNED) {            // per head [q | k | v]
      q = (char*)qkv; k = q + D * es; v = q + 2 * D * es;
      sq = skv = rows_of(nqkv, 3 * D);
    } else {
      q = (char*)qkv; k = q + nq * es; v = q + (nq + nkv) * es;
      sq = skv = rows_of(nqkv, D);
    }
  }
  float scale() const { return 1.f / sqrtf((float)D); }
  int run();
};

static size_t up256(size_t n) { return (n + 255) / 256 * 256; }

int Infer::run() {
  const int64_t B = s.batch, T = s.new_tokens, H = g.heads, Hk = g.kv_heads, F = g.hidden;
  const bool learned = g.kind == MT_GPT_LEARNED;
  const bool cached = s.k_cache != nullptr;
  const bool step = cached && s.past > 0 && T == 1 && B <= kStepRows && (D == 64 || D == 128);
  const size_t bx = up256((size_t)M * E * es), bqkv = up256((size_t)M * nqkv * es), bmlp = up256((size_t)M * F * es);
  const size_t brope = learned || step ? 0 : up256((size_t)M * (nq + nkv) * es);
  const size_t blse = step ? 0 : up256((size_t)M * H * 4), brstd = learned || step ? 0 : 2 * blse;
  // Two regions serve twice per block, so that what a kernel reads is still in the L2: the normed rows are dead when attention
  // writes its output, the projections when the up-projection writes the hidden rows.
  const size_t bwide = bqkv + brope > bmlp ? bqkv + brope : bmlp;
  TempBuf buf(2 * bx + bwide + blse + brstd, st);
  if (!buf.ok()) return MT_ERR_CUDA;
  char* at = (char*)buf.ptr;
  auto take = [&](size_t n) { char* p = at; at += n; return p; };
  char *x = take(bx), *h = take(bx), *qkv = take(bwide);
  char *att = h, *mlp = qkv, *roped = qkv + bqkv;
  float* lse = (float*)take(blse);
  float* rstd = (float*)take(brstd);
  void* stream = (void*)st;
  int rc = learned ? mt_embedding_pos_fwd(g.wte, (const char*)g.wpe + s.position * E * es, s.ids, x, M, T, E, g.vocab, g.dtype, stream)
                   : mt_embedding_fwd(g.wte, s.ids, x, M, E, g.vocab, g.dtype, stream);
  const int64_t nseg3[3] = {nq, nkv, nkv}, nseg1[1] = {nqkv};
  for (int64_t l = 0; l < g.blocks && !rc; ++l) {
    const void* const* w = g.block_ptrs + l * BP_COUNT;
    rc = norm_linear(x, M, w[BP_LN1_W], w[BP_LN1_B], h, learned ? 1 : 3, w + BP_Q, w + BP_BQ, learned ? nseg1 : nseg3, qkv, nqkv, 0,
                     0.f);
    if (rc) break;
    char *q, *k, *v;
    mt_strides3 sq, skv;
    split_qkv(qkv, q, k, v, sq, skv);
    const mt_strides3 so = rows_of(E, D);
    if (step) {
      DecodeStep d{};
      d.q = q; d.k_cache = s.k_cache[l]; d.v_cache = s.v_cache[l]; d.o = att;
      d.sq = sq; d.sc = s.cache_strides; d.so = so;
      d.batch = B; d.heads = H; d.kv_heads = Hk; d.q_len = 1; d.kv_len = s.kv_len; d.head_dim = D;
      d.scale = scale(); d.causal_offset = -1; d.dtype = g.dtype;
      d.fused = 1; d.k_new = k; d.v_new = v; d.sk_new = skv; d.sv_new = skv; d.append_slot = s.write_pos;
      d.early_cache = 1;
      if (!learned) { d.cos_row = g.cos_t + s.position * D; d.sin_row = g.sin_t + s.position * D; d.eps = g.eps; }
      rc = attn_decode_step(d, st);
    } else {
      if (!learned) {
        char* yq = roped;
        char* yk = roped + (size_t)M * nq * es;
        const float *cs = g.cos_t + s.position * D, *sn = g.sin_t + s.position * D;
        rc = mt_rope_rmsnorm_fwd(q, nullptr, yq, nullptr, rstd, nullptr, cs, sn, B, T, H, D, nqkv, nq, g.eps, g.dtype, stream);
        if (!rc) rc = mt_rope_rmsnorm_fwd(k, nullptr, yk, nullptr, rstd + M * H, nullptr, cs, sn, B, T, Hk, D, nqkv, nkv, g.eps, g.dtype, stream);
        if (rc) break;
        q = yq; k = yk;
        sq = rows_of(nq, D);
      }
      const mt_strides3 sk = learned ? skv : rows_of(nkv, D);
      if (cached) rc = kv_append(k, v, s.k_cache[l], s.v_cache[l], sk, skv, s.cache_strides, B, Hk, T, s.write_pos, s.max_len, D, g.dtype, st);
      if (rc) break;
      if (cached && s.past > 0)
        rc = mt_attn_decode_gqa(q, s.k_cache[l], s.v_cache[l], att, sq, s.cache_strides, so, B, H, Hk, T, s.kv_len, D, scale(),
                                learned ? -1 : (int)s.past, g.dtype, stream);
      else
        rc = mt_attn_fwd_gqa(q, k, v, att, lse, sq, sk, skv, so, B, H, Hk, T, D, scale(), 1, g.dtype, stream);
    }
    if (!rc) rc = linear_residual(att, w[BP_O], w[BP_BO], x, M, nq);
    const int64_t nf[1] = {F};
    if (!rc) rc = norm_linear(x, M, w[BP_LN2_W], w[BP_LN2_B], h, 1, w + BP_UP, w + BP_BUP, nf, mlp, F, learned ? MT_ACT_GELU : MT_ACT_RELU2, 0.f);
    if (!rc) rc = linear_residual(mlp, w[BP_DOWN], w[BP_BDOWN], x, M, F);
  }
  if (rc) return rc;
  int64_t rows = M;
  const void* last = x;
  if (s.last_only && T > 1) {                // the head only sees each sequence's last position
    MT_CHECK_CUDA(cudaMemcpy2DAsync(qkv, E * es, x + (T - 1) * E * es, T * E * es, E * es, B, cudaMemcpyDeviceToDevice, st));
    last = qkv;
    rows = B;
  }
  const int64_t nv[1] = {g.vocab};
  return norm_linear(last, rows, g.lnf_w, g.lnf_b, h, 1, &g.head_w, &g.head_b, nv, s.logits, g.vocab, 0, s.softcap);
}

// One block per row; two independent 16-byte loads per thread and step. A row is read once
// (50257 fp32 logits = 200 KB, latency-bound).
template <typename T>
__global__ void __launch_bounds__(1024)
argmax_rows_kernel(const T* __restrict__ x, int32_t* __restrict__ idx, int32_t* __restrict__ out, int64_t cols, int64_t ld_out) {
  constexpr int VN = Vec16<T>::N;
  __shared__ float best_v[32];
  __shared__ int best_i[32];
  grid_dependency_wait();
  allow_dependents();
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  float v = -INFINITY;
  int at = 0x7fffffff;
  // NaN counts as larger than everything; of equals the smaller index stays
  auto better = [](float a, int ia, float b, int ib) {
    const bool na = isnan(a), nb = isnan(b);
    if (na != nb) return na;
    if (!na && a != b) return a > b;
    return ia < ib;
  };
  auto see = [&](float a, int i) { if (better(a, i, v, at)) { v = a; at = i; } };
  const int64_t head = min(cols, (int64_t)(((16 - (reinterpret_cast<uintptr_t>(xr) & 15)) & 15) / sizeof(T)));
  for (int64_t i = threadIdx.x; i < head; i += blockDim.x) see(to_f(xr[i]), (int)i);
  const int64_t nvec = (cols - head) / VN;
#pragma unroll 4
  for (int64_t j = threadIdx.x; j < nvec; j += blockDim.x) {
    Vec16<T> t;
    t.load(xr + head + j * VN);
#pragma unroll
    for (int e = 0; e < VN; ++e) see(t.get(e), (int)(head + j * VN + e));
  }
  for (int64_t i = head + nvec * VN + threadIdx.x; i < cols; i += blockDim.x) see(to_f(xr[i]), (int)i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float vo = __shfl_xor_sync(0xffffffffu, v, o);
    const int io = __shfl_xor_sync(0xffffffffu, at, o);
    if (better(vo, io, v, at)) { v = vo; at = io; }
  }
  if ((threadIdx.x & 31) == 0) { best_v[threadIdx.x >> 5] = v; best_i[threadIdx.x >> 5] = at; }
  __syncthreads();
  if (threadIdx.x < 32) {
    v = best_v[threadIdx.x];
    at = best_i[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float vo = __shfl_xor_sync(0xffffffffu, v, o);
      const int io = __shfl_xor_sync(0xffffffffu, at, o);
      if (better(vo, io, v, at)) { v = vo; at = io; }
    }
    if (threadIdx.x == 0) {
      idx[row] = at;
      if (out) out[row * ld_out] = at;
    }
  }
}

}  // namespace mt

using namespace mt;

extern "C" int mt_argmax_rows(const void* x, int32_t* idx, int32_t* out, int64_t rows, int64_t cols, int64_t ld_out, int dtype,
                              void* stream) {
  MT_REQUIRE(x && idx && rows >= 0 && cols > 0 && cols < (1ll << 31) && rows < (1ll << 31), "argmax_rows: bad arguments");
  if (rows == 0) return MT_OK;
  MT_DISPATCH_FLOAT(dtype, T, MT_CHECK_CUDA(launch_overlapped(argmax_rows_kernel<T>, dim3((unsigned)rows), dim3(1024), 0, as_stream(stream),
                                                              (const T*)x, idx, out, cols, ld_out)));
  count_launch();
  return MT_OK;
}

extern "C" int mt_gpt_forward(const mt_gpt_model* model, const mt_gpt_pass* pass, void* stream) {
  MT_REQUIRE(model && pass, "gpt_forward: no model or pass");
  const mt_gpt_model& g = *model;
  const mt_gpt_pass& s = *pass;
  MT_REQUIRE(g.kind == MT_GPT_LEARNED || g.kind == MT_GPT_ROTARY, "gpt_forward: unknown model kind");
  MT_REQUIRE(g.dtype == MT_F32 || g.dtype == MT_F16 || g.dtype == MT_BF16, "gpt_forward: unsupported dtype code %d", g.dtype);
  MT_REQUIRE(g.blocks >= 0 && g.width > 0 && g.hidden > 0 && g.heads > 0 && g.kv_heads > 0 && g.vocab > 0 && g.width % g.heads == 0 &&
             g.heads % g.kv_heads == 0 && g.wte && g.head_w && (g.blocks == 0 || g.block_ptrs), "gpt_forward: bad model");
  MT_REQUIRE(g.kind == MT_GPT_ROTARY ? g.cos_t && g.sin_t : g.wpe && g.heads == g.kv_heads, "gpt_forward: bad position tables");
  MT_REQUIRE(s.ids && s.logits && s.batch >= 0 && s.new_tokens >= 0 && s.past >= 0 && s.position >= 0, "gpt_forward: bad pass");
  MT_REQUIRE(!s.k_cache == !s.v_cache && (!s.k_cache || (s.max_len > 0 && s.write_pos >= 0 && s.write_pos < s.max_len &&
             s.new_tokens <= s.max_len && s.kv_len >= 1 && s.kv_len <= s.max_len)), "gpt_forward: bad cache");
  const int64_t M = s.batch * s.new_tokens;
  if (M == 0) return MT_OK;
  MT_REQUIRE(M < (1ll << 31) && g.vocab < (1ll << 31), "gpt_forward: too many tokens");
  const int64_t D = g.width / g.heads;
  Infer run{g, s, as_stream(stream), M, g.width, D, g.heads * D, g.kv_heads * D, (g.heads + 2 * g.kv_heads) * D, (int64_t)dtype_size(g.dtype)};
  return run.run();
}
