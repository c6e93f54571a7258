// One call per sublayer of a transformer layer (vy_attn_block_fwd / _bwd, vy_ffn_block_fwd / _bwd): the launches of the attention block (projection with
// rotation and cache append, attention, output projection with residual, LayerNorm) and of the feed-forward block, forward and backward, from one
// argument block and one scratch buffer each. The launches, their order and their arguments are those of the single entry points; what goes is the time between
// them, which bounded these layers on the host: 18 us of argument handling and allocation per launch where the launch itself takes 4. One token of a
// 768-wide layer behind 300 cached ones: 160 us, so 93 (device 35); 8 x 512 tokens: 179, so 135 (device 118); forward and backward of 64 x 128 tokens: 961, so 599 (device 517).
#include "vy_common.cuh"

namespace vy {

struct Carve {   // consecutive pieces of a buffer, 256-byte aligned (base null: sizes only)
  char* base;
  int64_t at;
  template <typename T = void>
  T* take(int64_t bytes) {
    T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += (bytes + 255) / 256 * 256;
    return p;
  }
};

static void set_hint(VyGemm& g, int hint) {   // flavour | width << 4 | splits << 16
  g.hint_flavour = hint & 15;
  g.hint_bn = (hint >> 4) & 4095;
  g.hint_splits = hint >> 16;
}

// y = act(x W^T + b) + addend as nn.Linear has it; few rows go the other way round
struct Lin {
  int rows, n, k, dtype, act, hint, weights_static;
  const void *x, *w, *b, *addend;
  void *aux, *out;
  void* stream;
};
static int linear(const Lin& l) {
  VyGemm g;
  memset(&g, 0, sizeof(g));
  const bool swap = l.rows <= VY_BLOCK_SWAP_ROWS;
  g.M = swap ? l.n : l.rows;
  g.N = swap ? l.rows : l.n;
  g.K = l.k;
  g.in_dtype = l.dtype;
  g.A = swap ? l.w : l.x;
  g.B = swap ? l.x : l.w;
  g.lda = g.ldb = l.k;
  g.epi = VY_EPI_LINEAR;
  g.act = l.act;
  g.transposed_out = swap;
  g.bias = l.b;
  g.bias_dtype = l.dtype;
  g.addend = l.addend;
  g.ld_addend = l.n;
  g.addend_dtype = l.dtype;
  g.aux = l.aux;
  g.ld_aux = l.n;
  g.aux_dtype = l.dtype;
  g.out_scale = 1.f;
  g.out = l.out;
  g.ld_out = l.n;
  g.out_dtype = l.dtype;
  g.weights_static = swap && l.weights_static;
  g.stream = l.stream;
  set_hint(g, l.hint);
  return vy_gemm(&g);
}
// dX [rows, k] = dY [rows, n] W [n, k] (+ addend), times act'(aux) with an activation
static int dgrad(int rows, int n, int k, int dtype, const void* dy, const void* w, const void* addend, int act, void* aux, void* out, int out_dtype, int hint, void* stream) {
  VyGemm g;
  memset(&g, 0, sizeof(g));
  g.M = rows;
  g.N = k;
  g.K = n;
  g.in_dtype = dtype;
  g.A = dy;
  g.lda = n;
  g.B = w;
  g.ldb = k;
  g.b_mn_major = 1;
  g.epi = VY_EPI_LINEAR;
  g.act = act;
  g.addend = addend;
  g.ld_addend = k;
  g.addend_dtype = dtype;
  g.aux = aux;
  g.ld_aux = k;
  g.aux_dtype = dtype;
  g.out_scale = 1.f;
  g.out = out;
  g.ld_out = k;
  g.out_dtype = out_dtype;
  g.stream = stream;
  set_hint(g, hint);
  return vy_gemm(&g);
}
// dW [n, k] = dY^T X
static int wgrad(int rows, int n, int k, int dtype, const void* dy, const void* x, void* out, void* ws, int64_t ws_bytes, int hint, void* stream) {
  VyGemm g;
  memset(&g, 0, sizeof(g));
  g.M = n;
  g.N = k;
  g.K = rows;
  g.in_dtype = dtype;
  g.A = dy;
  g.lda = n;
  g.a_mn_major = 1;
  g.B = x;
  g.ldb = k;
  g.b_mn_major = 1;
  g.epi = VY_EPI_LINEAR;
  g.out_scale = 1.f;
  g.out = out;
  g.ld_out = k;
  g.out_dtype = dtype;
  g.workspace = ws;
  g.workspace_bytes = ws_bytes;
  g.stream = stream;
  set_hint(g, hint);
  return vy_gemm(&g);
}
static int norm(int rows, int width, int dtype, const void* s, const void* gamma, const void* beta, float eps, void* y, float* mean, float* rstd, void* stream) {
  VyNorm v;
  memset(&v, 0, sizeof(v));
  v.rows = rows;
  v.H = width;
  v.x = s;
  v.io_dtype = v.param_dtype = dtype;
  v.gamma = gamma;
  v.beta = beta;
  v.eps = eps;
  v.y = y;
  v.mean = mean;
  v.rstd = rstd;
  v.kind = VY_NORM_LAYER;
  v.stream = stream;
  return vy_add_layernorm_fwd(&v);
}
static int norm_bwd(int rows, int width, int dtype, const void* dy, const void* s, const void* gamma, const float* mean, const float* rstd, void* ds, void* dgamma,
                    void* dbeta, void* dbias, float* partials, void* stream) {
  VyNorm v;
  memset(&v, 0, sizeof(v));
  v.rows = rows;
  v.H = width;
  v.io_dtype = v.param_dtype = v.dparam_dtype = dtype;
  v.gamma = gamma;
  v.mean = const_cast<float*>(mean);
  v.rstd = const_cast<float*>(rstd);
  v.dy = dy;
  v.s = s;
  v.dx = ds;
  v.dgamma = dgamma;
  v.dbeta = dbeta;
  v.dbias = dbias;
  v.partials = partials;
  v.kind = VY_NORM_LAYER;
  v.stream = stream;
  return vy_add_layernorm_bwd(&v);
}

// ---- attention block ----
struct AttnParts {   // of `scratch`: what the backward call reads is kept there with `save`
  void *qkv, *q, *k, *v, *attn, *s;
  float *lse, *mean, *rstd, *split;
};
static VyDecode decode_args(const VyAttnBlock* p, const AttnParts& a) {
  VyDecode d;
  memset(&d, 0, sizeof(d));
  d.B = p->seqs;
  d.n_q_heads = p->heads;
  d.n_kv_heads = p->kv_heads;
  d.head_dim = 64;
  d.start_pos = p->start;
  d.cache_len = p->cache_len;
  d.qkv = a.qkv;
  d.ld_qkv = (p->heads + 2 * p->kv_heads) * 64;
  d.qkv_dtype = p->dtype;
  d.rope_cos = p->rope_cos;
  d.rope_sin = p->rope_sin;
  d.rope_pos_off = p->rope_pos - p->start;   // the tables are addressed by cache slot
  d.rope_rows = p->rope_rows;
  d.k_cache = p->k_cache;
  d.v_cache = p->v_cache;
  d.cache_sb = p->c_sb;
  d.cache_sh = p->c_sh;
  d.cache_sl = p->c_sl;
  d.cache_dtype = p->cache_dtype;
  d.out = a.attn;
  d.ld_out = p->heads * 64;
  d.out_dtype = p->dtype;
  d.tickets = p->tickets;
  d.stream = p->stream;
  return d;
}
static AttnParts carve(const VyAttnBlock* p, void* base, int64_t* bytes) {
  Carve c = {static_cast<char*>(base), 0};
  AttnParts a;
  memset(&a, 0, sizeof(a));
  const int64_t rows = static_cast<int64_t>(p->seqs) * p->tokens, es = dtype_size(p->dtype), hq = p->heads * 64, hk = p->kv_heads * 64;
  if (p->decode) {
    a.qkv = c.take(rows * (hq + 2 * hk) * es);
  } else {
    a.q = c.take(rows * hq * 2);
    if (!p->k_cache) {
      a.k = c.take(rows * hk * 2);
      a.v = c.take(rows * hk * 2);
    }
  }
  a.attn = c.take(rows * hq * es);
  a.s = c.take(rows * p->width * es);
  if (p->save) {
    a.lse = c.take<float>(rows * p->heads * 4);
    a.mean = c.take<float>(rows * 4);
    a.rstd = c.take<float>(rows * 4);
  }
  if (p->decode) {
    const VyDecode d = decode_args(p, a);
    const int splits = vy_attn_decode_plan(&d);
    if (splits > 1) a.split = c.take<float>(static_cast<int64_t>(p->seqs) * p->kv_heads * splits * (p->heads / p->kv_heads) * 66 * 4);
  }
  *bytes = c.at;
  return a;
}
static bool block_ok(const VyAttnBlock* p, const char* who) {
  if (p && p->seqs > 0 && p->tokens > 0 && p->width > 0 && p->heads > 0 && p->kv_heads > 0 && p->heads % p->kv_heads == 0 && dtype_ok(p->dtype) && p->x && p->w_qkv && p->w_out &&
      p->gamma && p->beta && (p->k_cache == nullptr) == (p->v_cache == nullptr) && (!p->decode || (p->tokens == 1 && p->k_cache)) && (!p->save || !p->k_cache) &&
      (!p->k_cache || p->decode || p->cache_dtype == VY_BF16))
    return true;
  set_error("%s: bad arguments", who);
  return false;
}

static int attn_args(const VyAttnBlock* p, const AttnParts& a, VyAttn& t) {
  memset(&t, 0, sizeof(t));
  const int64_t S = p->tokens;
  t.B = p->seqs;
  t.n_q_heads = p->heads;
  t.n_kv_heads = p->kv_heads;
  t.head_dim = 64;
  t.Sq = p->tokens;
  t.Skv = p->k_cache ? p->start + p->tokens : p->tokens;
  t.qkv_dtype = VY_BF16;
  t.q = a.q;
  t.q_sb = p->heads * S * 64;
  t.q_sh = S * 64;
  t.q_sl = 64;
  t.k = p->k_cache ? p->k_cache : a.k;
  t.v = p->k_cache ? p->v_cache : a.v;
  t.k_sb = t.v_sb = p->k_cache ? p->c_sb : p->kv_heads * S * 64;
  t.k_sh = t.v_sh = p->k_cache ? p->c_sh : S * 64;
  t.k_sl = t.v_sl = p->k_cache ? p->c_sl : 64;
  t.causal = p->causal;
  t.q_pos0 = p->q_pos0;
  t.key_padding_mask = p->key_padding;
  t.kpm_stride = p->kpm_stride;
  t.out = a.attn;
  t.o_sb = S * p->heads * 64;
  t.o_sl = p->heads * 64;
  t.out_dtype = p->dtype;
  t.lse = a.lse;
  t.stream = p->stream;
  return VY_OK;
}

// ---- feed-forward block ----
struct FfnParts { void *z, *a, *s; float *mean, *rstd; };
static FfnParts carve(const VyFfnBlock* p, void* base, int64_t* bytes) {
  Carve c = {static_cast<char*>(base), 0};
  FfnParts f;
  memset(&f, 0, sizeof(f));
  const int64_t rows = p->rows, es = dtype_size(p->dtype);
  if (p->save) f.z = c.take(rows * p->inner * es);
  f.a = c.take(rows * p->inner * es);
  f.s = c.take(rows * p->width * es);
  if (p->save) {
    f.mean = c.take<float>(rows * 4);
    f.rstd = c.take<float>(rows * 4);
  }
  *bytes = c.at;
  return f;
}
static bool block_ok(const VyFfnBlock* p, const char* who) {
  if (p && p->rows > 0 && p->width > 0 && p->inner > 0 && dtype_ok(p->dtype) && p->h && p->input && p->w1 && p->w2 && p->gamma && p->beta) return true;
  set_error("%s: bad arguments", who);
  return false;
}

// temporaries of the backward calls
struct AttnWork { void *ds, *dattn, *dqkv; float *partials, *dsum, *sums; };
static AttnWork carve_work(const VyAttnBlock* p, void* base, int64_t* bytes) {
  Carve c = {static_cast<char*>(base), 0};
  const int64_t rows = static_cast<int64_t>(p->seqs) * p->tokens, es = dtype_size(p->dtype), nq = (p->heads + 2 * p->kv_heads) * 64;
  AttnWork w;
  w.ds = c.take(rows * p->width * es);
  w.dattn = c.take(rows * p->heads * 64 * 2);
  w.dqkv = c.take(rows * nq * es);
  w.partials = c.take<float>(2LL * vy_norm_bwd_partial_rows() * p->width * 4);
  w.dsum = c.take<float>(rows * p->heads * 4);
  w.sums = c.take<float>(static_cast<int64_t>(vy_colsum_workspace_floats(static_cast<int>(nq))) * 4);
  *bytes = c.at;
  return w;
}
struct FfnWork { void* dz; float *partials, *sums; };
static FfnWork carve_work(const VyFfnBlock* p, void* base, int64_t* bytes) {
  Carve c = {static_cast<char*>(base), 0};
  FfnWork w;
  w.dz = c.take(static_cast<int64_t>(p->rows) * p->inner * dtype_size(p->dtype));
  w.partials = c.take<float>(2LL * vy_norm_bwd_partial_rows() * p->width * 4);
  w.sums = c.take<float>(static_cast<int64_t>(vy_colsum_workspace_floats(p->inner)) * 4);
  *bytes = c.at;
  return w;
}

}  // namespace vy

#define VY_NEED_DEVICE(name)                                        \
  do {                                                              \
    if (!vy_device_ok()) {                                          \
      set_error(name ": no sm_100 device (there is no CPU fallback)"); \
      return VY_ERR_NO_DEVICE;                                      \
    }                                                               \
  } while (0)
#define VY_STEP(call)             \
  do {                            \
    const int rc_ = (call);       \
    if (rc_ != VY_OK) return rc_; \
  } while (0)

extern "C" int64_t vy_attn_block_bytes(const VyAttnBlock* p) {
  int64_t n = 0;
  if (vy::block_ok(p, "vy_attn_block_bytes")) vy::carve(p, nullptr, &n);
  return n;
}
extern "C" int64_t vy_attn_block_work_bytes(const VyAttnBlock* p) {
  int64_t n = 0;
  if (vy::block_ok(p, "vy_attn_block_work_bytes")) vy::carve_work(p, nullptr, &n);
  return n;
}
extern "C" int64_t vy_ffn_block_bytes(const VyFfnBlock* p) {
  int64_t n = 0;
  if (vy::block_ok(p, "vy_ffn_block_bytes")) vy::carve(p, nullptr, &n);
  return n;
}
extern "C" int64_t vy_ffn_block_work_bytes(const VyFfnBlock* p) {
  int64_t n = 0;
  if (vy::block_ok(p, "vy_ffn_block_work_bytes")) vy::carve_work(p, nullptr, &n);
  return n;
}

extern "C" int vy_attn_block_fwd(const VyAttnBlock* p) {
  using namespace vy;
  VY_NEED_DEVICE("vy_attn_block_fwd");
  if (!block_ok(p, "vy_attn_block_fwd")) return VY_ERR_INVALID_ARG;
  int64_t bytes = 0;
  const AttnParts a = carve(p, p->scratch, &bytes);
  VY_CHECK_ARG(p->y && p->scratch && p->scratch_bytes >= bytes, "vy_attn_block_fwd: %lld bytes of scratch, %lld needed", (long long)p->scratch_bytes, (long long)bytes);
  const int rows = p->seqs * p->tokens, hq = p->heads * 64, nq = (p->heads + 2 * p->kv_heads) * 64;
  if (p->decode) {
    VY_STEP(linear({rows, nq, p->width, p->dtype, VY_ACT_NONE, p->hint_qkv, p->weights_static, p->x, p->w_qkv, p->b_qkv, nullptr, nullptr, a.qkv, p->stream}));
    VyDecode d = decode_args(p, a);
    d.splits = vy_attn_decode_plan(&d);
    d.workspace = a.split;
    VY_STEP(vy_attn_decode(&d));
  } else {
    VyGemm g;
    memset(&g, 0, sizeof(g));
    g.M = rows;
    g.N = nq;
    g.K = p->width;
    g.in_dtype = p->dtype;
    g.A = p->x;
    g.B = p->w_qkv;
    g.lda = g.ldb = p->width;
    g.epi = VY_EPI_QKV_ROPE;
    g.bias = p->b_qkv;
    g.bias_dtype = p->dtype;
    g.out_dtype = g.kv_out_dtype = VY_BF16;
    g.tokens_per_seq = p->tokens;
    g.start_pos = p->rope_pos;
    g.kv_dst_pos0 = p->k_cache ? p->start : 0;
    g.head_dim = 64;
    g.n_q_heads = p->heads;
    g.n_kv_heads = p->kv_heads;
    g.rope_cos = p->rope_cos;
    g.rope_sin = p->rope_sin;
    g.rope_rows = p->rope_rows;
    g.kv_cap = p->k_cache ? p->cache_len : p->tokens;
    VyAttn t;
    attn_args(p, a, t);
    g.q_out = a.q;
    g.q_sb = t.q_sb;
    g.q_sh = t.q_sh;
    g.q_sl = t.q_sl;
    g.k_out = const_cast<void*>(t.k);
    g.v_out = const_cast<void*>(t.v);
    g.k_sb = g.v_sb = t.k_sb;
    g.k_sh = g.v_sh = t.k_sh;
    g.k_sl = g.v_sl = t.k_sl;
    g.stream = p->stream;
    set_hint(g, p->hint_qkv);
    VY_STEP(vy_gemm(&g));
    VY_STEP(vy_attn_fwd(&t));
  }
  VY_STEP(linear({rows, p->width, hq, p->dtype, VY_ACT_NONE, p->hint_out, p->weights_static, a.attn, p->w_out, p->b_out, p->x, nullptr, a.s, p->stream}));
  return norm(rows, p->width, p->dtype, a.s, p->gamma, p->beta, p->eps, p->y, a.mean, a.rstd, p->stream);
}

extern "C" int vy_attn_block_bwd(const VyAttnBlock* p) {
  using namespace vy;
  VY_NEED_DEVICE("vy_attn_block_bwd");
  if (!block_ok(p, "vy_attn_block_bwd")) return VY_ERR_INVALID_ARG;
  int64_t bytes = 0, work = 0;
  const AttnParts a = carve(p, p->scratch, &bytes);
  const AttnWork w = carve_work(p, p->work, &work);
  VY_CHECK_ARG(p->save && !p->decode && p->scratch && p->scratch_bytes >= bytes && p->work && p->work_bytes >= work && p->dy && p->dx && p->dw_qkv && p->dw_out && p->dgamma && p->dbeta,
               "vy_attn_block_bwd: bad arguments");
  const int rows = p->seqs * p->tokens, hq = p->heads * 64, hk = p->kv_heads * 64, nq = hq + 2 * hk;
  VY_STEP(norm_bwd(rows, p->width, p->dtype, p->dy, a.s, p->gamma, a.mean, a.rstd, w.ds, p->dgamma, p->dbeta, p->db_out, w.partials, p->stream));
  VY_STEP(wgrad(rows, p->width, hq, p->dtype, w.ds, a.attn, p->dw_out, p->split_ws, p->split_bytes, p->hint_dw_out, p->stream));
  VY_STEP(dgrad(rows, p->width, hq, p->dtype, w.ds, p->w_out, nullptr, VY_ACT_NONE, nullptr, w.dattn, VY_BF16, p->hint_d_out, p->stream));
  VyAttn t;
  attn_args(p, a, t);
  VyAttnBwd b;
  memset(&b, 0, sizeof(b));
  b.B = t.B;
  b.n_q_heads = t.n_q_heads;
  b.n_kv_heads = t.n_kv_heads;
  b.head_dim = 64;
  b.Sq = t.Sq;
  b.Skv = t.Skv;
  b.q = t.q; b.q_sb = t.q_sb; b.q_sh = t.q_sh; b.q_sl = t.q_sl;
  b.k = t.k; b.k_sb = t.k_sb; b.k_sh = t.k_sh; b.k_sl = t.k_sl;
  b.v = t.v; b.v_sb = t.v_sb; b.v_sh = t.v_sh; b.v_sl = t.v_sl;
  b.o = a.attn; b.o_sb = t.o_sb; b.o_sl = t.o_sl; b.o_dtype = p->dtype;
  b.dout = w.dattn; b.do_sb = t.o_sb; b.do_sl = t.o_sl;
  b.lse = a.lse;
  b.dsum = w.dsum;
  b.causal = t.causal;
  b.q_pos0 = t.q_pos0;
  b.key_padding_mask = t.key_padding_mask;
  b.kpm_stride = t.kpm_stride;
  b.rope_cos = p->rope_cos;
  b.rope_sin = p->rope_sin;
  b.rope_pos0 = p->rope_pos;
  char* dqkv = static_cast<char*>(w.dqkv);
  b.dq = dqkv;
  b.dk = dqkv + static_cast<int64_t>(hq) * dtype_size(p->dtype);
  b.dv = dqkv + static_cast<int64_t>(hq + hk) * dtype_size(p->dtype);
  b.ld_dq = b.ld_dk = b.ld_dv = nq;
  b.out_dtype = p->dtype;
  b.stream = p->stream;
  VY_STEP(vy_attn_bwd(&b));
  VY_STEP(dgrad(rows, nq, p->width, p->dtype, w.dqkv, p->w_qkv, w.ds, VY_ACT_NONE, nullptr, p->dx, p->dtype, p->hint_d_qkv, p->stream));
  VY_STEP(wgrad(rows, nq, p->width, p->dtype, w.dqkv, p->x, p->dw_qkv, p->split_ws, p->split_bytes, p->hint_dw_qkv, p->stream));
  return p->db_qkv ? vy_colsum(rows, nq, w.dqkv, nq, p->dtype, p->db_qkv, p->dtype, 0, 1.f, w.sums, p->stream) : VY_OK;
}

extern "C" int vy_ffn_block_fwd(const VyFfnBlock* p) {
  using namespace vy;
  VY_NEED_DEVICE("vy_ffn_block_fwd");
  if (!block_ok(p, "vy_ffn_block_fwd")) return VY_ERR_INVALID_ARG;
  int64_t bytes = 0;
  const FfnParts f = carve(p, p->scratch, &bytes);
  VY_CHECK_ARG(p->y && p->scratch && p->scratch_bytes >= bytes, "vy_ffn_block_fwd: %lld bytes of scratch, %lld needed", (long long)p->scratch_bytes, (long long)bytes);
  VY_STEP(linear({p->rows, p->inner, p->width, p->dtype, p->act, p->hint_1, p->weights_static, p->h, p->w1, p->b1, nullptr, f.z, f.a, p->stream}));
  VY_STEP(linear({p->rows, p->width, p->inner, p->dtype, VY_ACT_NONE, p->hint_2, p->weights_static, f.a, p->w2, p->b2, p->input, nullptr, f.s, p->stream}));
  return norm(p->rows, p->width, p->dtype, f.s, p->gamma, p->beta, p->eps, p->y, f.mean, f.rstd, p->stream);
}

extern "C" int vy_ffn_block_bwd(const VyFfnBlock* p) {
  using namespace vy;
  VY_NEED_DEVICE("vy_ffn_block_bwd");
  if (!block_ok(p, "vy_ffn_block_bwd")) return VY_ERR_INVALID_ARG;
  int64_t bytes = 0, work = 0;
  const FfnParts f = carve(p, p->scratch, &bytes);
  const FfnWork w = carve_work(p, p->work, &work);
  VY_CHECK_ARG(p->save && p->scratch && p->scratch_bytes >= bytes && p->work && p->work_bytes >= work && p->dy && p->dh && p->d_input && p->dw1 && p->dw2 && p->dgamma && p->dbeta,
               "vy_ffn_block_bwd: bad arguments");
  VY_STEP(norm_bwd(p->rows, p->width, p->dtype, p->dy, f.s, p->gamma, f.mean, f.rstd, p->d_input, p->dgamma, p->dbeta, p->db2, w.partials, p->stream));
  VY_STEP(wgrad(p->rows, p->width, p->inner, p->dtype, p->d_input, f.a, p->dw2, p->split_ws, p->split_bytes, p->hint_dw2, p->stream));
  VY_STEP(dgrad(p->rows, p->width, p->inner, p->dtype, p->d_input, p->w2, nullptr, p->dact, f.z, w.dz, p->dtype, p->hint_d2, p->stream));
  VY_STEP(wgrad(p->rows, p->inner, p->width, p->dtype, w.dz, p->h, p->dw1, p->split_ws, p->split_bytes, p->hint_dw1, p->stream));
  if (p->db1) VY_STEP(vy_colsum(p->rows, p->inner, w.dz, p->inner, p->dtype, p->db1, p->dtype, 0, 1.f, w.sums, p->stream));
  return dgrad(p->rows, p->inner, p->width, p->dtype, w.dz, p->w1, nullptr, VY_ACT_NONE, nullptr, p->dh, p->dtype, p->hint_d1, p->stream);
}
