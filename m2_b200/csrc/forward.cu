// Whole modules in one call: the launches of the mixer, of the GLU MLP and of the encoder one after the other, with the
// buffers between them.  A forward of twelve layers is 73 launches; called one by one from Python they cost 37 us each
// (argument checks, output allocation, ctypes marshalling), 2.9 ms where the GPU needs less than one for a small batch.
//
// Computation replaced: bert/src/mm/monarch_mixer_sequence_mixer.py:100-154, bert/src/bert_layers.py:186-252, :482-508
// and :552-813 of the reference.
#include "common.cuh"

namespace m2 {

static long long round_up(long long n, long long m) { return (n + m - 1) / m * m; }

// Buffers of one encoder layer inside a workspace, in bytes from its start (every one on a 256-byte boundary).
struct Layout {
  long long rows, stride;                       // padded tokens; distance of two channels of a time-contiguous tensor
  size_t aug, tm, xin, conv, mix, h, o, total;
};
// The split weights of float32 layers: in_linear's and out_linear's, or the GLU's and wo's, one behind the other.
static size_t split_bytes(long long rows, int p) { return (size_t)round_up((long long)m2_split_weights_bytes(rows, p), 256); }
static size_t mixer_split_bytes(int d_model) { return split_bytes(3LL * d_model, d_model) + split_bytes(d_model, d_model); }
static size_t mlp_split_bytes(int d_model, int inter, int nblocks) {
  return split_bytes(2LL * inter, d_model / nblocks) + split_bytes(d_model, inter / nblocks);
}

static Layout layout_of(int batch, int pitch, int d_model, int inter, bool f32) {
  Layout l;
  l.rows = (long long)batch * pitch;
  l.stride = round_up(l.rows, 16);
  size_t at = 0;
  const int size = f32 ? 4 : 2;
  auto take = [&](long long elements) { const size_t p = at; at += (size_t)round_up(size * elements, 256); return p; };
  l.aug = take(f32 ? 0 : l.rows * d_model);      // float32 layers read each other's output as it is
  l.tm = take(f32 ? 0 : l.stride * d_model);
  l.mix = take(l.rows * d_model);
  l.o = take(l.rows * d_model);
  l.xin = l.h = at;                             // in_linear's and the conv's results are dead when the GLU writes h
  take(3 * l.stride * d_model);
  l.conv = take(l.stride * d_model);
  const size_t h_end = l.h + (size_t)round_up(size * l.rows * inter, 256);
  l.total = at > h_end ? at : h_end;
  return l;
}

// The weights that a call's float32 GEMMs take split: written to the call's workspace, ahead of the GEMMs, from what the weights hold
// when the call runs (also when it runs as part of a graph).
static void* split_at(void* split, size_t skip) { return split ? static_cast<unsigned char*>(split) + skip : nullptr; }
struct SplitWork {
  WeightRows rows[4];
  int n = 0;
  void add(bool used, const void* w, long long r, int p, const void* out) { if (used) rows[n++] = {w, r, p, const_cast<void*>(out)}; }
  int launch(long long elements, void* stream) const {
    return n ? split_weights_launch(rows, n, elements, static_cast<cudaStream_t>(stream)) : M2_OK;
  }
};

// in_linear and out_linear of the mixer on float32 token rows
static void mixer_linears(const m2_mixer_args* a, m2_linear_args& in, m2_linear_args& out, SplitWork& work) {
  const int L = a->seq_len, D = a->d_model;
  memset(&in, 0, sizeof(in));
  in.batch = a->batch; in.seq_len = L; in.in_features = D; in.dtype = M2_F32;
  in.x_sb = (long long)L * D; in.x_st = D; in.x_sc = in.out_sc = 1;
  out = in;
  in.x = a->x; in.w = a->w_in; in.bias = a->b_in; in.w_split = a->split;
  in.out = a->xin; in.out_features = 3 * D; in.out_sb = 3LL * L * D; in.out_st = 3LL * D;
  out.x = a->conv; out.w = a->w_out; out.bias = a->b_out; out.w_split = split_at(a->split, split_bytes(3LL * D, D));
  out.out = a->out; out.out_features = D; out.out_sb = (long long)L * D; out.out_st = D;
  work.add(linear_split_supported(&in), in.w, 3LL * D, D, in.w_split);
  work.add(linear_split_supported(&out), out.w, D, D, out.w_split);
}

static int mixer_f32(const m2_mixer_args* a, const m2_linear_args& in, const m2_linear_args& out, void* stream) {
  const int L = a->seq_len, D = a->d_model;
  int rc;
  if ((rc = m2_linear_fwd(&in, stream))) return rc;
  m2_longconv_args c;
  memset(&c, 0, sizeof(c));
  c.batch = a->batch; c.seq_len = L; c.d_model = D; c.n_filters = a->n_filters; c.kind = 0;
  c.act_dtype = M2_F32; c.u_dtype = M2_F32;
  c.xin = a->xin; c.xin_sb = 3LL * L * D; c.xin_st = 3LL * D; c.xin_sc = 1;
  c.u = a->x; c.u_sb = (long long)L * D; c.u_st = D; c.u_sc = 1;
  c.out = a->conv; c.out_sb = (long long)L * D; c.out_st = D; c.out_sc = 1;
  c.short_w = a->short_w; c.short_b = a->short_b;
  for (int f = 0; f < 2; ++f) { c.spec[f] = a->spec[f]; c.bias[f] = a->bias[f]; }
  if ((rc = m2_longconv_fwd(&c, stream))) return rc;
  return m2_linear_fwd(&out, stream);
}

// The two GEMMs of the MLP
static void mlp_blocks(const m2_mlp_args* a, m2_glu_args& g, m2_blockdiag_args& w, SplitWork& work) {
  const int p = a->d_model / a->nblocks;
  memset(&g, 0, sizeof(g));
  g.m = a->m; g.d_model = a->d_model; g.inter = a->inter; g.nblocks = a->nblocks; g.dtype = a->f32 ? M2_F32 : M2_BF16;
  g.x = a->x; g.ldx = a->d_model; g.wg = a->wg; g.h = a->h; g.ldh = a->inter;
  memset(&w, 0, sizeof(w));
  w.m = a->m; w.nblocks = a->nblocks; w.p = a->inter / a->nblocks; w.q = p;
  w.in_features = a->inter; w.out_features = a->d_model; w.dtype = g.dtype;
  w.x = a->h; w.ldx = a->inter; w.w = a->wo; w.bias = a->wo_bias; w.out = a->o; w.ldo = a->d_model;
  if (!a->f32) return;
  g.wg_split = a->split;
  w.w_split = split_at(a->split, split_bytes(2LL * a->inter, p));
  work.add(glu_split_supported(&g), g.wg, 2LL * a->inter, p, g.wg_split);
  work.add(blockdiag_split_supported(&w), w.w, a->d_model, w.p, w.w_split);
}

static int mlp_run(const m2_mlp_args* a, const m2_glu_args& g, const m2_blockdiag_args& w, void* stream) {
  int rc;
  if ((rc = m2_blockdiag_glu_fwd(&g, stream))) return rc;
  if ((rc = m2_blockdiag_fwd(&w, stream))) return rc;
  m2_add_layernorm_args n;
  memset(&n, 0, sizeof(n));
  n.m = a->m; n.n = a->d_model; n.in_dtype = g.dtype; n.out_dtype = M2_F32;
  n.a = a->o; n.lda = a->d_model; n.b = a->x; n.ldb = a->d_model;
  n.weight = a->ln_w; n.bias = a->ln_b; n.eps = a->eps;
  n.out = a->out; n.ldo = a->d_model;
  n.out_bf16 = a->out_bf16; n.ld_bf16 = a->d_model;
  n.out_tm_f16 = a->out_tm_f16; n.tm_sb = a->seq_len; n.tm_sc = a->tm_stride;
  n.seq_len = a->seq_len; n.valid_len = a->valid_len;
  return m2_add_layernorm_fwd(&n, stream);
}

}  // namespace m2

extern "C" int m2_mixer_fwd(const m2_mixer_args* a, void* stream) {
  M2_REQUIRE(a != nullptr, M2_ERR_ARG, "m2_mixer_fwd: args is NULL");
  M2_REQUIRE(a->batch >= 0 && a->seq_len > 0 && a->d_model > 0 && (a->f32 ? a->pitch == a->seq_len : a->pitch >= a->seq_len && a->pitch % 8 == 0) &&
             (a->out_pitch == a->pitch || a->out_pitch == a->seq_len) && a->stride >= (long long)a->batch * a->pitch, M2_ERR_ARG,
             "m2_mixer_fwd: bad sizes batch=%d seq_len=%d pitch=%d out_pitch=%d d_model=%d", a->batch, a->seq_len, a->pitch, a->out_pitch, a->d_model);
  M2_REQUIRE(a->f32 ? a->kind == 0 : a->kind >= 2 && a->kind <= 4, M2_ERR_UNSUPPORTED,
             "m2_mixer_fwd: kind must be 2, 3 or 4 (time-contiguous rows), or 0 in float32");
  if (a->batch == 0) return M2_OK;
  if (a->f32) {
    m2::SplitWork work;
    m2_linear_args in, out;
    m2::mixer_linears(a, in, out, work);
    const int rc = work.launch((long long)a->batch * a->seq_len * a->d_model, stream);
    return rc ? rc : m2::mixer_f32(a, in, out, stream);
  }
  const int rows = a->batch * a->pitch;
  int rc;
  m2_linear_args in;
  memset(&in, 0, sizeof(in));
  in.batch = 1; in.seq_len = rows; in.in_features = a->d_model; in.out_features = 3 * a->d_model; in.dtype = M2_BF16;
  in.x = a->x; in.x_sb = (long long)rows * a->d_model; in.x_st = a->d_model; in.x_sc = 1;
  in.w = a->w_in; in.bias = a->b_in;
  in.out = a->xin; in.out_sb = 3LL * a->d_model * a->stride; in.out_st = 1; in.out_sc = a->stride;
  if ((rc = m2_linear_fwd(&in, stream))) return rc;
  m2_longconv_args c;
  memset(&c, 0, sizeof(c));
  c.batch = a->batch; c.seq_len = a->seq_len; c.d_model = a->d_model; c.n_filters = a->n_filters; c.kind = a->kind;
  c.act_dtype = M2_BF16; c.u_dtype = M2_F16; c.bf16_rounding = 1;
  c.xin = a->xin; c.xin_sb = a->pitch; c.xin_st = 1; c.xin_sc = a->stride;
  c.u = a->u; c.u_sb = a->pitch; c.u_st = 1; c.u_sc = a->u_stride;
  c.out = a->conv; c.out_sb = a->pitch; c.out_st = 1; c.out_sc = a->stride;
  c.short_w = a->short_w; c.short_b = a->short_b;
  for (int f = 0; f < 2; ++f) { c.spec[f] = a->spec[f]; c.bias[f] = a->kind == 2 ? a->bias[f] : nullptr; }
  c.yu_bf16 = a->yu_bf16;
  if ((rc = m2_longconv_fwd(&c, stream))) return rc;
  m2_linear_args out;
  memset(&out, 0, sizeof(out));
  const bool flat = a->out_pitch == a->pitch;   // one long row of tokens, or the steps of each sequence without its padding
  out.batch = flat ? 1 : a->batch; out.seq_len = flat ? rows : a->seq_len;
  out.in_features = a->d_model; out.out_features = a->d_model; out.dtype = M2_BF16;
  out.x = a->conv; out.x_sb = a->pitch; out.x_st = 1; out.x_sc = a->stride;
  out.w = a->w_out; out.bias = a->b_out;
  out.out = a->out; out.out_sb = (long long)a->out_pitch * a->d_model; out.out_st = a->d_model; out.out_sc = 1;
  return m2_linear_fwd(&out, stream);
}

extern "C" int m2_mlp_fwd(const m2_mlp_args* a, void* stream) {
  M2_REQUIRE(a != nullptr, M2_ERR_ARG, "m2_mlp_fwd: args is NULL");
  M2_REQUIRE(a->m >= 0 && a->d_model > 0 && a->inter > 0 && a->nblocks > 0, M2_ERR_ARG, "m2_mlp_fwd: bad sizes");
  M2_REQUIRE(a->d_model % a->nblocks == 0 && a->inter % a->nblocks == 0, M2_ERR_UNSUPPORTED,
             "m2_mlp_fwd: d_model and inter must be multiples of nblocks");
  if (a->m == 0) return M2_OK;
  m2::SplitWork work;
  m2_glu_args g;
  m2_blockdiag_args w;
  m2::mlp_blocks(a, g, w, work);
  const int rc = work.launch((long long)a->m * a->d_model, stream);
  return rc ? rc : m2::mlp_run(a, g, w, stream);
}

extern "C" long long m2_mixer_split_bytes(int d_model) { return d_model > 0 ? (long long)m2::mixer_split_bytes(d_model) : 0; }

extern "C" long long m2_mlp_split_bytes(int d_model, int inter, int nblocks) {
  return d_model > 0 && inter > 0 && nblocks > 0 ? (long long)m2::mlp_split_bytes(d_model, inter, nblocks) : 0;
}

extern "C" long long m2_encoder_workspace(int batch, int pitch, int d_model, int inter) {
  if (batch <= 0 || pitch <= 0 || d_model <= 0 || inter <= 0) return 0;
  return (long long)m2::layout_of(batch, pitch, d_model, inter, false).total;
}

// behind the activations the split weights of one layer, written again for the next
static size_t m2_f32_activations(int batch, int seq_len, int d_model, int inter) {
  return (size_t)m2::round_up((long long)m2::layout_of(batch, seq_len, d_model, inter, true).total, 256);
}
extern "C" long long m2_encoder_workspace_f32(int batch, int seq_len, int d_model, int inter, int nblocks) {
  if (batch <= 0 || seq_len <= 0 || d_model <= 0 || inter <= 0 || nblocks <= 0) return 0;
  return (long long)(m2_f32_activations(batch, seq_len, d_model, inter) + m2::mixer_split_bytes(d_model) + m2::mlp_split_bytes(d_model, inter, nblocks));
}

// The layers in float32, from the embeddings' output.
static int encoder_f32(const m2_encoder_args* a, void* stream) {
  using namespace m2;
  M2_REQUIRE(a->x && a->kind == 0, M2_ERR_ARG, "m2_encoder_fwd: float32 layers need x and kind 0");
  M2_REQUIRE((long long)a->batch * a->seq_len < (1LL << 31) - 512, M2_ERR_UNSUPPORTED, "m2_encoder_fwd: more than 2^31 tokens");
  M2_REQUIRE(a->nblocks > 0 && a->d_model % a->nblocks == 0 && a->inter % a->nblocks == 0, M2_ERR_UNSUPPORTED,
             "m2_encoder_fwd: d_model and inter must be multiples of nblocks");
  const Layout l = layout_of(a->batch, a->seq_len, a->d_model, a->inter, true);
  unsigned char* ws = static_cast<unsigned char*>(a->workspace);
  unsigned char* split = ws + m2_f32_activations(a->batch, a->seq_len, a->d_model, a->inter);
  const float* in = a->x;
  for (int i = 0; i < a->n_layers; ++i, in = a->out) {         // a layer's input is dead when its MLP writes the output
    const m2_encoder_layer& y = a->layers[i];
    m2_mixer_args x;
    memset(&x, 0, sizeof(x));
    x.batch = a->batch; x.seq_len = x.pitch = x.out_pitch = a->seq_len; x.d_model = a->d_model; x.n_filters = a->n_filters; x.f32 = 1;
    x.x = in; x.w_in = y.w_in; x.b_in = y.b_in; x.short_w = y.short_w; x.short_b = y.short_b;
    for (int f = 0; f < 2; ++f) { x.spec[f] = y.spec[f]; x.bias[f] = y.bias[f]; }
    x.w_out = y.w_out; x.b_out = y.b_out; x.split = split;
    x.xin = ws + l.xin; x.conv = ws + l.conv; x.stride = l.stride; x.out = ws + l.mix;
    m2_mlp_args p;
    memset(&p, 0, sizeof(p));
    p.m = (int)l.rows; p.d_model = a->d_model; p.inter = a->inter; p.nblocks = a->nblocks; p.f32 = 1;
    p.x = ws + l.mix; p.wg = y.wg; p.wo = y.wo; p.wo_bias = y.wo_bias; p.ln_w = y.ln_w; p.ln_b = y.ln_b; p.eps = y.eps;
    p.split = split + mixer_split_bytes(a->d_model);
    p.h = ws + l.h; p.o = ws + l.o; p.out = a->out;
    SplitWork work;
    m2_linear_args first, second;
    m2_glu_args g;
    m2_blockdiag_args w;
    mixer_linears(&x, first, second, work);
    mlp_blocks(&p, g, w, work);
    int rc;
    if ((rc = work.launch(l.rows * a->d_model, stream))) return rc;
    if ((rc = mixer_f32(&x, first, second, stream))) return rc;
    if ((rc = mlp_run(&p, g, w, stream))) return rc;
  }
  return M2_OK;
}

// The mixer of one layer where the convolution runs in float32 (kind 0): token rows throughout, the layer input u float32.
static int mixer_rows(const m2_encoder_args* a, const m2_encoder_layer& y, const void* x, const float* u, void* xin, void* conv, void* out,
                      void* stream) {
  const int rows = a->batch * a->seq_len, D = a->d_model;
  m2_linear_args p;
  memset(&p, 0, sizeof(p));
  p.batch = 1; p.seq_len = rows; p.in_features = D; p.out_features = 3 * D; p.dtype = M2_BF16;
  p.x = x; p.x_sb = (long long)rows * D; p.x_st = D; p.x_sc = 1;
  p.w = y.w_in; p.bias = y.b_in;
  p.out = xin; p.out_sb = 3LL * rows * D; p.out_st = 3LL * D; p.out_sc = 1;
  int rc;
  if ((rc = m2_linear_fwd(&p, stream))) return rc;
  m2_longconv_args c;
  memset(&c, 0, sizeof(c));
  c.batch = a->batch; c.seq_len = a->seq_len; c.d_model = D; c.n_filters = a->n_filters; c.kind = 0;
  c.act_dtype = M2_BF16; c.u_dtype = M2_F32; c.bf16_rounding = 1;
  c.xin = xin; c.xin_sb = 3LL * a->seq_len * D; c.xin_st = 3LL * D; c.xin_sc = 1;
  c.u = u; c.u_sb = (long long)a->seq_len * D; c.u_st = D; c.u_sc = 1;
  c.out = conv; c.out_sb = (long long)a->seq_len * D; c.out_st = D; c.out_sc = 1;
  c.short_w = y.short_w; c.short_b = y.short_b;
  for (int f = 0; f < 2; ++f) { c.spec[f] = y.spec[f]; c.bias[f] = y.bias[f]; }
  if ((rc = m2_longconv_fwd(&c, stream))) return rc;
  p.x = conv; p.out_features = D; p.w = y.w_out; p.bias = y.b_out;
  p.out = out; p.out_sb = (long long)rows * D; p.out_st = D;
  return m2_linear_fwd(&p, stream);
}

extern "C" int m2_encoder_fwd(const m2_encoder_args* a, void* stream) {
  using namespace m2;
  M2_REQUIRE(a != nullptr, M2_ERR_ARG, "m2_encoder_fwd: args is NULL");
  M2_REQUIRE(a->batch > 0 && a->seq_len > 0 && a->n_layers > 0 && a->d_model > 0 && a->inter > 0, M2_ERR_ARG, "m2_encoder_fwd: bad sizes");
  M2_REQUIRE(a->layers && a->workspace && a->out && m2_aligned(a->workspace, 256), M2_ERR_ARG,
             "m2_encoder_fwd: NULL pointer or workspace not on a 256-byte boundary");
  if (a->f32) return encoder_f32(a, stream);
  M2_REQUIRE(a->kind == 0 || (a->kind >= 2 && a->kind <= 4), M2_ERR_UNSUPPORTED, "m2_encoder_fwd: kind must be 0, 2, 3 or 4");
  const bool rows = a->kind == 0;               // float32 convolution: token rows without padding, float32 layer inputs in `out`
  const int pitch = rows ? a->seq_len : (int)round_up(a->seq_len, 8), D = a->d_model;
  M2_REQUIRE((long long)a->batch * pitch < (1LL << 31) - 512, M2_ERR_UNSUPPORTED, "m2_encoder_fwd: more than 2^31 tokens");
  const Layout l = layout_of(a->batch, pitch, D, a->inter, false);
  unsigned char* ws = static_cast<unsigned char*>(a->workspace);
  int rc;
  m2_embed_layernorm_args e = a->embed;
  e.m = (int)l.rows; e.n = D; e.out = rows ? a->out : nullptr; e.ldo = D;
  e.out_bf16 = ws + l.aug; e.ld_bf16 = D; e.bf16_pad_cols = 0;
  e.out_tm_f16 = rows ? nullptr : ws + l.tm; e.tm_sb = pitch; e.tm_sc = l.stride; e.seq_len = pitch; e.valid_len = a->seq_len;
  if ((rc = m2_embed_layernorm_fwd(&e, stream))) return rc;
  for (int i = 0; i < a->n_layers; ++i) {
    const m2_encoder_layer& y = a->layers[i];
    if (rows) {
      if ((rc = mixer_rows(a, y, ws + l.aug, a->out, ws + l.xin, ws + l.conv, ws + l.mix, stream))) return rc;
    } else {
      m2_mixer_args x;
      memset(&x, 0, sizeof(x));
      x.batch = a->batch; x.seq_len = a->seq_len; x.pitch = pitch; x.out_pitch = pitch; x.d_model = D;
      x.kind = a->kind; x.n_filters = a->n_filters;
      x.x = ws + l.aug; x.u = ws + l.tm; x.u_stride = l.stride;
      x.w_in = y.w_in; x.b_in = y.b_in; x.short_w = y.short_w; x.short_b = y.short_b;
      for (int f = 0; f < 2; ++f) { x.spec[f] = y.spec[f]; x.bias[f] = y.bias[f]; }
      x.w_out = y.w_out; x.b_out = y.b_out;
      x.xin = ws + l.xin; x.conv = ws + l.conv; x.stride = l.stride; x.out = ws + l.mix;
      if ((rc = m2_mixer_fwd(&x, stream))) return rc;
    }
    m2_mlp_args p;
    memset(&p, 0, sizeof(p));
    const bool last = i + 1 == a->n_layers;
    p.m = (int)l.rows; p.d_model = D; p.inter = a->inter; p.nblocks = a->nblocks;
    p.x = ws + l.mix; p.wg = y.wg; p.wo = y.wo; p.wo_bias = y.wo_bias; p.ln_w = y.ln_w; p.ln_b = y.ln_b; p.eps = y.eps;
    p.h = ws + l.h; p.o = ws + l.o;
    p.seq_len = pitch; p.valid_len = a->seq_len;
    if (last || rows) p.out = a->out;
    if (!last) p.out_bf16 = ws + l.aug;         // only the next mixer reads this output, through its two copies
    if (!last && !rows) { p.out_tm_f16 = ws + l.tm; p.tm_stride = l.stride; }
    if ((rc = m2_mlp_fwd(&p, stream))) return rc;
  }
  return M2_OK;
}
