// Entry points of the fused gated long convolution: kernel-family selection, filter
// spectrum tables, argument validation.
#include "common.cuh"

namespace m2 {
int longconv_simt_launch(const m2_longconv_args* a, cudaStream_t st);
int spectrum_kind0_launch(int D, int L, const float* k, float* spec, cudaStream_t st);
int longconv_tc_supported(int seq_len, m2_dtype act_dtype, int d_model);
size_t spectrum_kind1_floats(int D, int L);
int spectrum_kind1_launch(int D, int L, const float* k, float* spec, cudaStream_t st);
int longconv_tc_launch(const m2_longconv_args* a, cudaStream_t st);
int longconv_tcl_supported(int seq_len, m2_dtype act_dtype);
size_t spectrum_kind2_floats(int D, int L);
int spectrum_kind2_launch(int D, int L, const float* k, float* spec, cudaStream_t st);
int longconv_tcl_launch(const m2_longconv_args* a, cudaStream_t st);
int longconv_tz_supported(int batch, int seq_len, m2_dtype act_dtype);
size_t spectrum_kind3_floats(int D, int L);
int spectrum_kind3_launch(int D, int L, const float* k, const float* bias, float* spec, cudaStream_t st);
int longconv_tz_launch(const m2_longconv_args* a, cudaStream_t st);
int longconv_bt_supported(int seq_len, m2_dtype act_dtype);
bool longconv_bt_preferred(int batch, int seq_len, int d_model);
size_t spectrum_kind4_floats(int D, int L);
int spectrum_kind4_launch(int D, int L, const float* k, const float* bias, float* spec, cudaStream_t st);
int longconv_bt_launch(const m2_longconv_args* a, cudaStream_t st);
bool longconv_bts_f32_preferred(int batch, int seq_len, int d_model);
bool longconv_bts_f32_supported(const m2_longconv_args* a);
size_t taps_f32_offset(int D, int L);
size_t taps_f32_floats(int D, int L);
int taps_f32_launch(int D, int L, const float* k, float* taps, cudaStream_t st);
int longconv_bts_f32_launch(const m2_longconv_args* a, cudaStream_t st);
int time_major_f16_launch(const m2_time_major_args* a, cudaStream_t st);
}  // namespace m2

extern "C" int m2_longconv_kind(int seq_len, m2_dtype act_dtype, int d_model) {
  if (m2::longconv_tc_supported(seq_len, act_dtype, d_model)) return 1;
  if (m2::longconv_tcl_supported(seq_len, act_dtype) && seq_len % 4 == 0) return 2;
  return 0;
}

extern "C" int m2_longconv_kind_batch(int batch, int seq_len, m2_dtype act_dtype, int d_model) {
  if (m2::longconv_tz_supported(batch, seq_len, act_dtype)) return 3;
  return m2_longconv_kind(seq_len, act_dtype, d_model);
}

extern "C" int m2_longconv_pick(int batch, int seq_len, m2_dtype act_dtype, int d_model) {
  if (act_dtype != M2_BF16 || batch <= 0 || d_model <= 0 || seq_len <= 0 || seq_len > 32768) return 0;
  // Tensor-core families hold taps (3, 4) or spectra (2) and the residual input in fp16.  They serve the lengths that no other
  // precision was ever promised for: 65 .. 128 steps of d_model % 128 == 0, batches of 64 and more of 16 .. 128 steps in
  // multiples of 8, and multiples of 4 beyond 128.  All others are computed in float32 throughout (0): against 64-bit arithmetic
  // on the same bf16 input (d_model 768, two filters) the float32 result is off by 1.71e-3 at 37 steps and 1.78e-3 at 1531,
  // nearly all of it the output's own rounding; kinds 3 and 4 by 1.73e-3 at 37, kind 2 by 1.91e-3 at 1531.
  const bool tz = m2::longconv_tz_supported(batch, seq_len, act_dtype);
  // up to 128 steps both families multiply by the same Toeplitz matrix; kind 3 walks tiles of 128 sequences whatever the
  // batch (34 us at D = 768, L = 128, B = 8 .. 64), kind 4 tiles as narrow as the batch (20 us at 8, 27 at 32, 51 at 64;
  // all launched alone with the L2 flushed)
  if (m2::longconv_tc_supported(seq_len, act_dtype, d_model)) return batch >= 48 ? 3 : 4;
  if (seq_len <= 128) return tz ? 3 : 0;
  if (seq_len % 4 != 0) return 0;
  if (m2::longconv_bt_supported(seq_len, act_dtype) && m2::longconv_bt_preferred(batch, seq_len, d_model)) return 4;
  return 2;
}

extern "C" int m2_longconv_padded(int batch, int seq_len, int d_model) {
  return batch > 0 && seq_len > 0 && d_model > 0 && m2::longconv_bts_f32_preferred(batch, seq_len, d_model);
}

extern "C" size_t m2_filter_spectrum_floats(int kind, int d_model, int seq_len) {
  if (d_model <= 0 || seq_len <= 0) return 0;
  if (kind == 3) return m2::spectrum_kind3_floats(d_model, seq_len);
  if (kind == 4) return m2::spectrum_kind4_floats(d_model, seq_len);
  if (kind == 1) return m2::spectrum_kind1_floats(d_model, seq_len);
  if (kind == 2) return m2::spectrum_kind2_floats(d_model, seq_len);
  return m2::taps_f32_offset(d_model, seq_len) + m2::taps_f32_floats(d_model, seq_len);
}

extern "C" int m2_filter_spectrum_bias(int kind, int d_model, int seq_len, const float* k, const float* bias,
                                       float* spec_out, void* stream) {
  if (kind != 3 && kind != 4) {
    M2_REQUIRE(bias == nullptr, M2_ERR_ARG,
               "m2_filter_spectrum_bias: only kinds 3 and 4 fold the bias into the table; kind %d takes it in m2_longconv_fwd", kind);
    return m2_filter_spectrum(kind, d_model, seq_len, k, spec_out, stream);
  }
  M2_REQUIRE(d_model > 0 && seq_len > 0, M2_ERR_ARG, "m2_filter_spectrum_bias: sizes must be positive");
  M2_REQUIRE(k && spec_out, M2_ERR_ARG, "m2_filter_spectrum_bias: NULL pointer");
  M2_REQUIRE(m2_aligned(spec_out, 16), M2_ERR_ALIGN, "m2_filter_spectrum_bias: spec_out must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return kind == 4 ? m2::spectrum_kind4_launch(d_model, seq_len, k, bias, spec_out, st)
                   : m2::spectrum_kind3_launch(d_model, seq_len, k, bias, spec_out, st);
}

extern "C" int m2_time_major_f16(const m2_time_major_args* a, void* stream) {
  M2_REQUIRE(a != nullptr, M2_ERR_ARG, "m2_time_major_f16: args is NULL");
  M2_REQUIRE(a->batch >= 0 && a->seq_len > 0 && a->d_model > 0, M2_ERR_ARG, "m2_time_major_f16: bad sizes");
  if (a->batch == 0) return M2_OK;
  M2_REQUIRE(a->src && a->dst, M2_ERR_ARG, "m2_time_major_f16: NULL tensor pointer");
  M2_REQUIRE(a->src_dtype == M2_F32 || a->src_dtype == M2_BF16, M2_ERR_UNSUPPORTED,
             "m2_time_major_f16: src must be float32 or bf16");
  M2_REQUIRE(a->batch <= 65535 && (a->d_model + 63) / 64 <= 65535, M2_ERR_UNSUPPORTED, "m2_time_major_f16: too large");
  return m2::time_major_f16_launch(a, static_cast<cudaStream_t>(stream));
}

extern "C" int m2_filter_spectrum(int kind, int d_model, int seq_len, const float* k, float* spec_out,
                                  void* stream) {
  M2_REQUIRE(d_model > 0 && seq_len > 0, M2_ERR_ARG, "m2_filter_spectrum: sizes must be positive");
  M2_REQUIRE(k && spec_out, M2_ERR_ARG, "m2_filter_spectrum: NULL pointer");
  M2_REQUIRE(m2_aligned(k, 8) && m2_aligned(spec_out, 16), M2_ERR_ALIGN,
             "m2_filter_spectrum: k must be 8-byte and spec_out 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (kind == 3) return m2::spectrum_kind3_launch(d_model, seq_len, k, nullptr, spec_out, st);
  if (kind == 4) return m2::spectrum_kind4_launch(d_model, seq_len, k, nullptr, spec_out, st);
  if (kind == 0) {
    const int rc = m2::spectrum_kind0_launch(d_model, seq_len, k, spec_out, st);
    return rc ? rc : m2::taps_f32_launch(d_model, seq_len, k, spec_out + m2::taps_f32_offset(d_model, seq_len), st);
  }
  if (kind == 1) return m2::spectrum_kind1_launch(d_model, seq_len, k, spec_out, st);
  if (kind == 2) return m2::spectrum_kind2_launch(d_model, seq_len, k, spec_out, st);
  return m2_set_error(M2_ERR_ARG, "m2_filter_spectrum: unknown kind %d", kind);
}

extern "C" int m2_longconv_fwd(const m2_longconv_args* a, void* stream) {
  M2_REQUIRE(a != nullptr, M2_ERR_ARG, "m2_longconv_fwd: args is NULL");
  M2_REQUIRE(a->batch >= 0 && a->seq_len > 0 && a->d_model > 0, M2_ERR_ARG,
             "m2_longconv_fwd: bad sizes batch=%d seq_len=%d d_model=%d", a->batch, a->seq_len, a->d_model);
  M2_REQUIRE(a->n_filters == 1 || a->n_filters == 2, M2_ERR_ARG, "m2_longconv_fwd: n_filters must be 1 or 2");
  M2_REQUIRE(!a->plain || a->n_filters == 1, M2_ERR_ARG, "m2_longconv_fwd: plain mode takes one filter");
  if (a->batch == 0) return M2_OK;
  const bool folded = (a->kind == 3 || a->kind == 4) && !a->plain;   // these have the bias inside their spectrum
  M2_REQUIRE(a->xin && a->out && (a->plain || (a->short_w && a->short_b)) && a->spec[0] && (folded || a->bias[0]), M2_ERR_ARG,
             "m2_longconv_fwd: NULL tensor pointer");
  M2_REQUIRE(a->n_filters == 1 || (a->u && a->spec[1] && (folded || a->bias[1])), M2_ERR_ARG,
             "m2_longconv_fwd: residual filter requested but u/spec[1]/bias[1] is NULL");
  M2_REQUIRE(a->act_dtype == M2_F32 || a->act_dtype == M2_BF16, M2_ERR_UNSUPPORTED, "m2_longconv_fwd: xin and out are float32 or bf16");
  M2_REQUIRE(a->n_filters == 1 || a->u_dtype == M2_F32 || a->u_dtype == M2_BF16 || (a->u_dtype == M2_F16 && a->kind >= 2), M2_ERR_UNSUPPORTED,
             "m2_longconv_fwd: u is float32 or bf16, fp16 for kinds 2, 3 and 4 only");
  M2_REQUIRE(a->xin_st == 1 || a->xin_sc == 1, M2_ERR_UNSUPPORTED,
             "m2_longconv_fwd: xin must be contiguous along time or along channels");
  M2_REQUIRE(a->batch <= 65535, M2_ERR_UNSUPPORTED, "m2_longconv_fwd: batch > 65535");
  M2_REQUIRE(m2_aligned(a->spec[0], 16) && (a->n_filters == 1 || m2_aligned(a->spec[1], 16)), M2_ERR_ALIGN,
             "m2_longconv_fwd: spectrum tables must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a->kind == 0 && m2::longconv_bts_f32_supported(a)) return m2::longconv_bts_f32_launch(a, st);
  if (a->kind == 0 || a->plain) return m2::longconv_simt_launch(a, st);
  if (a->kind == 1) return m2::longconv_tc_launch(a, st);
  if (a->kind == 2) return m2::longconv_tcl_launch(a, st);
  if (a->kind == 3) return m2::longconv_tz_launch(a, st);
  if (a->kind == 4) return m2::longconv_bt_launch(a, st);
  return m2_set_error(M2_ERR_ARG, "m2_longconv_fwd: unknown kind %d", a->kind);
}
