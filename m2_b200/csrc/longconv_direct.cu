// Fused gated long convolution of a few short rows on CUDA cores: the table, operands and rounding points of family 4
// (longconv_bt.cu), its products summed directly in float32.
//
// The tensor-core kernels pay for their structure whatever the batch: tensor memory, two Toeplitz strips in shared memory, a
// round trip of barriers per filter and columns that hold nothing (15 of 16 for one sequence).  At 768 channels of 128
// steps that is 16.5 us for one sequence and for eight, a quarter of a one-query forward.  The sums themselves are L^2
// fused multiply-adds a row, channel and filter: 0.7 us of the chip for one sequence, 5.7 us for eight.
// Here a CTA takes one channel of up to R sequences.  A thread owns eight outputs of one filter and slides a window of 16 taps
// in registers over (a part of) the row: two 16-byte shared loads of taps and two of data (broadcast) for 64 FMAs.
// All global loads are issued before the first barrier, so a CTA waits for memory once.
//
// Computation replaced: bert/src/mm/monarch_mixer_sequence_mixer.py:109-149 and
// bert/src/mm/hyena_utils.py:16-42, :219-248 of the reference.
#include "tc_common.cuh"

namespace m2 {
namespace dc {

constexpr int THREADS = 256;

struct Params {
  int B, L, D, nf, R, S, TG, tpad, half;       // R rows per CTA, S parts of the sum, TG = ceil(L / 8) groups of eight steps
  int u_f16, yu_bf16;                          // half: index of tap 0 in the table
  const __nv_bfloat16* xin; long long xsb, xsc;
  const void* u; long long usb, usc;
  __nv_bfloat16* out; long long osb, osc;
  const float* sw; const float* sb;
  const float* spec[2];
};

__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ float2 half2_to_float2(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }

// shared memory in floats: taps [nf][2 half], data [nf][R][8 TG], sums [S][nf][R][8 TG]
__global__ void __launch_bounds__(THREADS)
longconv_direct_kernel(const Params P) {
  using namespace lcl;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = P.L, R = P.R, TG = P.TG, row8 = 8 * TG, cells = R * TG;
  float* taps = reinterpret_cast<float*>(smem_raw);
  float* data = taps + P.nf * 2 * P.half;
  float* sums = data + P.nf * R * row8;
  const int tid = threadIdx.x, c = blockIdx.x, b0 = blockIdx.y * R;
  pdl_wait();

  // ---- a thread's eight steps of one row: short convs, gate, residual input ----
  const int tg = tid % TG, r = tid / TG, t0 = 8 * tg, b = b0 + r;
  const bool mine = tid < cells && b < P.B;
  uint32_t gate[4] = {0u, 0u, 0u, 0u};
  float inv[2] = {0.f, 0.f};
  if (mine) {
    uint4 x[3], v = make_uint4(0u, 0u, 0u, 0u);
    uint32_t before[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const __nv_bfloat16* row = P.xin + (long long)(i * P.D + c) * P.xsc + b * P.xsb + t0;
      x[i] = __ldg(reinterpret_cast<const uint4*>(row));
      before[i] = tg ? __ldg(reinterpret_cast<const uint32_t*>(row - 2)) : 0u;
    }
    if (P.nf == 2) v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(P.u) + c * P.usc + b * P.usb + t0));
#pragma unroll
    for (int f = 0; f < 2; ++f)
      if (f < P.nf) inv[f] = __ldg(P.spec[f] + (size_t)P.D * (P.tpad / 2) + c);
    uint32_t y[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint32_t w[5] = {before[i], x[i].x, x[i].y, x[i].z, x[i].w};
      conv_packed<8>(load_taps2(P.sw, P.sb, i * P.D + c), w, y[i]);
    }
    float a[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { gate[j] = y[1][j]; y[0][j] = bf2_mul(y[2][j], y[0][j]); }
    mask_tail(y[0], t0, L);
#pragma unroll
    for (int j = 0; j < 4; ++j) { a[2 * j] = bf_lo(y[0][j]); a[2 * j + 1] = bf_hi(y[0][j]); }
    store8(data + r * row8 + t0, a);
    if (P.nf == 2) {
      uint32_t h[4] = {v.x, v.y, v.z, v.w};
      mask_tail(h, t0, L);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 q = P.u_f16 ? half2_to_float2(h[j]) : make_float2(bf_lo(h[j]), bf_hi(h[j]));
        a[2 * j] = q.x; a[2 * j + 1] = q.y;
      }
      store8(data + (R + r) * row8 + t0, a);
    }
  }
  // ---- taps ----
  for (int i = tid; i < P.nf * (P.half / 4); i += blockDim.x) {
    const int f = i >= P.half / 4, k = i - f * (P.half / 4);
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(P.spec[f]) + (size_t)c * P.tpad) + k);
    const float2 h0 = half2_to_float2(q.x), h1 = half2_to_float2(q.y), h2 = half2_to_float2(q.z), h3 = half2_to_float2(q.w);
    const float h[8] = {h0.x, h0.y, h1.x, h1.y, h2.x, h2.y, h3.x, h3.y};
    store8(taps + f * 2 * P.half + 8 * k, h);
  }
  __syncthreads();

  // ---- sums: thread = (part, filter, row, group of eight outputs) ----
  {
    const int job = tid / cells, f = job % P.nf, s = job / P.nf;
    if (s < P.S && b0 + (tid - job * cells) / TG < P.B) {
      const int cell = tid - job * cells, og = cell % TG, orow = cell / TG;
      const int per = (TG + P.S - 1) / P.S, k0 = s * per, k1 = min(TG, k0 + per);
      const float* h = taps + f * 2 * P.half + P.half - 8 * og;        // h[d + 8 og] multiplies the step d behind an output
      const float* a = data + (f * R + orow) * row8;
      float acc[8] = {}, lo[8];
      load8(h + 8 * k0 - 8, lo);                                       // distances 8 (k - og) - 8 .. - 1
#pragma unroll 2
      for (int k = k0; k < k1; ++k) {
        float hi[8], v[8];
        load8(h + 8 * k, hi);
        load8(a + 8 * k, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = fmaf(v[j], j >= i ? hi[j - i] : lo[8 + j - i], acc[i]);
#pragma unroll
        for (int i = 0; i < 8; ++i) lo[i] = hi[i];
      }
      store8(sums + ((s * P.nf + f) * R + orow) * row8 + 8 * og, acc);
    }
  }
  __syncthreads();

  // ---- (conv + bias term) as bf16, times the gate as bf16; the residual conv joins in float32 (or bf16 first) ----
  if (mine) {
    uint32_t o[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (f >= P.nf) break;
      float z[8];
      load8(sums + (f * R + r) * row8 + t0, z);
      for (int s = 1; s < P.S; ++s) {
        float q[8];
        load8(sums + ((s * P.nf + f) * R + r) * row8 + t0, q);
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] += q[i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y0 = z[2 * j] * inv[f], y1 = z[2 * j + 1] * inv[f];
        if (f == 0) o[j] = bf2_mul(pack_bf2(y0, y1), gate[j]);
        else if (P.yu_bf16) o[j] = pack_bf2(bf_lo(o[j]) + bf16r(y0), bf_hi(o[j]) + bf16r(y1));
        else o[j] = pack_bf2(bf_lo(o[j]) + y0, bf_hi(o[j]) + y1);
      }
    }
    store_chunk8(P.out + c * P.osc + b * P.osb, t0, L, make_uint4(o[0], o[1], o[2], o[3]));
  }
}

}  // namespace dc

// Time of this kernel in us, as measured for D = 768 and 1536, L = 16 .. 512, B = 1 .. 32: 3 us for a launch in the stream of a
// forward and 1 us for every 20 M multiplications (128 steps, 768 channels: 5.1 us for 1 sequence, 9.5 for 4, 13.5 for 8;
// 256 steps: 9.6, 21.6, 37.8).  Rows beyond 512 steps would need more threads than a CTA of it has.
double longconv_direct_us(int B, int L, int D, int nf) {
  return L <= 512 ? 3.0 + (double)nf * B * D * L * L / 20e6 : 1e30;
}

// Called by longconv_bt_launch, which has checked the arguments.
int longconv_direct_launch(const m2_longconv_args* a, int tpad, int half, int u_f16, int yu_bf16, cudaStream_t st) {
  dc::Params P;
  P.B = a->batch; P.L = a->seq_len; P.D = a->d_model; P.nf = a->n_filters;
  P.TG = (P.L + 7) / 8;
  P.tpad = tpad; P.half = half;
  P.R = dc::THREADS / (P.TG * P.nf);                             // at least 2: L <= 512
  if (P.R > P.B) P.R = P.B;
  P.S = 1;
  while (P.S < 4 && 2 * P.S <= P.TG && 2 * P.S * P.nf * P.R * P.TG <= dc::THREADS) P.S *= 2;
  P.u_f16 = u_f16; P.yu_bf16 = yu_bf16;
  P.xin = (const __nv_bfloat16*)a->xin; P.xsb = a->xin_sb; P.xsc = a->xin_sc;
  P.u = a->u; P.usb = a->u_sb; P.usc = a->u_sc;
  P.out = (__nv_bfloat16*)a->out; P.osb = a->out_sb; P.osc = a->out_sc;
  P.sw = a->short_w; P.sb = a->short_b;
  P.spec[0] = a->spec[0]; P.spec[1] = a->spec[1];
  const int threads = (P.S * P.nf * P.R * P.TG + 31) / 32 * 32;
  const size_t smem = 4 * ((size_t)P.nf * 2 * half + (size_t)(1 + P.S) * P.nf * P.R * 8 * P.TG);   // at most 8 KB each
  return m2_launch("longconv_direct_kernel", (long long)P.B * P.L * P.D, dc::longconv_direct_kernel, dim3(P.D, (P.B + P.R - 1) / P.R), threads,
                   smem, st, P);
}

}  // namespace m2
