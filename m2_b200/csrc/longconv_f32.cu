// Fused gated long convolution in float32 on channel-contiguous activations (float32, or bf16 with the roundings of
// autocast), rows of up to 2048 steps: the arithmetic of longconv_simt.cu (same butterflies in the same order on the same
// tables) in register passes of up to three radix-2 stages.
//
// The stage-by-stage kernel crossed shared memory and a barrier 2 lg M times per filter, read every twiddle through L1,
// read the filter table eight bytes of a 32-byte sector at a time and evaluated the short convolution five times a step.
// Here one thread holds 8 points through three stages; the first pass takes its points from global memory (the upper
// half is padding and never read), the last one finishes the outputs, so shared memory is crossed 2 ceil(lg M / 3) - 1
// times.  Lanes run along channels (shared rows of an odd number of points, so every access is free of bank conflicts, and
// twiddles are broadcasts) except in the filter step, where they run along the table.  In bit-reversed order the
// partner of position p in [2^j, 2^(j+1)) is 3 * 2^j - 1 - p: both ends of a bin pair are read in consecutive order.
//
// Bound by the float32 pipe and shared memory together; the tables (16 bytes a point and channel) come from L2.  Measured
// at 768 channels, two filters (us, L2 flushed; the stage-by-stage kernel first): 8 x 128 115 -> 33, 4 x 512 283 -> 109,
// 8 x 1024 797 -> 254, 4 x 2048 920 -> 326, 3 x 500 210 -> 64, 1 x 64 49 -> 21.  On bf16 rows (float32
// residual input): 6 x 1531 1163 -> 393, 2 x 514 277 -> 91, 47 x 64 150 -> 86, 8 x 64 57 -> 37, 1 x 37 45 -> 18.
//
// Computation replaced: bert/src/mm/monarch_mixer_sequence_mixer.py:109-149 and bert/src/mm/hyena_utils.py:16-42, :219-248
// of the reference, float32.
#include "common.cuh"

namespace m2 {
namespace f32c {

constexpr int THREADS_MAX = 512;

// of a value that this thread has written: a plain load, not the read-only path of ld_as_float
__device__ __forceinline__ float to_float(const float& v) { return v; }
__device__ __forceinline__ float to_float(const __nv_bfloat16& v) { return __bfloat162float(v); }

// 2^R points at distance 2^lgq, starting at offset pos of a block of 2^(R + lgq) points: R decimation-in-frequency stages.
template <int R>
__device__ __forceinline__ void forward_stages(float2 (&z)[1 << R], int pos, int lgq, int lgM, const float2* tw, bool upper_zero) {
#pragma unroll
  for (int s = 0; s < R; ++s) {
    const int half = 1 << (R - 1 - s), lgh = R - 1 - s + lgq, shift = lgM - 1 - lgh;      // lgh: log2 of the pair's distance
#pragma unroll
    for (int i = 0; i < (1 << R); ++i) {
      if (i & half) continue;
      const float2 w = tw[(pos + ((i & (half - 1)) << lgq)) << shift];
      const float2 a = z[i], b = z[i + half];
      if (s == 0 && upper_zero) {
        z[i + half] = cmul(a, w);
      } else {
        z[i] = make_float2(a.x + b.x, a.y + b.y);
        z[i + half] = cmul(make_float2(a.x - b.x, a.y - b.y), w);
      }
    }
  }
}

// The decimation-in-time counterpart; with lower_only the last stage leaves the upper half out.
template <int R>
__device__ __forceinline__ void inverse_stages(float2 (&z)[1 << R], int pos, int lgq, int lgM, const float2* tw, bool lower_only) {
#pragma unroll
  for (int s = R - 1; s >= 0; --s) {
    const int half = 1 << (R - 1 - s), lgh = R - 1 - s + lgq, shift = lgM - 1 - lgh;
#pragma unroll
    for (int i = 0; i < (1 << R); ++i) {
      if (i & half) continue;
      const float2 w = tw[(pos + ((i & (half - 1)) << lgq)) << shift];
      const float2 a = z[i], b = cmul_conj(z[i + half], w);
      z[i] = make_float2(a.x + b.x, a.y + b.y);
      if (!(s == 0 && lower_only)) z[i + half] = make_float2(a.x - b.x, a.y - b.y);
    }
  }
}

// One channel of one batch row: short-conv weights of its three projections, pointers to its columns.
template <typename TA, bool ROUND>
struct Channel {
  const TA* x; long long xst; long long g;         // projection i starts at x + i * g
  float w[3][3], b[3];
  int L;
  // short-conv outputs of projection i at steps 2n and 2n + 1 (2n + 1 past the end: meaningless)
  __device__ __forceinline__ float2 conv(int i, int n) const {
    const TA* p = x + i * g + 2LL * n * xst;
    const float x0 = n > 0 ? ld_as_float(p - 2 * xst) : 0.f, x1 = n > 0 ? ld_as_float(p - xst) : 0.f, x2 = ld_as_float(p);
    const float x3 = 2 * n + 1 < L ? ld_as_float(p + xst) : 0.f;
    return make_float2(rnd<ROUND>(fmaf(w[i][2], x2, fmaf(w[i][1], x1, fmaf(w[i][0], x0, b[i])))),
                       rnd<ROUND>(fmaf(w[i][2], x3, fmaf(w[i][1], x2, fmaf(w[i][0], x1, b[i])))));
  }
  __device__ __forceinline__ float2 gated(int n) const {
    const float2 a = conv(0, n), v = conv(2, n);
    return make_float2(rnd<ROUND>(v.x * a.x), 2 * n + 1 < L ? rnd<ROUND>(v.y * a.y) : 0.f);
  }
};

// R0 = stages of the first forward and the last inverse pass: lg M = R0 + 3 * passes.  TA: activations, TU: residual input,
// ROUND: bf16 at the points where the reference's operators round under autocast
template <int R0, typename TA, typename TU, bool ROUND>
__global__ void __launch_bounds__(THREADS_MAX)
longconv_f32_kernel(const ConvParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = p.M, lgM = p.lgM, L = p.L, D = p.D, CT = p.CT;
  float2* tw = reinterpret_cast<float2*>(smem_raw);                          // [M / 2]
  float2* rows = tw + (M >> 1);                                              // [CT][M + 1]
  const int tid = threadIdx.x, threads = blockDim.x, ci = tid % CT, worker = tid / CT, workers = threads / CT;
  const int c = blockIdx.x * CT + ci;
  const bool live = c < D;
  const int cc = live ? c : D - 1;                                           // a channel to read where the tile reaches past the last one
  float2* s = rows + ci * (M + 1);
  const int npair = (L + 1) >> 1;
  Channel<TA, ROUND> ch;
  ch.x = reinterpret_cast<const TA*>(p.xin) + blockIdx.y * p.xsb + cc * p.xsc;
  ch.xst = p.xst; ch.g = D * p.xsc; ch.L = L;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int k = 0; k < 3; ++k) ch.w[i][k] = rnd<ROUND>(__ldg(p.sw + 3 * (i * D + cc) + k));
    ch.b[i] = rnd<ROUND>(__ldg(p.sb + i * D + cc));
  }
  const TU* u = reinterpret_cast<const TU*>(p.u) + blockIdx.y * p.usb + cc * p.usc;
  TA* out = reinterpret_cast<TA*>(p.out) + blockIdx.y * p.osb + cc * p.osc;
  auto input = [&](int f, int n) {
    if (n >= npair) return make_float2(0.f, 0.f);
    if (f == 0) return ch.gated(n);
    const TU* pu = u + 2LL * n * p.ust;
    return make_float2(ld_as_float(pu), 2 * n + 1 < L ? ld_as_float(pu + p.ust) : 0.f);
  };
  for (int i = tid; i < (M >> 1); i += threads) tw[i] = __ldg(reinterpret_cast<const float2*>(p.spec[0]) + i);   // the same in both tables
  __syncthreads();

  for (int f = 0; f < p.nf; ++f) {
    // ---- first R0 stages, points straight from the activations ----
    {
      const int lgq = lgM - R0;
      for (int pos = worker; pos < (1 << lgq); pos += workers) {
        float2 z[1 << R0];
#pragma unroll
        for (int i = 0; i < (1 << R0) / 2; ++i) z[i] = input(f, pos + (i << lgq));
        forward_stages<R0>(z, pos, lgq, lgM, tw, true);
#pragma unroll
        for (int i = 0; i < (1 << R0); ++i) s[pos + (i << lgq)] = z[i];
      }
      __syncthreads();
    }
    // ---- three stages a pass ----
    for (int lgq = lgM - R0 - 3; lgq >= 0; lgq -= 3) {
      for (int j = worker; j < (M >> 3); j += workers) {
        const int pos = j & ((1 << lgq) - 1);
        float2* base = s + ((j >> lgq) << (lgq + 3)) + pos;
        float2 z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = base[i << lgq];
        forward_stages<3>(z, pos, lgq, lgM, tw, false);
#pragma unroll
        for (int i = 0; i < 8; ++i) base[i << lgq] = z[i];
      }
      __syncthreads();
    }
    // ---- Zy[k] = alpha Z[k] + beta conj(Z[M - k]), lanes along the table ----
    const float2* tab = reinterpret_cast<const float2*>(p.spec[f] + M);
    for (int idx = tid; idx < CT << (lgM - 1); idx += threads) {
      const int k = idx & ((M >> 1) - 1), ri = idx >> (lgM - 1);
      if (blockIdx.x * CT + ri >= D) continue;
      const float2* al = tab + (size_t)(blockIdx.x * CT + ri) * 2 * M;
      float2* r = rows + ri * (M + 1);
      if (k == 0) {                                  // positions 0 and 1 hold bins 0 and M / 2, their own partners
        filter_pair(r, 0, 0, al, al + M, 0, 0);
        filter_pair(r, 1, 1, al, al + M, 1, 1);
      } else {                                       // k in [2^(j-1), 2^j) -> the lower half of positions [2^j, 2^(j+1))
        const int b = 1 << (31 - __clz(k));
        const int pk = k + b, pm = 6 * b - 1 - pk;
        filter_pair(r, pk, pm, al, al + M, pk, pm);
      }
    }
    __syncthreads();
    // ---- inverse: three stages a pass ----
    for (int lgq = 0; lgq < lgM - R0; lgq += 3) {
      for (int j = worker; j < (M >> 3); j += workers) {
        const int pos = j & ((1 << lgq) - 1);
        float2* base = s + ((j >> lgq) << (lgq + 3)) + pos;
        float2 z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = base[i << lgq];
        inverse_stages<3>(z, pos, lgq, lgM, tw, false);
#pragma unroll
        for (int i = 0; i < 8; ++i) base[i << lgq] = z[i];
      }
      __syncthreads();
    }
    // ---- last R0 stages, bias, gates, residual ----
    const float bc = __ldg(p.bias[f] + cc);
    {
      const int lgq = lgM - R0;
      for (int pos = worker; pos < (1 << lgq); pos += workers) {
        float2 z[1 << R0];
#pragma unroll
        for (int i = 0; i < (1 << R0); ++i) z[i] = s[pos + (i << lgq)];
        inverse_stages<R0>(z, pos, lgq, lgM, tw, true);
#pragma unroll
        for (int i = 0; i < (1 << R0) / 2; ++i) {
          const int n = pos + (i << lgq);
          if (!live || n >= npair) continue;
          TA* po = out + 2LL * n * p.ost;
          const bool two = 2 * n + 1 < L;
          if (f == 0) {
            const float2 a = ch.gated(n), x2 = ch.conv(1, n);
            st_from_float(po, rnd<ROUND>(fmaf(a.x, bc, z[i].x)) * x2.x);
            if (two) st_from_float(po + p.ost, rnd<ROUND>(fmaf(a.y, bc, z[i].y)) * x2.y);
          } else {                                   // adds to what this thread wrote for the first filter
            const float2 uo = input(1, n);
            float2 yu = make_float2(fmaf(uo.x, bc, z[i].x), fmaf(uo.y, bc, z[i].y));
            if (ROUND && sizeof(TU) == 2) yu = make_float2(bf16r(yu.x), bf16r(yu.y));   // a bf16 layer input: rounded before the sum
            st_from_float(po, to_float(po[0]) + yu.x);
            if (two) st_from_float(po + p.ost, to_float(po[p.ost]) + yu.y);
          }
        }
      }
      __syncthreads();                               // the rows are free for the next filter
    }
  }
}

template <int R0, typename TA, typename TU, bool ROUND>
static int launch(const ConvParams& p, int threads, size_t smem, cudaStream_t st) {
  auto kern = longconv_f32_kernel<R0, TA, TU, ROUND>;
  M2_SMEM_ONCE(kern, SIMT_SMEM_MAX);
  kern<<<dim3((p.D + p.CT - 1) / p.CT, p.B), threads, smem, st>>>(p);
  M2_LAUNCH_CHECK("longconv_f32_kernel");
  return M2_OK;
}

template <typename TA, typename TU, bool ROUND>
static int launch_stages(const ConvParams& p, int threads, size_t smem, cudaStream_t st) {
  switch (p.lgM % 3) {
    case 1: return launch<1, TA, TU, ROUND>(p, threads, smem, st);
    case 2: return launch<2, TA, TU, ROUND>(p, threads, smem, st);
    default: return launch<3, TA, TU, ROUND>(p, threads, smem, st);
  }
}

}  // namespace f32c

// Rows of up to 2048 steps: eight of them (a 32-byte sector of float32 channels) still fit one CTA.  float32 activations in
// float32, or bf16 ones with the roundings of autocast.
bool longconv_f32_supported(const m2_longconv_args* a) {
  const bool f32 = a->act_dtype == M2_F32 && !a->bf16_rounding, bf16 = a->act_dtype == M2_BF16 && a->bf16_rounding;
  return (f32 || bf16) && !a->plain && a->seq_len <= 2048 && a->xin_sc == 1 && a->out_sc == 1 &&
         (a->n_filters == 1 || (a->u_sc == 1 && (a->u_dtype == M2_F32 || (bf16 && a->u_dtype == M2_BF16))));
}

// channels per CTA: 32 make a warp's access one 128-byte line (64 bytes of bf16), fewer leave room for more CTAs; 64 KB of
// rows let three CTAs share an SM, and two CTAs per SM should exist
static int longconv_f32_channels(int B, int M, int D) {
  const size_t row = (size_t)(M + 1) * sizeof(float2);
  int ct = 32;
  while (ct > 8 && (ct * row > 66 * 1024 || (long long)((D + ct - 1) / ct) * B < 2 * m2_sm_count())) ct >>= 1;
  return ct;
}
long long longconv_f32_ctas(int B, int L, int D) {
  const int ct = longconv_f32_channels(B, m2_filter_row_len(L) / 2, D);
  return (long long)((D + ct - 1) / ct) * B;
}

int longconv_f32_launch(const m2_longconv_args* a, ConvParams p, cudaStream_t st) {
  const size_t row = (size_t)(p.M + 1) * sizeof(float2);
  const int ct = p.CT = longconv_f32_channels(p.B, p.M, p.D);
  const size_t smem = ct * row + (size_t)(p.M / 2) * sizeof(float2);
  const int threads = smem > 100 * 1024 ? 512 : 256;                         // the one CTA of an SM brings 16 warps
  if (a->act_dtype == M2_F32) return f32c::launch_stages<float, float, false>(p, threads, smem, st);
  if (a->n_filters == 2 && a->u_dtype == M2_F32) return f32c::launch_stages<__nv_bfloat16, float, true>(p, threads, smem, st);
  return f32c::launch_stages<__nv_bfloat16, __nv_bfloat16, true>(p, threads, smem, st);
}

}  // namespace m2
