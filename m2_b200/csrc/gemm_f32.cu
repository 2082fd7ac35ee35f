// Linear and block-diagonal layers on float32 activations where no split weights are given (gemm_split.cu, three times as fast and
// nearer to the exact sum): CUDA-core GEMM tiles with register blocking, operands brought to
// shared memory by cp.async, four stages deep.  Every output is one chain of fused multiply-adds in ascending k, the order
// of the one-element kernels in gemm_simt.cu and linear_tc.cu, so the results are the same bits whatever the tile.
//
// Bound by the float32 pipe (128 FMA per SM and clock).  The 64 x 64 tiles of the one-element kernels gave a thread 4 x 4
// outputs, eight scalar shared loads for 16 FMAs, scalar global loads and none in flight during the multiplications.  Here
// a thread owns up to 8 x 4 outputs and reads four columns of k at a time (12 shared loads of 16 bytes for 128 FMAs).  Rows
// stay k-contiguous in shared memory, 20 floats apart, so that the eight rows a warp reads at once start in eight different
// bank groups.  Three stages in flight are what a tile alone on its SM needs: with one (held in registers, transposed
// on the way) a K step of 16 took 2300 clocks at 64 tokens, 512 of them multiplications.
// Measured (us, L2 flushed; the one-element kernels first) for 768 -> 2304 / 768 -> 768 / GLU 768 -> 3072 / wo 3072 -> 768:
// 64 tokens 74 / 70 / 37 / 80 -> 37 / 37 / 25 / 37; 1024: 159 / 92 / 121 / 98 -> 92 / 57 / 86 / 55; 2048: 303 / 127 / 213 /
// 129 -> 178 / 86 / 158 / 86 (113 for the 768-column ones with two small tiles on an SM instead of three); 8192: 1168 / 420 /
// 780 / 410 -> 684 / 261 / 551 / 260, 58 % of the pipe.  There a third of the stalls are register-file conflicts at dispatch and as
// many shared loads.  Packed f32x2 FMAs over pairs of k need twice the accumulators, so 8 x 4 outputs are all a thread holds
// and shared memory (69 % busy) binds: 745 us at 8192 tokens.
//
// Computation replaced: nn.Linear of bert/src/mm/monarch_mixer_sequence_mixer.py:100-154, bert/src/mm/blockdiag_multiply.py:49-60,
// bert/src/mm/structured_linear.py:52-70, bert/src/bert_layers.py:492-506 of the reference, float32.
#include "common.cuh"

namespace m2 {
namespace f32g {

constexpr int BK = 16;
constexpr int PITCH = BK + 4;              // floats between rows in shared memory
constexpr int STAGES = 4;
constexpr int THREADS = 256;

struct Params {
  const float* x; long long xsb, xst;      // token t starts at x + (t / L) * xsb + (t % L) * xst, features contiguous
  const float* w;                          // [block][q][p]
  const float* bias;
  float* out; long long osb, ost, osc;
  int tokens, L, p, q;
  int partner;                             // GLU: block kb is gated, block kb + partner is its factor
};

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, const float* any, bool in) {   // zeros where !in
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? src : any), "r"(in ? 16 : 0) : "memory");
}

template <int RM, bool GLU>
__global__ void __launch_bounds__(THREADS, RM == 1 && !GLU ? 3 : 2)
gemm_f32_kernel(const Params P) {
  constexpr int BM = 64 * RM, BN = 64, STAGE = (BM + BN) * PITCH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* smem = reinterpret_cast<float*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN, kb = blockIdx.z;
  // rows that this thread brings to shared memory, four columns of each K step; NULL where the tile reaches past the matrix
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  const float* xr[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int t = row0 + lr + 64 * i;
    xr[i] = t < P.tokens ? P.x + (t / P.L) * P.xsb + (t % P.L) * P.xst + (long long)kb * P.p + lk : nullptr;
  }
  const int wn = col0 + lr;
  const float* wr = wn < P.q ? P.w + ((long long)kb * P.q + wn) * P.p + lk : nullptr;
  const uint32_t put = static_cast<uint32_t>(__cvta_generic_to_shared(smem + lr * PITCH + lk));
  const int steps = (P.p + BK - 1) / BK, total = GLU ? 2 * steps : steps;
  auto fetch = [&](int c) {               // K step c; those of the GLU's factor follow those of its gate
    if (c < total) {
      const bool second = GLU && c >= steps;
      const int k = (second ? c - steps : c) * BK;
      const long long xo = k + (second ? (long long)P.partner * P.p : 0), wo = k + (second ? (long long)P.partner * P.q * P.p : 0);
      const uint32_t dst = put + (c % STAGES) * STAGE * 4;
      const bool in = k + lk < P.p;
#pragma unroll
      for (int i = 0; i < RM; ++i) copy16(dst + 64 * i * PITCH * 4, xr[i] + xo, P.x, in && xr[i]);
      copy16(dst + BM * PITCH * 4, wr + wo, P.w, in && wr);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // this thread's outputs: rows a0 + 4 i, columns b0 + 8 j
  const int a0 = (warp >> 1) * (16 * RM) + (lane >> 3), b0 = (warp & 1) * 32 + (lane & 7);
  float acc[GLU ? 2 : 1][4 * RM][4] = {};
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) fetch(c);
#pragma unroll
  for (int half = 0; half < (GLU ? 2 : 1); ++half)
    for (int c = half * steps; c < (half + 1) * steps; ++c) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      __syncthreads();                    // K step c has landed for everybody, and step c - 1 has been read
      fetch(c + STAGES - 1);
      const float* sa = smem + (c % STAGES) * STAGE + a0 * PITCH;
      const float* sb = smem + (c % STAGES) * STAGE + (BM + b0) * PITCH;
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        float4 a[4 * RM];
#pragma unroll
        for (int i = 0; i < 4 * RM; ++i) a[i] = *reinterpret_cast<const float4*>(sa + 4 * i * PITCH + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 b = *reinterpret_cast<const float4*>(sb + 8 * j * PITCH + k);
          const float bk[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)      // neighbouring FMAs share b and nothing else
#pragma unroll
            for (int i = 0; i < 4 * RM; ++i) {
              const float ak[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
              acc[half][i][j] = fmaf(ak[e], bk[e], acc[half][i][j]);
            }
        }
      }
    }
#pragma unroll
  for (int i = 0; i < 4 * RM; ++i) {
    const int t = row0 + a0 + 4 * i;
    if (t >= P.tokens) continue;
    float* po = P.out + (t / P.L) * P.osb + (t % P.L) * P.ost;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cq = col0 + b0 + 8 * j;
      if (cq >= P.q) continue;
      const long long c = (long long)kb * P.q + cq;
      float v = acc[0][i][j];
      if constexpr (GLU) v = gelu_erf(v) * acc[GLU ? 1 : 0][i][j];
      else if (P.bias) v += __ldg(P.bias + c);
      po[c * P.osc] = v;
    }
  }
}

template <int RM, bool GLU>
static int launch(const Params& P, int blocks, cudaStream_t st) {
  dim3 grid((P.q + 63) / 64, (P.tokens + 64 * RM - 1) / (64 * RM), blocks);
  const int smem = STAGES * 64 * (RM + 1) * PITCH * (int)sizeof(float);
  auto kern = gemm_f32_kernel<RM, GLU>;
  M2_SMEM_ONCE(kern, smem);
  kern<<<grid, THREADS, smem, st>>>(P);
  M2_LAUNCH_CHECK("gemm_f32_kernel");
  return M2_OK;
}

// The tile that finishes first if every SM works its share off: tall tiles multiply at a higher rate (twelve shared loads
// for 128 FMAs instead of eight for 64), small ones leave fewer SMs without work.  128 x 128 tiles with 8 x 8 outputs a
// thread are no faster (8192 tokens, 768 -> 2304: 762 us) and idle more SMs (1024 tokens: 125 us).
template <bool GLU>
static int run(const Params& P, int blocks, cudaStream_t st) {
  const int sms = m2_sm_count();
  auto cost = [&](int rm, double rate) {
    const long long tiles = (long long)((P.tokens + 64 * rm - 1) / (64 * rm)) * ((P.q + 63) / 64) * blocks;
    return (double)((tiles + sms - 1) / sms) * rm / rate;
  };
  return cost(1, 0.8) < cost(2, 1.0) ? launch<1, GLU>(P, blocks, st) : launch<2, GLU>(P, blocks, st);
}

// What the 16-byte loads along k need: rows that start on 16-byte boundaries and are a multiple of four columns long.
static bool rows_ok(const void* x, long long ld, const void* w, int p) {
  return p % 4 == 0 && ld % 4 == 0 && m2_aligned(x, 16) && m2_aligned(w, 16);
}

}  // namespace f32g

bool linear_f32_supported(const m2_linear_args* a) {
  return a->dtype == M2_F32 && !a->force_simt && a->x_sc == 1 && (a->batch == 1 || a->x_sb % 4 == 0) &&
         f32g::rows_ok(a->x, a->x_st, a->w, a->in_features);
}

int linear_f32_launch(const m2_linear_args* a, cudaStream_t st) {
  f32g::Params P = {};
  P.x = (const float*)a->x; P.xsb = a->x_sb; P.xst = a->x_st;
  P.w = (const float*)a->w; P.bias = a->bias;
  P.out = (float*)a->out; P.osb = a->out_sb; P.ost = a->out_st; P.osc = a->out_sc;
  P.tokens = a->batch * a->seq_len; P.L = a->seq_len; P.p = a->in_features; P.q = a->out_features;
  return f32g::run<false>(P, 1, st);
}

bool blockdiag_f32_supported(const m2_blockdiag_args* a) {
  return a->dtype == M2_F32 && a->in_features == a->nblocks * a->p && a->out_features == a->nblocks * a->q &&
         f32g::rows_ok(a->x, a->ldx, a->w, a->p);
}

int blockdiag_f32_launch(const m2_blockdiag_args* a, cudaStream_t st) {
  f32g::Params P = {};
  P.x = (const float*)a->x; P.xst = a->ldx;
  P.w = (const float*)a->w; P.bias = a->bias;
  P.out = (float*)a->out; P.ost = a->ldo; P.osc = 1;
  P.tokens = P.L = a->m; P.p = a->p; P.q = a->q;
  return f32g::run<false>(P, a->nblocks, st);
}

bool glu_f32_supported(const m2_glu_args* a) {
  return a->dtype == M2_F32 && f32g::rows_ok(a->x, a->ldx, a->wg, a->d_model / a->nblocks);
}

int glu_f32_launch(const m2_glu_args* a, cudaStream_t st) {
  f32g::Params P = {};
  P.x = (const float*)a->x; P.xst = a->ldx;
  P.w = (const float*)a->wg;
  P.out = (float*)a->h; P.ost = a->ldh; P.osc = 1;
  P.tokens = P.L = a->m; P.p = a->d_model / a->nblocks; P.q = 2 * a->inter / a->nblocks;
  P.partner = a->nblocks / 2;
  return f32g::run<true>(P, a->nblocks / 2, st);
}

}  // namespace m2
