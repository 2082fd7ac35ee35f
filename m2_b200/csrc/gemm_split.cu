// Linear and block-diagonal layers on float32 activations as tcgen05 GEMMs over triples of bf16 values, with float32 results.
//
// Every value of x and w is written as hi + mid + lo, three bf16 values of eight bits each: rounded to nearest, they hold the 24 bits
// of a float32 exactly (down to 2^-110, where lo leaves the range), whatever its neighbours are.  x . w is then lo.hi + hi.lo + mid.mid +
// mid.hi + hi.mid + hi.hi on the tensor cores (mid.lo and lo.mid are at most 2^-25 of |x||w| each), summed over 64 columns in tensor
// memory, small terms first.  Each such sum is added to a float32 register, rounded to nearest: the tensor core's own
// accumulation drops what does not fit, always towards zero, so a chain of K / 16 of its additions would be further from the
// exact sum than a float32 chain; the four of the large terms are nearer.  Relative 2-norm against 64 bits, chain / this: N(0, 1)
// operands 128 columns 2.0e-7 / 0.8e-7, 768 5.0e-7 / 1.0e-7; of one sign 1.7e-7 / 0.9e-7, 3.7e-7 / 1.0e-7.  Results that are one large
// product are truncated, up to 2^-23, where a chain rounds them (2.6e-8 / 9.3e-8).
// Two fp16 values with a scale for 64 columns take half the MMAs and a sixth less time, but keep 22 bits, and fewer of what is below
// 2^-17 of the largest beside it: with one column in 64 scaled by 2^24 in x and by 2^-24 in w the result was 1.4e-5 off (here it is the
// same bits as without), and operands of one sign in 128 columns 2.1e-7.
//
// A result that is not finite is summed again as the ascending float32 chain of gemm_f32.cu: products of infinities with the parts of
// a value, and values that round up to an infinite hi, end here.  So is one below 2^-100 that is not zero, as rows of such values have
// lost parts; beyond that a part below 2^-133 is missed only where its partner in the product is beyond 2^100 or so.
//
// Roles: warp 0 brings float32 rows of x and split rows of w to shared memory by TMA, warps 12-19 convert (a thread owns a row
// of x; four warps take the even K blocks, four the odd ones) and leave the three parts in tensor memory, from where the MMAs take
// them as their A operand, warp 1 issues the MMAs, warps 4-11 add up.
//
// Bound: 64 columns of a 128 x 128 tile bring 80 KB to the SM, 2150 of its 2300 clocks at the 38 bytes a clock that TMA tile loads reach
// in every GEMM here; the 24 MMAs of 64 clocks take 1540, shared memory is busy for 1650 (80 KB written, 32 read by the conversion, 96
// by the MMAs).  Splitting x too before the launch would cost a pass and move more bytes.  Few rows: the first loads and one K block
// after the other.
// Measured (us, L2 flushed; the float32 chain of gemm_f32.cu / fp16 pairs / this): 768 -> 2304 at 64 tokens 38 / 15 / 15, 1024 94 / 23 / 27,
// 2048 180 / 35 / 41, 8192 684 / 107 / 130; 768 -> 768 at 64 37 / 15 / 14, 1024 57 / 16 / 18, 2048 87 / 23 / 25; GLU 768 -> 3072 at 2048
// 158 / 44 / 46; wo 88 / 25 / 25.
//
// Computation replaced: nn.Linear of bert/src/mm/monarch_mixer_sequence_mixer.py:100-154, bert/src/mm/blockdiag_multiply.py:49-60,
// bert/src/mm/structured_linear.py:52-70, bert/src/bert_layers.py:492-506 of the reference, float32.
#include "tc_common.cuh"

namespace m2 {
namespace f32s {

constexpr int BM = 128, BK = 64;
constexpr int FLUSH0 = 4, FLUSH_WARPS = 8, CONV0 = 12, CONV_WARPS = 4, THREADS = 32 * (CONV0 + 2 * CONV_WARPS);
constexpr int PARTS = 3, A_COLS = PARTS * BK / 2;       // tensor-memory columns of a K block of x: hi, mid, lo, 32 each
constexpr uint32_t TINY = 27u << 23;       // 2^-100
constexpr int X_BYTES = BM * 256;          // two boxes of 32 float32 columns

template <int BN> struct Geo {
  static constexpr int W_BYTES = BN * PARTS * 128;                   // hi, mid, lo of 64 columns of the rows of w
  // K blocks of x and of w in shared memory: x is free when it is converted, w when it is multiplied.  The two groups of conversion
  // warps take the K blocks in turn, so the stages of x and its buffers in tensor memory are even in number: then each is always the
  // same group's, which sees every phase of its barrier.  (A wait on a parity cannot tell a phase from the one two before.)
  static constexpr int NX = BN == 128 ? 2 : 4, NW = BN == 128 ? 3 : BN == 64 ? 4 : 5;
  static constexpr int NACC = BN == 32 ? 4 : 2, NA = BN == 128 ? 2 : 4;   // accumulators, buffers of x
  static_assert(NX % 2 == 0 && NA % 2 == 0, "a stage and a buffer of x belong to one group");
  static constexpr int OFF_W = NX * X_BYTES;
  static constexpr int OFF_COLS = OFF_W + NW * W_BYTES;              // [2] a tile's bias
  static constexpr int OFF_BAR = OFF_COLS + 2 * BN * 4;
  static constexpr int NBARS = 2 * NX + 2 * NW + 2 * NA + 2 * NACC + 4;
  static constexpr int SMEM = OFF_BAR + NBARS * 8 + 16 + 1024;
  static constexpr uint32_t TCOLS = 512;
  static_assert(NACC * BN + NA * A_COLS <= (int)TCOLS && NACC * BN + NA * A_COLS > 256, "tensor memory");
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
};

struct Params {
  const float* x; long long ldx;           // row t of x, block kb: x + t * ldx + kb * p
  const float* w;                          // [block][q][p]
  const __nv_bfloat16* ws;                 // the same rows split
  const float* bias;
  float* out; long long osb, ost, osc;     // token t at (t / L) * osb + (t % L) * ost
  int tokens, L, p, q, steps;
  int partner;                             // GLU: block kb is gated, block kb + partner is its factor
  int n_tiles, m_tiles, total;
  int vec;                                 // 32-byte stores are legal for eight neighbouring columns
};

__device__ __forceinline__ uint32_t bf16_pair(float y0, float y1) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(y0, y1);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// two values as pairs of their parts; what is left after each is exact
__device__ __forceinline__ void split_triple(float y0, float y1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = bf16_pair(y0, y1);
  y0 -= __uint_as_float(hi << 16);
  y1 -= __uint_as_float(hi & 0xffff0000u);
  mid = bf16_pair(y0, y1);
  lo = bf16_pair(y0 - __uint_as_float(mid << 16), y1 - __uint_as_float(mid & 0xffff0000u));
}

// weight rows: per 64 columns hi, mid, lo; zeros up to the next multiple of 64.  A warp per row, up to four matrices a launch.
struct SplitJobs {
  struct { const float* w; __nv_bfloat16* ws; int rows, p, steps, first, vec; } job[4];   // first: its first block of eight rows
  int n;
};
__global__ void __launch_bounds__(256)
split_weights_kernel(const SplitJobs J) {
  pdl_wait();
  int j = 0;
  while (j + 1 < J.n && (int)blockIdx.x >= J.job[j + 1].first) ++j;
  const float* __restrict__ w = J.job[j].w;
  const int rows = J.job[j].rows, p = J.job[j].p, steps = J.job[j].steps, vec = J.job[j].vec;
  const int row = (blockIdx.x - J.job[j].first) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float* r = w + (size_t)row * p;
  __nv_bfloat16* __restrict__ o = J.job[j].ws + (size_t)row * steps * (PARTS * BK);
#pragma unroll 4
  for (int k = 4 * lane; k < steps * BK; k += 128) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
      if (k < p) v = __ldg(reinterpret_cast<const float4*>(r + k));
    } else {
      if (k < p) v.x = r[k];
      if (k + 1 < p) v.y = r[k + 1];
      if (k + 2 < p) v.z = r[k + 2];
      if (k + 3 < p) v.w = r[k + 3];
    }
    uint2 hi, mid, lo;
    split_triple(v.x, v.y, hi.x, mid.x, lo.x);
    split_triple(v.z, v.w, hi.y, mid.y, lo.y);
    __nv_bfloat16* d = o + (k / BK) * (PARTS * BK) + k % BK;
    *reinterpret_cast<uint2*>(d) = hi;
    *reinterpret_cast<uint2*>(d + BK) = mid;
    *reinterpret_cast<uint2*>(d + 2 * BK) = lo;
  }
}

// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// the sum as the float32 kernels have it: one chain of fused multiply-adds in ascending k
__device__ __noinline__ float chain(const float* x, const float* w, int p) {
  float s = 0.f;
  for (int k = 0; k < p && s == s; ++k) s = fmaf(__ldg(x + k), __ldg(w + k), s);   // a NaN stays one
  return s;
}

template <int BN, bool GLU>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Params P) {
  using G = Geo<BN>;
  constexpr int NX = G::NX, NW = G::NW, NACC = G::NACC, NA = G::NA, CPW = BN / 2;          // accumulator columns of a flush warp
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* cvals = reinterpret_cast<float*>(smem + G::OFF_COLS);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);
  uint64_t* xfull = bars;                  // [NX] x has landed
  uint64_t* xempty = xfull + NX;           // [NX] and has been read by the converters
  uint64_t* wfull = xempty + NX;           // [NW] w has landed
  uint64_t* wempty = wfull + NW;           // [NW] and has been read by the MMAs
  uint64_t* afull = wempty + NW;           // [NA] the parts of x are in tensor memory
  uint64_t* aempty = afull + NA;           // [NA] and have been read
  uint64_t* tfull = aempty + NA;           // [NACC] the K block's sums are complete
  uint64_t* tempty = tfull + NACC;         // [NACC] the sums have been read
  uint64_t* cfull = tempty + NACC;         // [2] a tile's biases are there
  uint64_t* cempty = cfull + 2;            // [2] and have been used
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + G::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = tc::uniform_warp_id(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NX; ++s) { tc::mbar_init(xfull + s, 1); tc::mbar_init(xempty + s, CONV_WARPS); }
    for (int s = 0; s < NW; ++s) { tc::mbar_init(wfull + s, 1); tc::mbar_init(wempty + s, 1); }
    for (int b = 0; b < NA; ++b) { tc::mbar_init(afull + b, CONV_WARPS); tc::mbar_init(aempty + b, 1); }
    for (int b = 0; b < 2; ++b) { tc::mbar_init(cfull + b, 32); tc::mbar_init(cempty + b, FLUSH_WARPS); }
    for (int b = 0; b < NACC; ++b) { tc::mbar_init(tfull + b, 1); tc::mbar_init(tempty + b, FLUSH_WARPS); }
    *abort_flag = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tmX);
    tc::tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, G::TCOLS);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot, tmem_a = tmem + NACC * BN;       // buffer b from A_COLS b on
  pdl_wait();

  const int blocks = GLU ? 2 * P.steps : P.steps;    // K blocks of a tile; those of the GLU's factor follow those of its gate
  auto decode = [&](int tile, int& mt, int& nt, int& kb) {
    nt = tile % P.n_tiles;
    const int r = tile / P.n_tiles;
    mt = r % P.m_tiles;
    kb = r / P.m_tiles;
  };

  if (warp == 0) {
    // ---- TMA producer ----
    if (tc::elect_one()) {
      int xs = 0, ws = 0; uint32_t xphase = 0, wphase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total && ok; tile += gridDim.x) {
        int mt, nt, kb;
        decode(tile, mt, nt, kb);
        for (int c = 0; c < blocks; ++c) {
          const bool second = GLU && c >= P.steps;
          const int b = second ? kb + P.partner : kb, s = second ? c - P.steps : c;
          ok = tc::mbar_wait(xempty + xs, xphase ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY);
          if (!ok) break;
          unsigned char* sx = smem + xs * X_BYTES;
          tc::mbar_expect_tx(xfull + xs, X_BYTES);
          tc::tma_load_3d(sx, &tmX, xfull + xs, s * BK, b, mt * BM);
          tc::tma_load_3d(sx + BM * 128, &tmX, xfull + xs, s * BK + 32, b, mt * BM);
          if (++xs == NX) { xs = 0; xphase ^= 1; }
          ok = tc::mbar_wait(wempty + ws, wphase ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY);
          if (!ok) break;
          unsigned char* sw = smem + G::OFF_W + ws * G::W_BYTES;
          tc::mbar_expect_tx(wfull + ws, G::W_BYTES);
#pragma unroll
          for (int i = 0; i < PARTS; ++i)
            tc::tma_load_2d(sw + i * BN * 128, &tmW, wfull + ws, (s * PARTS + i) * BK, b * P.q + nt * BN);
          if (++ws == NW) { ws = 0; wphase ^= 1; }
        }
      }
      tc::drain_loads(xfull, NX, tc::ring_parities(xs, xphase));
      tc::drain_loads(wfull, NW, tc::ring_parities(ws, wphase));
    }
  } else if (warp == 1) {
    // ---- MMA issue ----
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::make_idesc(BM, BN, 1);
      const uint64_t w0 = tc::smem_desc_k_sw128(tc::smem_u32(smem + G::OFF_W));
      int stage = 0; uint32_t phase = 0, it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total && ok; tile += gridDim.x) {
        for (int c = 0; c < blocks; ++c, ++it) {
          const int buf = it % NACC, ab = it % NA;
          ok = tc::mbar_wait(wfull + stage, phase, abort_flag, tc::ST_TIMEOUT_TMA) &&
               tc::mbar_wait(tempty + buf, ((it / NACC) & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_MMA) &&
               tc::mbar_wait(afull + ab, (it / NA) & 1, abort_flag, tc::ST_TIMEOUT_MMA);
          if (!ok) break;
          tc::tc_fence_after();
          const uint32_t acc = tmem + buf * BN, a = tmem_a + ab * A_COLS, off = (uint32_t)(stage * (G::W_BYTES >> 4));
          constexpr int PART_X[6] = {2, 0, 1, 1, 0, 0}, PART_W[6] = {0, 2, 1, 0, 1, 0};      // small terms first
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              mma_ts(acc, a + 32 * PART_X[i] + 8 * kk, tc::desc_advance(w0, off + PART_W[i] * (BN * 128 >> 4) + 2 * kk), idesc, i || kk ? 1u : 0u);
          tc::mma_commit(wempty + stage);
          tc::mma_commit(aempty + ab);
          tc::mma_commit(tfull + buf);
          if (++stage == NW) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 2 && !GLU) {
    // ---- biases of the tiles ----
    uint32_t n = 0;
    for (int tile = blockIdx.x; tile < P.total; tile += gridDim.x, ++n) {
      int mt, nt, kb;
      decode(tile, mt, nt, kb);
      bool ok = tc::mbar_wait(cempty + (n & 1), ((n >> 1) & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      float* dst = cvals + (n & 1) * BN;
      for (int j = lane; j < BN; j += 32) dst[j] = P.bias && nt * BN + j < P.q ? __ldg(P.bias + (long long)kb * P.q + nt * BN + j) : 0.f;
      tc::mbar_arrive(cfull + (n & 1));
    }
  } else if (warp >= CONV0) {
    // ---- conversion: a thread owns one row of x ----
    const int group = (warp - CONV0) / CONV_WARPS, cw = warp & 3, r = cw * 32 + lane, sw = (r & 7) * 16;
    const uint32_t tq = tmem_a + ((uint32_t)(cw * 32) << 16);
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < P.total && ok; tile += gridDim.x) {
      for (int c = 0; c < blocks; ++c, ++it) {
        if ((int)(it & 1) != group) continue;
        const uint32_t stage = it % NX;
        ok = tc::mbar_wait(xfull + stage, (it / NX) & 1, abort_flag, tc::ST_TIMEOUT_TMA);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const unsigned char* p0 = smem + stage * X_BYTES + r * 128;
        uint4 v[16];
        uint32_t bits = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          v[j] = *reinterpret_cast<const uint4*>(p0 + (j < 8 ? 0 : BM * 128) + (((j & 7) * 16) ^ sw));
          bits |= v[j].x | v[j].y | v[j].z | v[j].w;
        }
        // The vote needs every lane's values, and its result decides who arrives (either may): the arrival finds all loads complete.
        // (Right behind the loads it overtook them, and the next rows landed under those that were still waiting for shared memory.)
        if (lane == __any_sync(0xffffffffu, bits == 1u)) tc::mbar_arrive(xempty + stage);
        const uint32_t ab = it % NA, ta = tq + ab * A_COLS;
        ok = tc::mbar_wait(aempty + ab, ((it / NA) & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_MMA);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc::tc_fence_after();
#pragma unroll
        for (int j = 0; j < 4; ++j) {                  // 16 columns: eight tensor-memory columns of pairs
          uint32_t hi[8], mid[8], lo[8];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const uint4& q = v[4 * j + (i >> 1)];
            split_triple(__uint_as_float(q.x), __uint_as_float(q.y), hi[i], mid[i], lo[i]);
            split_triple(__uint_as_float(q.z), __uint_as_float(q.w), hi[i + 1], mid[i + 1], lo[i + 1]);
          }
          tmem_st8(ta + 8 * j, hi);
          tmem_st8(ta + 32 + 8 * j, mid);
          tmem_st8(ta + 64 + 8 * j, lo);
        }
        tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(afull + ab);
      }
    }
  } else if (warp >= FLUSH0) {
    // ---- K-block sums to float32 registers, then the tile's results ----
    const int quarter = warp & 3, half = (warp - FLUSH0) >> 2;
    const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16) + half * CPW;
    uint32_t it = 0, n = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < P.total && ok; tile += gridDim.x, ++n) {
      int mt, nt, kb;
      decode(tile, mt, nt, kb);
      f32x2 acc[GLU ? 2 : 1][CPW / 2];
#pragma unroll
      for (int g = 0; g < (GLU ? 2 : 1); ++g) {
#pragma unroll
        for (int j = 0; j < CPW / 2; ++j) acc[g][j] = 0;
        for (int c = 0; c < P.steps; ++c, ++it) {
          const int buf = it % NACC;
          ok = tc::mbar_wait(tfull + buf, (it / NACC) & 1, abort_flag, tc::ST_TIMEOUT_EPI);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc::tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < CPW; c0 += 16) {
            uint32_t t[16];
            tc::tmem_ld16(tl + buf * BN + c0, t);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              acc[g][c0 / 2 + j] = f2_add(f2_pack(__uint_as_float(t[2 * j]), __uint_as_float(t[2 * j + 1])), acc[g][c0 / 2 + j]);
          }
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(tempty + buf);
        }
      }
      if (!ok) break;
      if (!GLU) {
        ok = tc::mbar_wait(cfull + (n & 1), (n >> 1) & 1, abort_flag, tc::ST_TIMEOUT_EPI);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      const int t = mt * BM + quarter * 32 + lane, c0 = nt * BN + half * CPW;
      const long long base = (long long)(t / P.L) * P.osb + (long long)(t % P.L) * P.ost;
      const float* cv = cvals + (n & 1) * BN + half * CPW;
      float* orow = P.out + base + ((long long)kb * P.q + c0) * P.osc;
      float bad = 0.f;                       // a NaN where a result is not finite
      uint32_t least = ~0u;                  // twice the smallest result's bits but its sign, less one: zeros are the largest
#pragma unroll
      for (int j8 = 0; j8 < CPW; j8 += 8) {
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          float a0, a1, a2, a3;
          if (GLU) {
            float n0, n1, n2, n3;
            f2_unpack(acc[0][(j8 + j) / 2], a0, a1);
            f2_unpack(acc[0][(j8 + j) / 2 + 1], a2, a3);
            f2_unpack(acc[GLU ? 1 : 0][(j8 + j) / 2], n0, n1);
            f2_unpack(acc[GLU ? 1 : 0][(j8 + j) / 2 + 1], n2, n3);
            a0 = gelu_erf(a0) * n0; a1 = gelu_erf(a1) * n1; a2 = gelu_erf(a2) * n2; a3 = gelu_erf(a3) * n3;
          } else {
            const float4 b = *reinterpret_cast<const float4*>(cv + j8 + j);
            f2_unpack(f2_add(acc[0][(j8 + j) / 2], f2_pack(b.x, b.y)), a0, a1);
            f2_unpack(f2_add(acc[0][(j8 + j) / 2 + 1], f2_pack(b.z, b.w)), a2, a3);
          }
          bad = fmaf(0.f, a0, fmaf(0.f, a1, fmaf(0.f, a2, fmaf(0.f, a3, bad))));
          least = min(min(least, 2 * __float_as_uint(a0) - 1), min(2 * __float_as_uint(a1) - 1, min(2 * __float_as_uint(a2) - 1, 2 * __float_as_uint(a3) - 1)));
          v[j] = __float_as_uint(a0); v[j + 1] = __float_as_uint(a1); v[j + 2] = __float_as_uint(a2); v[j + 3] = __float_as_uint(a3);
        }
        if (t >= P.tokens) continue;
        if (P.vec && c0 + j8 + 8 <= P.q) {
          stg256(orow + j8, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (c0 + j8 + j < P.q) orow[(j8 + j) * P.osc] = __uint_as_float(v[j]);
        }
      }
      __syncwarp();
      if (!GLU && lane == 0) tc::mbar_arrive(cempty + (n & 1));
      if ((bad != bad || least < 2 * TINY - 1) && t < P.tokens) {
        const float* xr = P.x + (long long)t * P.ldx + (long long)kb * P.p;
        for (int j = 0; j < CPW && c0 + j < P.q; ++j) {
          const long long c = (long long)kb * P.q + c0 + j;
          float* po = P.out + base + c * P.osc;
          const float size = fabsf(*po);
          if (size == 0.f || (size >= __uint_as_float(TINY) && size <= 3.402823466e38f)) continue;
          float v = chain(xr, P.w + c * P.p, P.p);
          if (GLU) v = gelu_erf(v) * chain(xr + (long long)P.partner * P.p, P.w + (c + (long long)P.partner * P.q) * P.p, P.p);
          else if (P.bias) v += __ldg(P.bias + c);
          *po = v;
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, G::TCOLS);
  }
}

// float32 rows {p (contiguous), nb blocks, tokens}, box 32 x 1 x 128, 128-byte swizzle, zeros out of range
static int make_tmap_rows(CUtensorMap* map, const void* base, uint64_t p, uint64_t nb, uint64_t tokens, uint64_t ld) {
  m2_encode_tiled_fn enc;
  int rc = m2_get_encode_fn(&enc);
  if (rc) return rc;
  cuuint64_t dims[3] = {p, nb, tokens};
  cuuint64_t strides[2] = {p * 4, ld * 4};
  cuuint32_t box[3] = {32, 1, BM};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return m2_set_error(M2_ERR_CUDA, "cuTensorMapEncodeTiled (float32) failed with code %d", (int)r);
  return M2_OK;
}

template <int BN, bool GLU>
static int launch(Params& P, int nblocks, cudaStream_t st) {
  CUtensorMap tmX, tmW;
  int rc;
  const uint64_t rows = (uint64_t)nblocks * P.q, pitch = (uint64_t)P.steps * PARTS * BK;
  if ((rc = make_tmap_rows(&tmX, P.x, P.p, nblocks, P.tokens, P.ldx))) return rc;
  if ((rc = m2_make_tmap_bf16_2d(&tmW, P.ws, rows, pitch, pitch, BN))) return rc;
  P.n_tiles = (P.q + BN - 1) / BN;
  P.m_tiles = (P.tokens + BM - 1) / BM;
  P.total = P.n_tiles * P.m_tiles * (GLU ? nblocks / 2 : nblocks);
  auto kern = gemm_split_kernel<BN, GLU>;
  constexpr int SMEM = Geo<BN>::SMEM;
  M2_SMEM_ONCE(kern, SMEM);
  const int sms = m2_sm_count();
  return m2_launch("gemm_split_kernel", (long long)P.tokens * P.p * nblocks, kern, P.total < sms ? P.total : sms, THREADS, SMEM, st, tmX, tmW, P);
}

// Columns of a tile: a K block of 64 takes some 2300 clocks at 128 columns, 1490 at 64, 1130 at 32 (768 -> 2304, 8192 rows: 138, 169, 245 us
// with each width alone).  Over 25 shapes from 1 to 8192 rows the width picked so is the fastest of the three or within 2 % of it.
static int pick_bn(const Params& P, int blocks) {
  const int sms = m2_sm_count();
  auto cost = [&](int bn, double per) {
    const long long tiles = (long long)((P.tokens + BM - 1) / BM) * ((P.q + bn - 1) / bn) * blocks;
    return (double)((tiles + sms - 1) / sms) * P.steps * per;
  };
  const double c128 = cost(128, 2300), c64 = cost(64, 1490), c32 = cost(32, 1130);
  return c128 <= c64 && c128 <= c32 ? 128 : (c64 <= c32 ? 64 : 32);
}

// Below 128 products a chain is about as exact (68 columns: 1.3e-7 of the result) and as fast (36 columns, 100 rows: 10.3 us both).
static bool columns_ok(int p) { return p >= 2 * BK && p % 4 == 0; }
// What the TMA loads need: rows that start on 16-byte boundaries; `ws` as m2_split_weights writes it.
static bool rows_ok(const void* x, long long ld, const void* ws, int p) {
  return ws && columns_ok(p) && ld % 4 == 0 && m2_aligned(x, 16) && m2_aligned(ws, 16);
}
static size_t split_halves(long long rows, int p) { return (size_t)rows * ((p + BK - 1) / BK) * PARTS * BK; }
static void set_weights(Params& P, const void* w, const void* ws) {
  P.w = (const float*)w;
  P.ws = (const __nv_bfloat16*)ws;
  P.steps = (P.p + BK - 1) / BK;
}

static int run(Params& P, int blocks, cudaStream_t st) {
  const int bn = pick_bn(P, blocks);
  if (bn == 128) return launch<128, false>(P, blocks, st);
  if (bn == 64) return launch<64, false>(P, blocks, st);
  return launch<32, false>(P, blocks, st);
}

}  // namespace f32s

bool linear_split_supported(const m2_linear_args* a) {
  return a->dtype == M2_F32 && !a->force_simt && a->x_sc == 1 && (a->batch == 1 || a->x_sb == (long long)a->seq_len * a->x_st) &&
         a->x_st >= a->in_features && f32s::rows_ok(a->x, a->x_st, a->w_split, a->in_features);
}

int linear_split_launch(const m2_linear_args* a, cudaStream_t st) {
  f32s::Params P = {};
  P.x = (const float*)a->x; P.ldx = a->x_st;
  P.bias = a->bias;
  P.out = (float*)a->out; P.osb = a->out_sb; P.ost = a->out_st; P.osc = a->out_sc;
  P.tokens = a->batch * a->seq_len; P.L = a->seq_len; P.p = a->in_features; P.q = a->out_features;
  f32s::set_weights(P, a->w, a->w_split);
  P.vec = a->out_sc == 1 && m2_aligned(a->out, 32) && a->out_st % 8 == 0 && (a->batch == 1 || a->out_sb % 8 == 0);
  return f32s::run(P, 1, st);
}

bool blockdiag_split_supported(const m2_blockdiag_args* a) {
  return a->dtype == M2_F32 && a->in_features == a->nblocks * a->p && a->out_features == a->nblocks * a->q && a->ldx >= a->in_features &&
         f32s::rows_ok(a->x, a->ldx, a->w_split, a->p);
}

int blockdiag_split_launch(const m2_blockdiag_args* a, cudaStream_t st) {
  f32s::Params P = {};
  P.x = (const float*)a->x; P.ldx = a->ldx;
  P.bias = a->bias;
  P.out = (float*)a->out; P.ost = a->ldo; P.osc = 1;
  P.tokens = P.L = a->m; P.p = a->p; P.q = a->q;
  f32s::set_weights(P, a->w, a->w_split);
  P.vec = m2_aligned(a->out, 32) && a->ldo % 8 == 0 && a->q % 8 == 0;
  return f32s::run(P, a->nblocks, st);
}

bool glu_split_supported(const m2_glu_args* a) {
  return a->dtype == M2_F32 && a->ldx >= a->d_model && f32s::rows_ok(a->x, a->ldx, a->wg_split, a->d_model / a->nblocks);
}

int glu_split_launch(const m2_glu_args* a, cudaStream_t st) {
  f32s::Params P = {};
  P.x = (const float*)a->x; P.ldx = a->ldx;
  P.out = (float*)a->h; P.ost = a->ldh; P.osc = 1;
  P.tokens = P.L = a->m; P.p = a->d_model / a->nblocks; P.q = 2 * a->inter / a->nblocks;
  P.partner = a->nblocks / 2;
  f32s::set_weights(P, a->wg, a->wg_split);
  P.vec = m2_aligned(a->h, 32) && a->ldh % 8 == 0 && P.q % 8 == 0;
  return f32s::launch<64, true>(P, a->nblocks, st);
}

struct WeightRows { const void* w; long long rows; int p; void* out; };
// One launch for up to four matrices; `elements` as in m2_launch.
static int split_weights_launch(const WeightRows* rows, int n, long long elements, cudaStream_t st) {
  using namespace f32s;
  SplitJobs J = {};
  long long blocks = 0;
  for (int i = 0; i < n; ++i) {
    const WeightRows& r = rows[i];
    M2_REQUIRE(r.rows > 0 && r.rows < (1LL << 31) - 8 && r.p > 0, M2_ERR_ARG, "m2_split_weights: bad sizes rows=%lld p=%d", r.rows, r.p);
    M2_REQUIRE(r.w && r.out, M2_ERR_ARG, "m2_split_weights: NULL pointer");
    M2_REQUIRE(m2_aligned(r.out, 16), M2_ERR_ALIGN, "m2_split_weights: out must be 16-byte aligned");
    J.job[i] = {static_cast<const float*>(r.w), static_cast<__nv_bfloat16*>(r.out), (int)r.rows, r.p, (r.p + BK - 1) / BK, (int)blocks,
                r.p % 4 == 0 && m2_aligned(r.w, 16)};
    blocks += (r.rows + 7) / 8;
  }
  M2_REQUIRE(blocks < (1LL << 31), M2_ERR_UNSUPPORTED, "m2_split_weights: too many rows");
  J.n = n;
  return m2_launch("split_weights_kernel", elements, split_weights_kernel, (unsigned)blocks, 256, 0, st, J);
}

}  // namespace m2

extern "C" size_t m2_split_weights_bytes(long long rows, int p) {
  if (rows <= 0 || p <= 0) return 0;
  return m2::f32s::split_halves(rows, p) * 2;
}

extern "C" int m2_split_weights_used(int p) { return m2::f32s::columns_ok(p); }

extern "C" int m2_split_weights(const float* w, long long rows, int p, void* out, void* stream) {
  const m2::WeightRows r = {w, rows, p, out};
  return m2::split_weights_launch(&r, 1, rows * p, static_cast<cudaStream_t>(stream));
}
