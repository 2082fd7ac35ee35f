// Fused gated long convolution of family 0 (float32 taps and residual input) on bf16 activations in time-contiguous rows, up to 2048
// steps: block-Toeplitz GEMMs over pairs of fp16 values, with a warp for every part of the work.  For callers that ask for it
// (rows_padded): the modules take the float32 transform at these lengths, whatever the batch.
//
// The product is that of longconv_bt.cu: a sequence is cut into NB = ceil(L / 128) blocks, the Toeplitz block of a distance
// delta is the MMA's A operand, all (block, sequence) pairs of a tile of Bt sequences its columns:
//   D[128 steps n, columns (jt, b)] += T_delta[128 x 128] . X[128 steps k, columns (js = jt - delta, b)].
// There one group of warps loads, builds strips, gates and writes in turn and two CTAs of an SM overlap by chance.  Here one
// CTA per SM keeps four things under way at once: eight warps bring the operands of the next filter, three build the strips of
// the next two deltas, one thread issues MMAs, eight warps turn finished accumulators into outputs.  A filter's operand and its
// 256 accumulator columns are free again while the other filter's MMAs run, so two filters alternate without a second buffer.
//
// Taps h (bias folded into h(0)) and the residual input u are float32.  Each is scaled by a power of two (taps
// per channel, u per channel and sequence, as is v * x1) that brings its largest value to [2^14, 2^15) and written as hi + lo, two
// fp16 values that keep 22 bits; v * x1 is a bf16 value, which one fp16 value holds exactly down to 2^-31 of the largest.  The products are
// lo.hi + hi.hi for v * x1 and lo.hi + hi.lo + hi.hi for u, accumulated in float32, the small terms apart.  An accumulation
// in tensor memory drops what does not fit, always towards zero, and up to 128 follow one another: before the rounding to bf16 the
// sums are off by 2.2e-7 / 1.7e-6 / 2.6e-6 / 3.5e-6 of the result at 129 / 1000 / 1531 / 2045 steps of random data, 1.7e-5 at 2045
// where inputs and taps have one sign (the transform: 0.8e-7 to 1.5e-7).  Taken out of tensor memory and added up in float32 every
// 64 steps they were off by 1.2e-7 to 2.5e-7, and 6 x 1531 through twelve layers took 6048 us (transform 5950).  Any non-finite value makes all outputs of its row NaN, as in a transform.
//
// Bound: the MMAs, which shared memory feeds: each reads 4 KB of strip and 32 bytes a column, 56 to 60 clocks beside the other warps'
// traffic (6 x 1531 at 768 channels: 920 a unit, 55 of its 63 thousand clocks); units that fill the SMs unevenly (five or six each);
// few or short sequences by one unit's chain of latencies, 9 thousand clocks.  longconv_bts_f32_preferred draws the line.
// Measured (us, L2 flushed; the transform on token rows first): 6 x 1531 391 -> 211, 8 x 2045 640 -> 310, 16 x 1000 463 -> 196, 16 x 514
// 338 -> 117, 30 x 300 316 -> 113, 40 x 61 81 -> 65.  Against 64-bit arithmetic both are off by the same: 1.8129e-3 at 6 x 1531, 1.7756e-3
// at 16 x 1000, 1.7153e-3 at 40 x 61 (bf16 roundings all but some 1e-6 of it).  With the gate's values loaded when the accumulators were
// complete and the gated result passed through the output tensor 6 x 1531 took 252 us.
//
// Computation replaced: bert/src/mm/monarch_mixer_sequence_mixer.py:109-149 and
// bert/src/mm/hyena_utils.py:16-42, :219-248 of the reference.
#include "tc_common.cuh"

namespace m2 {
namespace bts {

constexpr int BUILD0 = 1, BUILD_WARPS = 3, LOAD0 = 4, LOAD_WARPS = 8, EPI0 = 12, EPI_WARPS = 8;   // five warps to a scheduler
constexpr int THREADS = 32 * (EPI0 + EPI_WARPS);
constexpr int MAX_L = 2048;
constexpr int WROWS = 368;                      // strip rows of two deltas: 2 * 128 + 112
constexpr int SLOTS = 4;                        // units whose scales are kept
constexpr int REGION = 256;                     // accumulator columns of a filter
constexpr int BATCHES = 8;                      // of eight columns in an epilogue warp, two warps to a quarter of the lanes
constexpr int MAXCOLS = 16 * BATCHES;
constexpr int SMALL = 128;                      // where the columns of the small terms start in a region

__host__ __device__ constexpr int tap_count(int nb) { return 256 * nb + 64; }   // taps of a channel, d = -128 nb ..
__host__ __device__ constexpr int window_rows(int nb) { return nb == 1 ? 240 : WROWS; }

struct Params {
  int B, L, D, nf, NB, Bt, cols, ntile, units, ksteps;
  int u_bf16, yu_bf16;
  const __nv_bfloat16* xin; long long xsb, xsc;
  const void* u; long long usb, usc;
  __nv_bfloat16* out; long long osb, ost, osc;
  const float* sw; const float* sb;
  const float* spec[2];                         // float32 taps, then the largest of each channel but h(0)
  const float* bias[2];
};

struct Layout { uint32_t u, win, taps, raw, row, xinv, smax, tinv, bars, total; };
__host__ __device__ inline Layout layout_of(int cols, int nb) {
  Layout l;
  const uint32_t reg = (uint32_t)(cols + 16) * 256;
  l.u = reg;                                        // hi and lo
  l.win = l.u + 2 * reg;
  l.taps = l.win + 4 * window_rows(nb) * 32;         // two windows, two segments, hi and lo each
  l.raw = l.taps + 4 * tap_count(nb) * 2;
  l.row = l.raw + tap_count(nb) * 4;
  l.xinv = l.row + MAXCOLS * 4;
  l.smax = l.xinv + 2 * SLOTS * MAXCOLS * 4;
  l.tinv = l.smax + 2 * 2 * MAXCOLS * 4;
  l.bars = l.tinv + 2 * SLOTS * 4;
  l.total = l.bars + 24 * 8 + 16;
  return l;
}

// ---- table of family 0: float32 taps h(d) at index d + 128 NB (zero for |d| >= L, without the bias), then per channel the largest
// magnitude of d != 0 (NaN where any tap is not finite) ----
__global__ void __launch_bounds__(256)
taps_f32_kernel(const float* __restrict__ kfilt, float* __restrict__ taps, int D, int L, int R, int nb) {
  __shared__ float red[8];
  const int c = blockIdx.x, tid = threadIdx.x, n = tap_count(nb);
  const float* row = kfilt + (size_t)c * R;
  float* T = taps + (size_t)c * n;
  float m = 0.f;
  int bad = 0;
  for (int i = tid; i < n; i += blockDim.x) {
    const int d = i - 128 * nb;
    const float v = d > -L && d < L ? row[d > 0 ? R - d : -d] : 0.f;
    T[i] = v;
    bad |= !(fabsf(v) <= 3.402823466e38f);
    if (d != 0) m = fmaxf(m, fabsf(v));
  }
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) red[tid >> 5] = m;
  bad = __syncthreads_or(bad);
  if (tid == 0) {
    for (int i = 1; i < 8; ++i) m = fmaxf(m, red[i]);
    taps[(size_t)D * n + c] = bad ? __int_as_float(0x7fffffff) : m;
  }
}

template <int ID, int N> __device__ __forceinline__ void group_sync() { asm volatile("barrier.cta.sync %0, %1;" ::"n"(ID), "n"(N) : "memory"); }

// the largest magnitude's biased exponent -> scale that brings it to [2^14, 2^15), and its inverse
__device__ __forceinline__ float split_scale(uint32_t ex) { return __uint_as_float((268u - ex) << 23); }
__device__ __forceinline__ float split_inverse(uint32_t ex) { return __uint_as_float((ex - 14u) << 23); }
__device__ __forceinline__ uint32_t split_exponent(float m) { return max(27u, __float_as_uint(m) >> 23); }
__device__ __forceinline__ void split_pair(float y0, float y1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(y0, y1);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(y0 - hf.x, y1 - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// scale of a row whose largest magnitude is m: NaN (and with it the whole row) where m is not finite
__device__ __forceinline__ float row_scale(float m) { return m <= 3.402823466e38f ? split_scale(split_exponent(m)) : __int_as_float(0x7fffffff); }
__device__ __forceinline__ float row_inverse(float m) { return m <= 3.402823466e38f ? split_inverse(split_exponent(m)) : __int_as_float(0x7fffffff); }

__global__ void __launch_bounds__(THREADS, 1)
longconv_bts_kernel(const Params P) {
  using namespace lcl;
  constexpr int PL = 2;                              // planes of the taps and of u: hi, lo
  extern __shared__ __align__(128) unsigned char smem[];
  const Layout LY = layout_of(P.cols, P.NB);
  const int tid = threadIdx.x, warp = tc::uniform_warp_id(), lane = tid & 31;
  const int cols = P.cols, Bt = P.Bt, NB = P.NB, L = P.L;
  const uint32_t LBO = (uint32_t)(cols + 16) * 16, REG = LBO * 16;
  const uint32_t wrows = window_rows(NB), WB = wrows * 32, TB = (uint32_t)tap_count(NB) * 2;
  const uint32_t base = tc::smem_u32(smem), opa = base, opu = base + LY.u, win = base + LY.win, taps = base + LY.taps;
  uint32_t* rowjb = reinterpret_cast<uint32_t*>(smem + LY.row);        // operand row -> block << 16 | sequence
  float* xinv = reinterpret_cast<float*>(smem + LY.xinv);              // [f][slot][128]
  int* smax = reinterpret_cast<int*>(smem + LY.smax);                  // [f][unit & 1][128]
  float* tinv = reinterpret_cast<float*>(smem + LY.tinv);              // [f][slot]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + LY.bars);
  uint64_t* opfull = bars;                 // [2] a filter's operand is written
  uint64_t* opempty = opfull + 2;          // [2] and has been read
  uint64_t* wfull = opempty + 2;           // [2] a strip window is written
  uint64_t* wempty = wfull + 2;            // [2] and has been read
  uint64_t* tfull = wempty + 2;            // [2] a filter's accumulators are complete
  uint64_t* tempty = tfull + 2;            // [2] and have been read
  uint64_t* hfull = tempty + 2;            // a segment's float32 taps have landed
  uint64_t* sfull = hfull + 1;             // [f][slot] the scales of a unit are written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(opfull + i, LOAD_WARPS / 2);
      tc::mbar_init(opempty + i, 1);
      tc::mbar_init(wfull + i, BUILD_WARPS);
      tc::mbar_init(wempty + i, 1);
      tc::mbar_init(tfull + i, 1);
      tc::mbar_init(tempty + i, EPI_WARPS);
    }
    for (int i = 0; i < 2 * SLOTS; ++i) tc::mbar_init(sfull + i, LOAD_WARPS / 2 + BUILD_WARPS);
    tc::mbar_init(hfull, 1);
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  for (int r = tid; r < cols; r += THREADS) rowjb[r] = (uint32_t)(r / Bt) << 16 | (uint32_t)(r % Bt);
  for (int i = tid; i < 2 * 2 * MAXCOLS; i += THREADS) smax[i] = 0;
  // eight zero rows before and behind the data of every plane, which an MMA of N = 16 n takes beside its own
  for (int i = tid; i < 16 * 16 * (1 + PL); i += THREADS) {
    const uint32_t plane = i >> 4, r = i & 15;
    sts128((plane < 16 ? opa + plane * LBO : opu + (plane - 16) * LBO) + (r < 8 ? r : cols + r) * 16, 0u, 0u, 0u, 0u);
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tm = *tmem_slot;
  pdl_wait();

  const int u0 = (int)((long long)blockIdx.x * P.units / gridDim.x), u1 = (int)((long long)(blockIdx.x + 1) * P.units / gridDim.x);
  const int wpos = (NB + 1) >> 1, nwin = wpos + (NB >> 1);      // windows of deltas 0.., then of deltas -1 downwards
  auto window = [&](int s, int& dlo, int& dhi) {
    dlo = s < wpos ? 2 * s : max(1 - NB, -2 * (s - wpos + 1));
    dhi = s < wpos ? min(NB - 1, 2 * s + 1) : -2 * (s - wpos) - 1;
  };

  if (warp == 0) {
    // ---- MMA issue ----
    if (tc::elect_one()) {
      bool ok = true;
      uint32_t w = 0, n = 0;
      for (int unit = u0; unit < u1 && ok; ++unit, ++n) {
        for (int f = 0; f < P.nf && ok; ++f) {
          ok = tc::mbar_wait(tempty + f, (n & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_MMA) &&
               tc::mbar_wait(opfull + f, n & 1, abort_flag, tc::ST_TIMEOUT_TMA);
          if (!ok) break;
          const uint32_t data = f ? opu : opa;
          // (taps, data) planes of the products, small terms first
          const int products = f && !P.u_bf16 ? 3 : 2;
          for (int s = 0; s < nwin && ok; ++s, ++w) {
            int dlo, dhi;
            window(s, dlo, dhi);
            ok = tc::mbar_wait(wfull + (w & 1), (w >> 1) & 1, abort_flag, tc::ST_TIMEOUT_TMA);
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t wb = win + (w & 1) * PL * WB;
            for (int d = dlo; d <= dhi; ++d) {
              const int nc = (NB - abs(d)) * Bt, e = (16 - (nc & 15)) & 15;    // e = 0 or 8 zero rows
              const uint32_t idesc = tc::make_idesc(128, nc + e, 0);
              const uint32_t dcol = tm + f * REGION + (d > 0 ? d * Bt - e : 0);
              const uint32_t brow = data + 16 * (8 + (d > 0 ? -e : -d * Bt));
              const uint32_t arow = wb + 16 * (112 + 128 * (d - dlo));
              constexpr uint32_t hi = (128u >> 4) | 1u << 14;                  // 128 bytes between row groups, version
              const uint32_t step = LBO >> 3;
              for (int p = 0; p < products; ++p) {
                const uint32_t ap = p == 0 ? WB : 0, bp = products == 3 && p == 1 ? REG : 0;
                const uint32_t acc = p + 1 < products ? dcol + SMALL : dcol;      // small terms have columns of their own
                const uint32_t alo = ((arow + ap) >> 4) | wrows << 16, blo = ((brow + bp) >> 4) | (LBO >> 4) << 16;
                tc::mma_ss(acc, tc::desc_words(alo, hi), tc::desc_words(blo, hi), idesc,
                           (s != 0 || d != 0 || (p != 0 && p + 1 < products)) ? 1u : 0u);
                if (P.ksteps == 8) {
#pragma unroll
                  for (int kk = 1; kk < 8; ++kk) tc::mma_ss(acc, tc::desc_words(alo - 16 * kk, hi), tc::desc_words(blo + step * kk, hi), idesc, 1u);
                } else {
                  for (int kk = 1; kk < P.ksteps; ++kk) tc::mma_ss(acc, tc::desc_words(alo - 16 * kk, hi), tc::desc_words(blo + step * kk, hi), idesc, 1u);
                }
              }
            }
            tc::mma_commit(wempty + (w & 1));
          }
          if (!ok) break;
          tc::mma_commit(opempty + f);
          tc::mma_commit(tfull + f);
        }
      }
    }
  } else if (warp < LOAD0) {
    // ---- strips ----
    const int bt = tid - 32 * BUILD0;
    uint32_t w = 0, n = 0, seg = 0;
    bool ok = true;
    // the taps of a segment (one filter of one unit) are fetched while the strips of the one before are built
    uint32_t fetched = 1u;                           // parity of the last fetch
    auto fetch_taps = [&](uint32_t s) {
      const uint32_t k = s / P.nf, f = s - k * P.nf;
      if (bt != 0 || u0 + (int)k >= u1) return;
      fetched = s & 1u;
      const size_t c = (u0 + k) / P.ntile;
      tc::mbar_expect_tx(hfull, 2 * TB);
      tc::bulk_load(smem + LY.raw, P.spec[f] + c * (TB / 2), 2 * TB, hfull);
    };
    fetch_taps(0);
    bool go = true;                                  // the same for all warps of the role, `ok` is the warp's own
    for (int unit = u0; unit < u1 && go; ++unit, ++n) {
      const int c = unit / P.ntile;
      for (int f = 0; f < P.nf && go; ++f, ++seg) {
        const uint32_t tb = taps + (seg & 1) * PL * TB;
        const int slot = f * SLOTS + (n & (SLOTS - 1));
        const uint32_t T = base + LY.raw;
        const float m0 = __ldg(P.spec[f] + (size_t)P.D * (TB / 2) + c), hb = __ldg(P.bias[f] + c);
        go = ok = tc::group_and<2, 32 * BUILD_WARPS>(ok && tc::mbar_wait(hfull, seg & 1, abort_flag, tc::ST_TIMEOUT_TMA));
        if (!go) break;
        const float h0 = __uint_as_float(lds32(T + 4 * 128 * NB)) + hb;
        const float m = m0 <= 3.402823466e38f && fabsf(h0) <= 3.402823466e38f ? fmaxf(m0, fabsf(h0)) : __int_as_float(0x7f800000);
        const float sc = row_scale(m);
        if (bt == 0) tinv[slot] = row_inverse(m);
        for (uint32_t i = 2 * bt; i < TB / 2; i += 2 * 32 * BUILD_WARPS) {
          uint32_t t0, t1, hi, lo;
          asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(t0), "=r"(t1) : "r"(T + 4 * i));
          split_pair((i == 128u * NB ? h0 : __uint_as_float(t0)) * sc, __uint_as_float(t1) * sc, hi, lo);   // 128 NB is even
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tb + 2 * i), "r"(hi) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tb + TB + 2 * i), "r"(lo) : "memory");
        }
        group_sync<2, 32 * BUILD_WARPS>();           // the taps are there; those of the filter before the last have been read by all
        fetch_taps(seg + 1);
        if (lane == 0) tc::mbar_arrive(sfull + slot);
        for (int s = 0; s < nwin; ++s, ++w) {
          int dlo, dhi;
          window(s, dlo, dhi);
          const uint32_t wn = 128 * (dhi - dlo + 1) + 112;
          ok = tc::mbar_wait(wempty + (w & 1), ((w >> 1) & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_MMA);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;                            // this warp; the others hear of it at the next segment's barrier
          // strip row m: taps h(i - m + 112 - 128 dlo), i = 0 .. 15, the first and the last eight in planes of their own
          const int pbase = 112 - 128 * dlo + 128 * NB;
#pragma unroll
          for (int pl = 0; pl < PL; ++pl) {
            const uint32_t tg = tb + pl * TB, wg = win + ((w & 1) * PL + pl) * WB;
            // rows m (even, its taps start on a word) and m + 1 (one tap earlier): nine words make both
#pragma unroll 2
            for (uint32_t m = 2 * bt; m < wn; m += 2 * 32 * BUILD_WARPS) {
              const uint32_t wa = tg + 2 * (pbase - (int)m) - 4;
              uint32_t x[9];
#pragma unroll
              for (int i = 0; i < 9; ++i) x[i] = lds32(wa + 4 * i);
              const uint32_t o = wg + m * 16;
              sts128(o, x[1], x[2], x[3], x[4]);
              sts128(o + wrows * 16, x[5], x[6], x[7], x[8]);
              uint32_t y[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) y[i] = __byte_perm(x[i], x[i + 1], 0x5432u);
              sts128(o + 16, y[0], y[1], y[2], y[3]);
              sts128(o + wrows * 16 + 16, y[4], y[5], y[6], y[7]);
            }
          }
          tc::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(wfull + (w & 1));
        }
      }
    }
    if (bt == 0) tc::drain_loads(hfull, 1, fetched);
  } else if (warp < EPI0) {
    // ---- operands: four warps for v * x1, four for the residual input; a warp covers 64 bytes of eight rows, a quarter warp writes
    // one core matrix ----
    const int f = warp >= LOAD0 + LOAD_WARPS / 2, lw = warp & 3, lt = 32 * lw + lane;
    const int okc = 4 * lw + (lane >> 3), orow = lane & 7;
    const int iters = cols >> 3;
    const uint32_t op = (f ? opu : opa) + okc * LBO + (8 + orow) * 16;           // this thread's chunk of the first eight rows
    constexpr int U = 4;
    uint32_t n = 0;
    bool ok = f < P.nf;
    for (int unit = u0; unit < u1 && ok; ++unit, ++n) {
      const int c = unit / P.ntile, b0 = (unit - c * P.ntile) * Bt;
      const int slot = n & (SLOTS - 1);
      // steps of row k (0: none), and where it starts
      auto where = [&](int k, long long sb, long long sc, long long& off) {
        if (k >= cols) return 0;
        const uint32_t jb = rowjb[k];
        const int j = jb >> 16, b = b0 + (int)(jb & 0xffffu);
        off = c * sc + b * sb + 128 * j;
        return b < P.B ? min(128, L - 128 * j) : 0;
      };
      // the largest magnitude of each sequence: of eight values of this thread, then of the row, then of its blocks
      int* mx = smax + (2 * f + (n & 1)) * 128;
      auto maximum = [&](int k, float m) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        if (lane < 8 && k < cols) atomicMax(mx + (rowjb[k] & 0xffffu), __float_as_int(m));
      };
      // between the maxima and the conversion; then the other unit's are cleared
      auto maxima_done = [&]() {
        if (f) group_sync<3, 16 * LOAD_WARPS>(); else group_sync<1, 16 * LOAD_WARPS>();
        if (lt < Bt) {
          xinv[(f * SLOTS + slot) * 128 + lt] = row_inverse(__int_as_float(mx[lt]));
          smax[(2 * f + ((n & 1) ^ 1)) * 128 + lt] = 0;
        }
      };
      if (f == 0) {
        // ---- x1, v: short conv, product ----
        const Taps tx = load_taps(P.sw, P.sb, c), tv = load_taps(P.sw, P.sb, 2 * P.D + c);
        const f32x2 w0 = f2_pack(tx.w0, tv.w0), w1 = f2_pack(tx.w1, tv.w1), w2 = f2_pack(tx.w2, tv.w2), wb = f2_pack(tx.b, tv.b);
        const long long vdist = 2LL * P.D * P.xsc;
#pragma unroll 1
        for (int k0 = 0; k0 < iters; k0 += U) {
          uint4 x[U], v[U];
          uint32_t px[U], pv[U];
          int lim[U];
#pragma unroll
          for (int i = 0; i < U; ++i) {
            x[i] = v[i] = make_uint4(0u, 0u, 0u, 0u);
            px[i] = pv[i] = 0u;
            long long off = 0;
            const int k = 8 * (k0 + i) + orow;
            lim[i] = where(k, P.xsb, P.xsc, off);
            if (8 * okc < lim[i]) {
              const __nv_bfloat16* xr = P.xin + off + 8 * okc;
              x[i] = __ldg(reinterpret_cast<const uint4*>(xr));
              v[i] = __ldg(reinterpret_cast<const uint4*>(xr + vdist));
              if (lane < 8 && (okc > 0 || k >= Bt)) {          // the two steps before the warp's first chunk of a row
                px[i] = __ldg(reinterpret_cast<const uint32_t*>(xr - 2));
                pv[i] = __ldg(reinterpret_cast<const uint32_t*>(xr + vdist - 2));
              }
            }
          }
          if (k0 == 0) {                             // the first loads are on their way
            // (the maxima are cleared when all are here)
            ok = tc::group_and<1, 16 * LOAD_WARPS>(tc::mbar_wait(opempty, (n & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY));
            if (!ok) break;
          }
#pragma unroll
          for (int i = 0; i < U; ++i) {
            uint32_t hx = __shfl_up_sync(0xffffffffu, x[i].w, 8), hv = __shfl_up_sync(0xffffffffu, v[i].w, 8);
            if (lane < 8) { hx = px[i]; hv = pv[i]; }
            const uint32_t wx[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, wv[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            f32x2 pa = f2_pack(bf_lo(hx), bf_lo(hv)), pb = f2_pack(bf_hi(hx), bf_hi(hv));
            uint32_t h[4];
            float m = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const f32x2 e0 = f2_pack(bf_lo(wx[j]), bf_lo(wv[j])), e1 = f2_pack(bf_hi(wx[j]), bf_hi(wv[j]));
              const f32x2 y0 = f2_fma(w2, e0, f2_fma(w1, pb, f2_fma(w0, pa, wb)));
              const f32x2 y1 = f2_fma(w2, e1, f2_fma(w1, e0, f2_fma(w0, pb, wb)));
              pa = e0; pb = e1;
              float cx0, cv0, cx1, cv1;
              f2_unpack(y0, cx0, cv0);
              f2_unpack(y1, cx1, cv1);
              h[j] = bf2_mul(pack_bf2(cv0, cv1), pack_bf2(cx0, cx1));
            }
            mask_tail(h, 8 * okc, lim[i]);
            const int k = 8 * (k0 + i) + orow;
            if (k < cols) sts128(op + (k0 + i) * 128, h[0], h[1], h[2], h[3]);          // as bf16 until the scale is known
#pragma unroll
            for (int j = 0; j < 4; ++j) m = fmaxf(m, fmaxf(fabsf(bf_lo(h[j])), fabsf(bf_hi(h[j]))));
            maximum(k, m);
          }
        }
        if (!ok) break;
        maxima_done();
#pragma unroll 4
        for (int it = 0; it < iters; ++it) {
          const float sc = row_scale(__int_as_float(mx[rowjb[8 * it + orow] & 0xffffu]));
          const uint4 q = lds128(op + it * 128);
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
          uint32_t h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = pack_h2(bf_lo(w[j]) * sc, bf_hi(w[j]) * sc);
          sts128(op + it * 128, h[0], h[1], h[2], h[3]);
        }
      } else {
        // ---- the residual input as hi and lo; in their places as float32 until the scale is known ----
#pragma unroll 1
        for (int k0 = 0; k0 < iters; k0 += U) {
          float v[U][8];
#pragma unroll
          for (int i = 0; i < U; ++i) {
            long long off = 0;
            const int lim = where(8 * (k0 + i) + orow, P.usb, P.usc, off);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[i][e] = 0.f;
            if (8 * okc < lim) {
              if (P.u_bf16) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(P.u) + off + 8 * okc));
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) { v[i][2 * e] = bf_lo(w[e]); v[i][2 * e + 1] = bf_hi(w[e]); }
              } else {
                const float4* q = reinterpret_cast<const float4*>(static_cast<const float*>(P.u) + off + 8 * okc);
                const float4 q0 = __ldg(q), q1 = __ldg(q + 1);
                v[i][0] = q0.x; v[i][1] = q0.y; v[i][2] = q0.z; v[i][3] = q0.w; v[i][4] = q1.x; v[i][5] = q1.y; v[i][6] = q1.z; v[i][7] = q1.w;
              }
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (8 * okc + e >= lim) v[i][e] = 0.f;
            }
          }
          if (k0 == 0) {
            ok = tc::group_and<3, 16 * LOAD_WARPS>(tc::mbar_wait(opempty + 1, (n & 1) ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY));
            if (!ok) break;
          }
#pragma unroll
          for (int i = 0; i < U; ++i) {
            const int k = 8 * (k0 + i) + orow;
            float m = 0.f;
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              m = fmaxf(m, fabsf(v[i][e]));
              w[e] = __float_as_uint(v[i][e]);
            }
            if (k < cols) {
              sts128(op + (k0 + i) * 128, w[0], w[1], w[2], w[3]);
              sts128(op + (k0 + i) * 128 + REG, w[4], w[5], w[6], w[7]);
            }
            maximum(k, m);
          }
        }
        if (!ok) break;
        maxima_done();
#pragma unroll 4
        for (int it = 0; it < iters; ++it) {
          const float sc = row_scale(__int_as_float(mx[rowjb[8 * it + orow] & 0xffffu]));
          const uint4 q0 = lds128(op + it * 128), q1 = lds128(op + it * 128 + REG);
          const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) split_pair(__uint_as_float(w[2 * j]) * sc, __uint_as_float(w[2 * j + 1]) * sc, hi[j], lo[j]);
          sts128(op + it * 128, hi[0], hi[1], hi[2], hi[3]);
          sts128(op + it * 128 + REG, lo[0], lo[1], lo[2], lo[3]);
        }
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive(opfull + f);
        tc::mbar_arrive(sfull + f * SLOTS + slot);
      }
    }
  } else {
    // ---- outputs: a lane is a step, a column (block, sequence); a warp has every other eight of them, at most BATCHES times.  The
    // gate's rows are in registers before the first filter's accumulators are complete, and the gated results stay there until
    // the residual filter's are ----
    const int quarter = warp & 3, half = (warp - EPI0) >> 2;
    const uint32_t tl = tm + ((uint32_t)(32 * quarter) << 16);
    const int nb8 = cols >> 3, t0 = 32 * quarter, tq = t0 + lane;
    uint32_t n = 0;
    bool ok = true;
    for (int unit = u0; unit < u1 && ok; ++unit, ++n) {
      const int c = unit / P.ntile, b0 = (unit - c * P.ntile) * Bt;
      const int slot = n & (SLOTS - 1);
      const Taps T = load_taps(P.sw, P.sb, P.D + c);
      const __nv_bfloat16* x2 = P.xin + (P.D + c) * P.xsc + b0 * P.xsb + tq;
      __nv_bfloat16* oc = P.out + c * P.osc + b0 * P.osb + tq * P.ost;
      // row of column i of batch k; whether this lane's step of it exists
      auto row_of = [&](int k, int i) { return 8 * (half + 2 * k) + i; };
      auto live = [&](uint32_t jb) { return 128 * (int)(jb >> 16) + tq < L && b0 + (int)(jb & 0xffffu) < P.B; };
      uint32_t xp[4 * BATCHES], edge[BATCHES / 4];
#pragma unroll
      for (int e = 0; e < BATCHES / 4; ++e) {        // lane i: the two steps before the quarter's first in column 32 e + i
        const int r = row_of(4 * e + (lane >> 3), lane & 7);
        edge[e] = 0u;
        if (r < cols) {
          const uint32_t jb = rowjb[r];
          const int t = 128 * (int)(jb >> 16) + t0;
          if (t > 0 && t < L && b0 + (int)(jb & 0xffffu) < P.B)
            edge[e] = __ldg(reinterpret_cast<const uint32_t*>(x2 - lane + (jb & 0xffffu) * P.xsb + 128 * (int)(jb >> 16) - 2));
        }
      }
#pragma unroll
      for (int k = 0; k < BATCHES; ++k) {
        if (half + 2 * k >= nb8) break;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          uint32_t h[2] = {0u, 0u};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t jb = rowjb[row_of(k, i + e)];
            if (live(jb)) h[e] = __ldg(reinterpret_cast<const unsigned short*>(x2 + (jb & 0xffffu) * P.xsb + 128 * (int)(jb >> 16)));
          }
          xp[4 * k + i / 2] = h[0] | h[1] << 16;
        }
      }
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        if (f >= P.nf) break;
        ok = tc::mbar_wait(sfull + f * SLOTS + slot, (n / SLOTS) & 1, abort_flag, tc::ST_TIMEOUT_EPI) &&
             tc::mbar_wait(tfull + f, n & 1, abort_flag, tc::ST_TIMEOUT_EPI);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc::tc_fence_after();
        const float ti = tinv[f * SLOTS + slot];
        const float* xi = xinv + (f * SLOTS + slot) * 128;
        const bool store = f + 1 == P.nf;
#pragma unroll
        for (int k = 0; k < BATCHES; ++k) {
          if (half + 2 * k >= nb8) break;
          uint32_t z[8], zs[8];
          tmem_ld8(tl + f * REGION + row_of(k, 0), z);
          tmem_ld8(tl + f * REGION + SMALL + row_of(k, 0), zs);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            uint32_t& q = xp[4 * k + i / 2];
            const uint32_t jb[2] = {rowjb[row_of(k, i)], rowjb[row_of(k, i + 1)]};
            float o[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float y = (__uint_as_float(z[i + e]) + __uint_as_float(zs[i + e])) * xi[jb[e] & 0xffffu] * ti;
              const float cur = e ? bf_hi(q) : bf_lo(q);
              if (f == 0) {
                // (conv + bias term) as bf16, times the gate as bf16
                float m1 = __shfl_up_sync(0xffffffffu, cur, 1), m2 = __shfl_up_sync(0xffffffffu, cur, 2);
                const uint32_t before = __shfl_sync(0xffffffffu, edge[k >> 2], 8 * (k & 3) + i + e);
                if (lane == 0) m1 = bf_hi(before);
                if (lane < 2) m2 = lane ? bf_hi(before) : bf_lo(before);
                o[e] = bf16r(y) * bf16r(fmaf(T.w2, cur, fmaf(T.w1, m1, fmaf(T.w0, m2, T.b))));
              } else {
                // the residual conv joins in float32, or as bf16 where the layer input was
                o[e] = cur + (P.yu_bf16 ? bf16r(y) : y);
              }
            }
            q = pack_bf2(o[0], o[1]);
            if (store) {
#pragma unroll
              for (int e = 0; e < 2; ++e)
                if (live(jb[e]))
                  reinterpret_cast<unsigned short*>(oc)[(jb[e] & 0xffffu) * P.osb + 128 * (int)(jb[e] >> 16) * P.ost] = (unsigned short)(e ? q >> 16 : q);
            }
          }
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(tempty + f);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tm, 512);
  }
}

// Blocks and sequences per tile: columns in multiples of eight.
struct Shape { int nb, bt, cols; };
__host__ inline Shape shape_of(int L, int B) {
  Shape s;
  s.nb = (L + 127) / 128;
  const int cap = MAXCOLS / s.nb / 8 * 8, want = (B + 7) / 8 * 8;
  s.bt = want < cap ? want : cap;
  s.cols = s.nb * s.bt;
  return s;
}

static int launch(const m2_longconv_args* a, const float* const spec[2], cudaStream_t st) {
  Params P;
  const Shape sh = shape_of(a->seq_len, a->batch);
  P.B = a->batch; P.L = a->seq_len; P.D = a->d_model; P.nf = a->n_filters;
  P.NB = sh.nb; P.Bt = sh.bt; P.cols = sh.cols;
  P.ntile = (P.B + P.Bt - 1) / P.Bt;
  M2_REQUIRE((long long)P.ntile * P.D < (1LL << 30), M2_ERR_UNSUPPORTED, "m2_longconv_fwd: too many units");
  P.units = P.ntile * P.D;
  P.ksteps = P.NB == 1 ? (P.L + 15) / 16 : 8;
  P.u_bf16 = P.nf == 2 && a->u_dtype == M2_BF16;
  P.yu_bf16 = P.u_bf16 || (P.nf == 2 && a->yu_bf16);
  P.xin = (const __nv_bfloat16*)a->xin; P.xsb = a->xin_sb; P.xsc = a->xin_sc;
  P.u = a->u; P.usb = a->u_sb; P.usc = a->u_sc;
  P.out = (__nv_bfloat16*)a->out; P.osb = a->out_sb; P.ost = a->out_st; P.osc = a->out_sc;
  P.sw = a->short_w; P.sb = a->short_b;
  for (int f = 0; f < 2; ++f) { P.spec[f] = spec[f]; P.bias[f] = a->bias[f]; }
  const int smem = (int)layout_of(P.cols, P.NB).total;
  auto kern = longconv_bts_kernel;
  M2_SMEM_ONCE(kern, 227 * 1024);
  M2_REQUIRE(smem <= 227 * 1024, M2_ERR_UNSUPPORTED, "m2_longconv_fwd: block-Toeplitz tile of %d bytes", smem);
  const int sms = m2_sm_count();
  return m2_launch("longconv_bts_kernel", (long long)P.B * P.L * P.D, kern, P.units < sms ? P.units : sms, THREADS, smem, st, P);
}

}  // namespace bts

// Family 0 on time-contiguous bf16 rows that may be read up to a multiple of eight steps.
bool longconv_bts_f32_supported(const m2_longconv_args* a) {
  return a->rows_padded && a->act_dtype == M2_BF16 && a->bf16_rounding && !a->plain && a->seq_len <= bts::MAX_L && a->xin_st == 1 &&
         m2_aligned(a->xin, 16) && a->xin_sb % 8 == 0 && a->xin_sc % 8 == 0 &&
         (a->n_filters == 1 || (a->u_st == 1 && m2_aligned(a->u, 16) && a->u_sb % 8 == 0 && a->u_sc % 8 == 0));
}

// Which of the two float32 convolutions finishes first.  Launched alone with the L2 flushed (768 channels, two filters) this kernel
// takes 8 us and, for each unit of an SM, 1.2 us + 0.0228 an MMA + 0.125 a column, at least 4.8 (37 x 1 37 us, 131 x 2 43, 300 x 4 60,
// 300 x 30 113, 1000 x 4 145, 1000 x 16 196, 1531 x 6 211, 2045 x 8 310, 2047 x 2 287); the transform of longconv_f32.cu 4 us and,
// for each CTA of an SM, 8 us + 0.035 a point, 105 where one CTA fills it (19, 31, 86, 316, 132, 463, 391, 640 and 225 us).  In the
// stream of a forward the transform gains more from operands in the L2 (12 layers at 37 x 44 1212 us with it, 1326 with this kernel), so the
// line lies at 0.8 of its time and beyond one block.
bool longconv_bts_f32_preferred(int batch, int seq_len, int d_model) {
  if (seq_len <= 128 || seq_len > bts::MAX_L) return false;
  const bts::Shape s = bts::shape_of(seq_len, batch);
  const int sms = m2_sm_count();
  const long long units = (long long)((batch + s.bt - 1) / s.bt) * d_model, ctas = longconv_f32_ctas(batch, seq_len, d_model);
  const double unit = 1.2 + 0.0228 * 5 * 8 * (2 * s.nb - 1) + 0.125 * s.cols;
  const int points = m2_filter_row_len(seq_len) / 2;
  const double cta = points > 1024 ? 105.0 : 8.0 + 0.035 * points;
  return 8.0 + (units + sms - 1) / sms * (unit > 4.8 ? unit : 4.8) < 0.8 * (4.0 + (ctas + sms - 1) / sms * cta);
}

// its taps lie behind the transform's table, on a 16-byte boundary
size_t taps_f32_offset(int D, int L) {
  const size_t M = (size_t)m2_filter_row_len(L) / 2;
  return (M + 4 * M * D + 3) / 4 * 4;
}
size_t taps_f32_floats(int D, int L) { return L > bts::MAX_L ? 0 : (size_t)D * (bts::tap_count((L + 127) / 128) + 1); }
int taps_f32_launch(int D, int L, const float* k, float* taps, cudaStream_t st) {
  if (L > bts::MAX_L) return M2_OK;
  bts::taps_f32_kernel<<<D, 256, 0, st>>>(k, taps, D, L, m2_filter_row_len(L), (L + 127) / 128);
  M2_LAUNCH_CHECK("taps_f32_kernel");
  return M2_OK;
}
int longconv_bts_f32_launch(const m2_longconv_args* a, cudaStream_t st) {
  const size_t skip = taps_f32_offset(a->d_model, a->seq_len);
  const float* const spec[2] = {a->spec[0] + skip, a->spec[1] ? a->spec[1] + skip : nullptr};
  return bts::launch(a, spec, st);
}

}  // namespace m2
