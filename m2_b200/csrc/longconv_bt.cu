// Fused gated long convolution as block-Toeplitz GEMMs on tcgen05 tensor cores, sequence lengths up to 1024
// (any length, any batch), bf16 activations, time-contiguous tensors (kernel family 4).
//
// A sequence is cut into NB = ceil(L / 128) blocks of 128 steps.  The bidirectional convolution of one channel is
// then y[jt] = sum_js T_{jt - js} a[js] with 128 x 128 Toeplitz blocks, and all (block, sequence) pairs of a tile of
// Bt sequences share every T_delta:
//   D[128 steps n, columns (jt, b)] += T_delta[128 x 128] . A[128 steps k, columns (js = jt - delta, b)].
// The Toeplitz block is the MMA's A operand (a TMEM lane is a step inside the block), the data its B operand, N =
// (NB - |delta|) Bt columns: only the block pairs that exist are multiplied, NB^2 Bt columns of eight K = 16 steps per
// filter.  Data rows are ordered (block, sequence), 16 bytes per row and K chunk, so moving by delta blocks is a
// start address; likewise the eight K steps of T_delta, and T_delta and T_{delta+1}, are one Toeplitz strip
//   S[m, j] = h(j - m + 112 - 128 delta),  h(d) = tap multiplying a[t + d],
// at different start rows.  The strip is built in shared memory from the channel's 2 L fp16 taps, two deltas (368
// rows) at a time, while the tensor core works on the two before.
//
// Bound: few rows by one unit's chain of phases (load, 2 NB strip windows with a hand-over each, gate, write); many short ones
// (NB <= 4) by the memory traffic of 10 bytes per step and channel.  Beyond that it is neither that nor the MMAs: 16 x 1024 at
// 768 channels takes 123 us (ncu, caches cold), of which the 240 MMAs of a unit, 40 to 65 clocks each, are some 35 and the
// traffic 20; two CTAs share an SM and overlap one's phases with the other's, no more.  More than 128 columns per CTA would share
// a unit's strips among more data but leave room for one CTA.  The FFT family at the same shapes moves 18.9 kclk of
// shared-memory traffic per sequence whatever its length up to 2048: longconv_bt_preferred draws the line.
//
// The range and rounding of the operands are those of family 3: v * x1 is a bf16 value converted to fp16 (exactly between
// 2^-14 and 65504, saturating beyond; the direct kernel of longconv_direct.cu sums it as it is), the residual input an fp16
// copy, taps fp16 after a per-channel power-of-two scaling with the bias folded into h(0),
// float32 accumulation in TMEM.  Every mbarrier wait is bounded.
//
// Computation replaced: bert/src/mm/monarch_mixer_sequence_mixer.py:109-149 and
// bert/src/mm/hyena_utils.py:16-42, :219-248 of the reference.
#include "tc_common.cuh"

namespace m2 {
namespace bt {

constexpr int WORKERS = 256;                    // eight warps load, build strips and write; a ninth issues the MMAs
constexpr int THREADS = WORKERS + 32;
constexpr int MAXCOLS = 128;
constexpr int MAX_L = 1024;                     // beyond it the FFT family is faster at every batch size
constexpr int WROWS = 368;                      // strip rows of two deltas: 2 * 128 + 112
constexpr int WIN_BYTES = WROWS * 32;
constexpr int SMEM_MAX = 113 * 1024;            // per CTA with two on an SM
constexpr long long REACH = 1LL << 33;          // elements from the first to the last of a tensor: offsets are kept as int, in units of 8
constexpr int YROW = 272;                       // bytes of a 128-step row in the x2 / output buffers (16 of padding)

__host__ __device__ constexpr int tap_count(int nb) { return 256 * nb + 64; }   // fp16 taps of a channel, d = -128 nb ..

// Blocks and sequences per tile.  N = (NB - |delta|) Bt is rounded up to a multiple of 16 with eight zero rows; NB Bt
// itself is a multiple of 16.
struct Shape { int nb, bt, cols; };
__host__ inline Shape shape_of(int L, int B) {
  Shape s;
  s.nb = (L + 127) / 128;
  const int unit = (s.nb & 1) ? 16 : 8;
  const int most = MAXCOLS / s.nb / unit * unit, want = (B + unit - 1) / unit * unit;
  s.bt = want < most ? want : most;
  s.cols = s.nb * s.bt;
  return s;
}

// ---------------------------------------------------------------------------------------
// Filter table (kind 4): per channel tap_count(NB) fp16 taps h(d) 2^e at index d + 128 NB (zero for |d| >= L), then
// d_model floats 2^-e.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
spectrum_kind4_kernel(const float* __restrict__ kfilt, const float* __restrict__ bias, float* __restrict__ spec,
                      int D, int L, int R, int nb) {
  __shared__ float red[8];
  const int c = blockIdx.x, tid = threadIdx.x, n = tap_count(nb);
  const float* row = kfilt + (size_t)c * R;
  auto tap = [&](int i) {
    const int d = i - 128 * nb;
    float v = 0.f;
    if (d > -L && d < L) v = row[d > 0 ? R - d : -d];
    if (d == 0 && bias) v += bias[c];
    return v;
  };
  float m = 0.f;
  for (int i = tid; i < n; i += blockDim.x) {
    const float v = fabsf(tap(i));
    if (v < 3.0e38f) m = fmaxf(m, v);                          // non-finite taps do not pick the scale
  }
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int i = 1; i < 8; ++i) m = fmaxf(m, red[i]);
  int e = 0;
  if (m > 0.f) {
    int ex;
    frexpf(m, &ex);
    e = 14 - ex;                                               // m * 2^e in [2^13, 2^14)
    e = e < -60 ? -60 : (e > 60 ? 60 : e);
  }
  const float scale = ldexpf(1.0f, e);
  __half* T = reinterpret_cast<__half*>(spec) + (size_t)c * n;
  for (int i = tid; i < n; i += blockDim.x) T[i] = __float2half_rn(tap(i) * scale);
  if (tid == 0) spec[(size_t)D * (n / 2) + c] = ldexpf(1.0f, -e);
}

// 16 K chunks of (cols + 16) rows of 16 bytes; the same place later holds cols rows of YROW bytes
__host__ __device__ constexpr int operand_bytes(int cols) { return (cols + 16) * 256 > cols * YROW ? (cols + 16) * 256 : cols * YROW; }
// one strip window: 240 rows for a single block, else two deltas
__host__ __device__ constexpr int window_rows(int nb) { return nb == 1 ? 240 : WROWS; }

__host__ inline int smem_of(const Shape& s, int g, int nf) {
  return 2 * operand_bytes(g * s.cols) + 2 * g * window_rows(s.nb) * 32 + nf * g * tap_count(s.nb) * 2 + 48 * g + 16 * MAXCOLS + 64;
}
// channels per unit; one where an MMA takes eight rows beside its channel's data, which must be the zero rows around it
__host__ inline int group_of(const Shape& s, int B, int D, int nf) {
  if (s.bt % 16) return 1;
  const long long seqs = (long long)((B + s.bt - 1) / s.bt) * D;
  int g = 1;
  while (g < 4 && (g + 1) * s.cols <= MAXCOLS && smem_of(s, g + 1, nf) <= SMEM_MAX && seqs > 2LL * g * m2_sm_count()) ++g;
  return g;
}

struct Params {
  int B, L, D, nf, NB, Bt, G, cols, ntile, units, tcols, tpad, ksteps;
  int u_f16, yu_bf16;
  const __nv_bfloat16* xin; long long xsb, xsc;
  const void* u; long long usb, usc;
  __nv_bfloat16* out; long long osb, osc;
  const float* sw; const float* sb;
  const float* spec[2];
};

// 16 lanes x 8 columns of 32-bit as 8 x 8 fragments: registers 0, 1 are row lane / 4, columns 2 (lane % 4) and the next;
// registers 2, 3 the same columns of row lane / 4 + 8
__device__ __forceinline__ void tmem_ld_16x256(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// bf16x2 -> fp16x2, exact inside fp16's range and its largest value beyond, as family 3 has it (a NaN stays one)
__device__ __forceinline__ uint32_t bf2_to_h2_sat(uint32_t v) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(lcl::bf_hi(v)), "f"(lcl::bf_lo(v)));
  return r;
}
// barrier of the worker warps, true where `v` is for all of them
__device__ __forceinline__ bool workers_and(bool v) { return tc::group_and<1, WORKERS>(v); }
__device__ __forceinline__ void workers_sync() { asm volatile("barrier.cta.sync 1, %0;" ::"n"(WORKERS) : "memory"); }

// A unit is G channels x Bt sequences (G > 1 only where one channel's columns leave most of the CTA idle and there are
// more channels than resident CTAs: the loads, barriers and epilogue of G channels then share one latency).  Row r of the
// operands = column r of an accumulator = (channel g, block j, sequence b), r = (g NB + j) Bt + b.
__global__ void __launch_bounds__(THREADS, 2)
longconv_bt_kernel(const Params P) {
  using namespace lcl;                               // packed-arithmetic and shared-memory helpers of the long-row family
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, warp = tc::uniform_warp_id(), lane = tid & 31;
  const int cols = P.cols, Bt = P.Bt, NB = P.NB, L = P.L, G = P.G, gcols = NB * Bt;   // cols = G gcols
  const uint32_t LBO = (uint32_t)(cols + 16) * 16;   // a multiple of 128: no core matrix straddles two 128-byte lines
  const uint32_t REG = operand_bytes(cols), TB = (uint32_t)P.tpad * 2;
  const uint32_t wrows = window_rows(NB), WB = wrows * 32;
  const uint32_t a1 = tc::smem_u32(smem), a2 = a1 + REG, win = a2 + REG, taps = win + 2 * G * WB;
  unsigned char* tail = smem + 2 * REG + 2 * G * WB + P.nf * G * TB;
  float4* prm = reinterpret_cast<float4*>(tail);     // [g][x1, x2, v]: short-conv taps w0 w1 w2 b, rounded to bf16
  int4* rows = reinterpret_cast<int4*>(prm + 3 * G); // row -> offsets of its first step in xin, u, out in units of 8
                                                     // elements (rows start on 16-byte boundaries), steps that exist
  uint64_t* bars = reinterpret_cast<uint64_t*>(rows + MAXCOLS);
  uint64_t* wfull = bars + 2;                        // strip window written (by every worker warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (tid == 0) {
    tc::mbar_init(bars, 1);
    tc::mbar_init(bars + 1, 1);
    tc::mbar_init(wfull, WORKERS / 32);
    tc::mbar_init(wfull + 1, WORKERS / 32);
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tmem_slot, P.tcols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tm = *tmem_slot;
  pdl_wait();

  bool ok = true;
  uint32_t commits = 0;                              // groups of MMAs committed so far; group i signals bars[i & 1]
  auto wait_group = [&](uint32_t i) {
    if (ok) ok = tc::mbar_wait(bars + (i & 1), (i >> 1) & 1, abort_flag, tc::ST_TIMEOUT_MMA);
  };
  const int wpos = (NB + 1) >> 1, nwin = wpos + (NB >> 1);      // windows of deltas 0.., then of deltas -1 downwards
  const int iters = cols >> 4;                       // operand chunks per thread
  int have_c = -1;
  const int u0 = (int)((long long)blockIdx.x * P.units / gridDim.x), u1 = (int)((long long)(blockIdx.x + 1) * P.units / gridDim.x);
  // deltas of window s
  auto window = [&](int s, int& dlo, int& dhi) {
    dlo = s < wpos ? 2 * s : max(1 - NB, -2 * (s - wpos + 1));
    dhi = s < wpos ? min(NB - 1, 2 * s + 1) : -2 * (s - wpos) - 1;
  };
  if (warp == WORKERS / 32) {
    // ---- MMA issuer ----
    if (tc::elect_one()) {
      for (int unit = u0; unit < u1 && ok; ++unit) {
        const int gn = min(G, P.D - unit / P.ntile * G);
        for (int fs = 0; fs < P.nf * nwin && ok; ++fs) {
          const int f = fs >= nwin, s = fs - f * nwin;
          int dlo, dhi;
          window(s, dlo, dhi);
          const uint32_t data = f ? a2 : a1, wb = win + (commits & 1) * G * WB;
          ok = tc::mbar_wait(wfull + (commits & 1), (commits >> 1) & 1, abort_flag, tc::ST_TIMEOUT_TMA);
          if (!ok) break;
          tc::tc_fence_after();
          for (int g = 0; g < gn; ++g)
            for (int d = dlo; d <= dhi; ++d) {
              const int n = (NB - abs(d)) * Bt, e = (16 - (n & 15)) & 15;    // e = 0 or 8 zero rows
              const uint32_t idesc = tc::make_idesc(128, n + e, 0);
              const uint32_t dcol = tm + f * cols + g * gcols + (d > 0 ? d * Bt - e : 0);
              const uint32_t brow = data + 16 * (8 + g * gcols + (d < 0 ? -d * Bt : -e));
              const uint32_t arow = wb + g * WB + 16 * (112 + 128 * (d - dlo));
              // descriptors differ in the address field only: a K step moves A by -16 rows, B by two planes
              const uint32_t alo = (arow >> 4) | wrows << 16, blo = (brow >> 4) | (LBO >> 4) << 16;
              constexpr uint32_t hi = (128u >> 4) | 1u << 14;                // 128 bytes between row groups, version
              const uint32_t step = LBO >> 3;
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)
                if (kk < P.ksteps)
                  tc::mma_ss(dcol, tc::desc_words(alo - 16 * kk, hi), tc::desc_words(blo + step * kk, hi), idesc,
                             (d != 0 || kk != 0) ? 1u : 0u);
            }
          tc::mma_commit(bars + (commits & 1));
          ++commits;
        }
      }
    }
    __syncwarp();
  } else
  for (int unit = u0; unit < u1; ++unit) {
    const int cg = unit / P.ntile, c0 = cg * G, b0 = (unit - cg * P.ntile) * Bt;
    const int gn = min(G, P.D - c0);                 // channels of this unit that exist
    // ---- taps of the filters and of the short conv (once per channel), zero rows around the data ----
    if (c0 != have_c) {
      have_c = c0;
      for (int f = 0; f < P.nf; ++f) {
        const unsigned char* src = reinterpret_cast<const unsigned char*>(P.spec[f]) + (size_t)c0 * TB;
        for (uint32_t i = tid; i < gn * (TB >> 4); i += WORKERS) cp_async16(taps + f * G * TB + 16 * i, src + 16 * i);
      }
      if (tid < 3 * gn) {
        const Taps T = load_taps(P.sw, P.sb, (tid % 3) * P.D + c0 + tid / 3);
        prm[tid] = make_float4(T.w0, T.w1, T.w2, T.b);
      }
    }
    {
      const uint32_t plane = tid >> 4, r = tid & 15;             // 16 planes x 16 zero rows
      const uint32_t o = plane * LBO + (r < 8 ? r : cols + r) * 16;
      sts128(a1 + o, 0u, 0u, 0u, 0u);
      sts128(a2 + o, 0u, 0u, 0u, 0u);
    }
    if (tid < cols) {
      const int g = tid / gcols, j = (tid - g * gcols) / Bt, b = b0 + tid - (g * NB + j) * Bt;
      const long long c = c0 + g, t = 128 * j;
      int4 q = make_int4(0, 0, 0, 0);
      if (b < P.B && g < gn)
        q = make_int4((int)((c * P.xsc + b * P.xsb + t) >> 3), (int)((c * P.usc + b * P.usb + t) >> 3),
                      (int)((c * P.osc + b * P.osb + t) >> 3), min(128, L - (int)t));
      rows[tid] = q;
    }
    auto taps2 = [&](int g, int k) {
      const float4 q = prm[3 * g + k];
      Taps2 T;
      T.w0 = f2_splat(q.x); T.w1 = f2_splat(q.y); T.w2 = f2_splat(q.z); T.b = f2_splat(q.w);
      return T;
    };
    workers_sync();                                  // rows, prm
    // Operand chunks: a warp covers 64 bytes of eight rows, a quarter warp writes one core matrix.
    const int okc = 4 * (warp & 3) + (lane >> 3), orow = 8 * (warp >> 2) + (lane & 7);
    // ---- the residual input: copied into its operand as it is ----
    if (P.nf == 2) {
      const uint4* ub = reinterpret_cast<const uint4*>(P.u) + okc;
      const uint32_t d0 = a2 + okc * LBO + (8 + orow) * 16;
#pragma unroll 4
      for (int it = 0; it < iters; ++it) {
        const int4 q = rows[16 * it + orow];
        const uint32_t dst = d0 + it * 256;
        if (P.u_f16 && 8 * okc + 8 <= q.w) {
          cp_async16(dst, ub + q.y);
        } else {
          uint32_t h[4] = {0u, 0u, 0u, 0u};
          if (8 * okc < q.w) {
            const uint4 v = __ldg(ub + q.y);
            h[0] = v.x; h[1] = v.y; h[2] = v.z; h[3] = v.w;
            if (!P.u_f16) {
#pragma unroll
              for (int j = 0; j < 4; ++j) h[j] = bf2_to_h2_sat(h[j]);
            }
            mask_tail(h, 8 * okc, q.w);
          }
          sts128(dst, h[0], h[1], h[2], h[3]);
        }
      }
    }
    cp_async_commit();
    // ---- x1, v: short conv, product, fp16 ----
    constexpr int U = 4;
    const long long vdist = 2 * P.D * P.xsc;
    for (int g = 0; g < G; ++g) {
      // both short convs advance in one f32x2 chain: packed pairs are (x1, v)
      const float4 qx = prm[3 * g], qv = prm[3 * g + 2];
      const f32x2 w0 = f2_pack(qx.x, qv.x), w1 = f2_pack(qx.y, qv.y), w2 = f2_pack(qx.z, qv.z), wb = f2_pack(qx.w, qv.w);
      for (int k0 = 0; k0 < gcols; k0 += 16 * U) {
        uint4 x[U], v[U];
        uint32_t px[U], pv[U];
        int lim[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          x[i] = v[i] = make_uint4(0u, 0u, 0u, 0u);
          px[i] = pv[i] = 0u;
          lim[i] = 0;
          const int k = k0 + 16 * i + orow;                      // row inside the channel's group
          if (k0 + 16 * i < gcols) {
            const int4 q = rows[g * gcols + k];
            lim[i] = q.w;
            if (8 * okc < q.w) {
              const __nv_bfloat16* xr = P.xin + 8 * ((long long)q.x + okc);
              x[i] = __ldg(reinterpret_cast<const uint4*>(xr));
              v[i] = __ldg(reinterpret_cast<const uint4*>(xr + vdist));
              if (lane < 8 && (okc > 0 || k >= Bt)) {            // the two steps before the warp's first chunk of a row
                px[i] = __ldg(reinterpret_cast<const uint32_t*>(xr - 2));
                pv[i] = __ldg(reinterpret_cast<const uint32_t*>(xr + vdist - 2));
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
          if (k0 + 16 * i < gcols) {
            uint32_t hx = __shfl_up_sync(0xffffffffu, x[i].w, 8), hv = __shfl_up_sync(0xffffffffu, v[i].w, 8);
            if (lane < 8) { hx = px[i]; hv = pv[i]; }
            const uint32_t wx[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, wv[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            f32x2 pa = f2_pack(bf_lo(hx), bf_lo(hv)), pb = f2_pack(bf_hi(hx), bf_hi(hv));
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const f32x2 e0 = f2_pack(bf_lo(wx[j]), bf_lo(wv[j])), e1 = f2_pack(bf_hi(wx[j]), bf_hi(wv[j]));
              const f32x2 y0 = f2_fma(w2, e0, f2_fma(w1, pb, f2_fma(w0, pa, wb)));
              const f32x2 y1 = f2_fma(w2, e1, f2_fma(w1, e0, f2_fma(w0, pb, wb)));
              pa = e0; pb = e1;
              float cx0, cv0, cx1, cv1;
              f2_unpack(y0, cx0, cv0);
              f2_unpack(y1, cx1, cv1);
              h[j] = bf2_to_h2_sat(bf2_mul(pack_bf2(cv0, cv1), pack_bf2(cx0, cx1)));
            }
            mask_tail(h, 8 * okc, lim[i]);
            sts128(a1 + okc * LBO + (8 + g * gcols + k0 + 16 * i + orow) * 16, h[0], h[1], h[2], h[3]);
          }
        }
      }
    }
    cp_async_wait<0>();
    workers_sync();                                  // taps are read by every thread below

    // the gate: short conv of x2 as bf16 rows [row][128 steps], into the first operand region once its MMAs are done
    // (half a warp covers the 256 bytes of one row)
    const int gkc = tid & 15, grow = tid >> 4;
    auto make_gate = [&]() {
      for (int g = 0; g < G; ++g) {
        const Taps2 T = taps2(g, 1);
        for (int k0 = 0; k0 < gcols; k0 += 16 * U) {
          uint4 x[U];
          uint32_t px[U];
#pragma unroll
          for (int i = 0; i < U; ++i) {
            x[i] = make_uint4(0u, 0u, 0u, 0u);
            px[i] = 0u;
            const int k = k0 + 16 * i + grow;
            if (k0 + 16 * i < gcols) {
              const int4 q = rows[g * gcols + k];
              if (8 * gkc < q.w) {
                const __nv_bfloat16* xr = P.xin + 8 * ((long long)q.x + gkc) + (vdist >> 1);
                x[i] = __ldg(reinterpret_cast<const uint4*>(xr));
                if (gkc == 0 && k >= Bt) px[i] = __ldg(reinterpret_cast<const uint32_t*>(xr - 2));
              }
            }
          }
#pragma unroll
          for (int i = 0; i < U; ++i)
            if (k0 + 16 * i < gcols) {
              uint32_t hx = __shfl_up_sync(0xffffffffu, x[i].w, 1);
              if (gkc == 0) hx = px[i];
              const uint32_t wx[5] = {hx, x[i].x, x[i].y, x[i].z, x[i].w};
              uint32_t cx[4];
              conv_packed<8>(T, wx, cx);
              sts128(a1 + (g * gcols + k0 + 16 * i + grow) * YROW + gkc * 16, cx[0], cx[1], cx[2], cx[3]);
            }
        }
      }
    };
    for (int f = 0; f < P.nf; ++f) {
      // the gate is made while the last filter's MMAs run, as soon as those of the first are known to be done
      if (f == 1 && nwin <= 2) wait_group(commits - 1);
      for (int s = 0; s < nwin; ++s) {
        int dlo, dhi;
        window(s, dlo, dhi);
        const uint32_t wn = 128 * (dhi - dlo + 1) + 112;
        const uint32_t wb = win + (commits & 1) * G * WB;
        if (commits >= 2) wait_group(commits - 2);   // the MMAs that read this window buffer are done
        // strip chunk (m, hf): taps h(8 hf + i - m + 112 - 128 dlo), i = 0 .. 7
        for (int g = 0; g < G; ++g) {
          const uint32_t tg = taps + (f * G + g) * TB, wg = wb + g * WB;
          const int pbase = 112 - 128 * dlo + 128 * NB;
#pragma unroll 3
          for (uint32_t q = tid; q < 2 * wn; q += WORKERS) {
            const uint32_t hf = q >= wn, m = q - hf * wn;
            const int p = pbase + 8 * (int)hf - (int)m;
            const uint32_t wa = tg + 4 * (p >> 1);
            uint32_t w[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) w[i] = lds32(wa + 4 * i);
            const uint32_t sel = (p & 1) ? 0x5432u : 0x3210u;
            sts128(wg + hf * (wrows * 16) + m * 16, __byte_perm(w[0], w[1], sel), __byte_perm(w[1], w[2], sel),
                   __byte_perm(w[2], w[3], sel), __byte_perm(w[3], w[4], sel));
          }
        }
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(wfull + (commits & 1));
        ++commits;
        // step 2 of the second filter has waited for its step 0, and with it for all of the first filter's MMAs
        if (f == 1 && s == (nwin <= 2 ? 0 : 2) && ok) make_gate();
      }
    }
    wait_group(commits - 1);
    if (ok && P.nf == 1) make_gate();
    ok = workers_and(ok);
    if (!ok) break;
    tc::tc_fence_after();

    // ---- epilogue in 8 x 8 fragments: a 16x256b read of the accumulators gives a thread two neighbouring columns of
    // one step, the layout of ldmatrix / stmatrix, whose transposed forms read the gate's and write the output's rows
    // (a column each, 16 bytes = 8 steps) ----
    {
      const uint32_t tl = tm + ((uint32_t)(32 * (warp & 3)) << 16);
      const int half = cols >> 1, cb = (warp >> 2) * half;
      // matrix q = lane / 8 of an x4 access covers steps 32 (warp & 3) + 8 q .., its row lane % 8 is column + lane % 8
      const uint32_t frag = (cb + (lane & 7)) * YROW + 2 * (32 * (warp & 3) + 8 * (lane >> 3));
      const uint32_t gate = a1 + frag, dst = a2 + frag;
      f32x2 ig0 = 0, ig1 = 0;
      int hg = -1;
      for (int i0 = 0; i0 < half; i0 += 8) {
        const int g = min((cb + i0) / gcols, gn - 1);             // gcols is a multiple of 16: one channel per batch
        if (g != hg) {
          hg = g;
          ig0 = f2_splat(__ldg(P.spec[0] + (size_t)P.D * (P.tpad / 2) + c0 + g));
          if (P.nf == 2) ig1 = f2_splat(__ldg(P.spec[1] + (size_t)P.D * (P.tpad / 2) + c0 + g));
        }
        uint32_t z0[8], z1[8], w[4], o[4];
        tmem_ld_16x256(tl + cb + i0, z0);
        tmem_ld_16x256(tl + (16u << 16) + cb + i0, z0 + 4);
        if (P.nf == 2) {
          tmem_ld_16x256(tl + cols + cb + i0, z1);
          tmem_ld_16x256(tl + (16u << 16) + cols + cb + i0, z1 + 4);
        }
        ldmatrix_x4_trans(gate + i0 * YROW, w);
        tc::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // (conv + bias term) as bf16, times the gate as bf16; the residual conv joins in float32 (or bf16 first)
          float y0, y1;
          f2_unpack(f2_mul(f2_pack(__uint_as_float(z0[2 * i]), __uint_as_float(z0[2 * i + 1])), ig0), y0, y1);
          o[i] = bf2_mul(pack_bf2(y0, y1), w[i]);
          if (P.nf == 2) {
            const f32x2 z = f2_pack(__uint_as_float(z1[2 * i]), __uint_as_float(z1[2 * i + 1]));
            if (P.yu_bf16) {
              f2_unpack(f2_mul(z, ig1), y0, y1);
              o[i] = pack_bf2(bf_lo(o[i]) + bf16r(y0), bf_hi(o[i]) + bf16r(y1));
            } else {
              f2_unpack(f2_mul(z, ig1), y0, y1);
              o[i] = pack_bf2(bf_lo(o[i]) + y0, bf_hi(o[i]) + y1);
            }
          }
        }
        stmatrix_x4_trans(dst + i0 * YROW, o);
      }
    }
    tc::tc_fence_before();
    workers_sync();
    for (int it = 0; it < iters; ++it) {
      const int r = 16 * it + grow;
      const int4 q = rows[r];
      if (8 * gkc < q.w)
        store_chunk8(P.out + 8 * (long long)q.z, 8 * gkc, q.w, lds128(a2 + r * YROW + gkc * 16));
    }
    workers_sync();                                  // the buffers become operand regions again
  }
  cp_async_wait<0>();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tm, P.tcols);
  }
}

}  // namespace bt

int longconv_bt_supported(int seq_len, m2_dtype act_dtype) {
  return act_dtype == M2_BF16 && seq_len >= 1 && seq_len <= bt::MAX_L;
}

// Time of the block-Toeplitz kernel in us.  It runs in waves of two units per SM; launched alone with the L2 flushed (D = 768,
// L = 256 .. 1024, B = 1 .. 64) a wave takes 0.25 us per column and 2 us per block, and in the stream of a forward, its start
// overlapped and its operands in L2, 0.8 of that (D = 768, one sequence to eight: 12 us at 128 steps, 18 at 256, 40 at 384;
// D = 1536: 28, 34, 58).  The same launch at 8 x 128 is 20 us alone and 16.5 under ncu, which runs it alone with other clocks.
static double bt_us(int batch, int seq_len, int d_model, int nf) {
  const bt::Shape s = bt::shape_of(seq_len, batch);
  const int g = bt::group_of(s, batch, d_model, nf), sms = m2_sm_count();
  const long long units = (long long)((batch + s.bt - 1) / s.bt) * ((d_model + g - 1) / g);
  return 0.8 * (0.25 * g * s.cols + 2.0 * s.nb) * ((units + 2 * sms - 1) / (2 * sms));
}

// Whether this family beats the FFT family at 128 < L <= 1024, whose waves of 8 sequences per SM take 19 us whatever the
// length (0.8 of it in the stream of a forward).
bool longconv_bt_preferred(int batch, int seq_len, int d_model) {
  // the widest tensor, 3 d_model rows of batch * seq_len steps with their padding (3.7 M tokens at d_model 768)
  if ((3LL * d_model + 1) * ((long long)batch * ((seq_len + 7) / 8 * 8) + 16) >= bt::REACH) return false;
  const long long waves = ((long long)batch * d_model + 8 * m2_sm_count() - 1) / (8 * m2_sm_count());
  const double bt = bt_us(batch, seq_len, d_model, 2), direct = longconv_direct_us(batch, seq_len, d_model, 2);
  return 0.8 * 19.0 * waves > (bt < direct ? bt : direct);
}

size_t spectrum_kind4_floats(int D, int L) {
  return (size_t)D * (bt::tap_count(bt::shape_of(L, 1).nb) / 2) + (size_t)D;
}

int spectrum_kind4_launch(int D, int L, const float* k, const float* bias, float* spec, cudaStream_t st) {
  M2_REQUIRE(longconv_bt_supported(L, M2_BF16), M2_ERR_UNSUPPORTED, "m2_filter_spectrum: kind 4 covers seq_len <= %d", bt::MAX_L);
  bt::spectrum_kind4_kernel<<<D, 256, 0, st>>>(k, bias, spec, D, L, m2_filter_row_len(L), bt::shape_of(L, 1).nb);
  M2_LAUNCH_CHECK("spectrum_kind4_kernel");
  return M2_OK;
}

int longconv_bt_launch(const m2_longconv_args* a, cudaStream_t st) {
  using namespace bt;
  M2_REQUIRE(longconv_bt_supported(a->seq_len, a->act_dtype), M2_ERR_UNSUPPORTED,
             "m2_longconv_fwd: kind 4 needs bf16 activations and seq_len <= %d", MAX_L);
  M2_REQUIRE(a->xin_st == 1 && a->out_st == 1 && (a->n_filters == 1 || a->u_st == 1), M2_ERR_UNSUPPORTED,
             "m2_longconv_fwd: kind 4 needs time-contiguous tensors");
  M2_REQUIRE(a->n_filters == 1 || a->u_dtype == M2_F16 || a->u_dtype == M2_BF16, M2_ERR_UNSUPPORTED,
             "m2_longconv_fwd: kind 4 reads the residual input as fp16 (m2_time_major_f16) or bf16");
  M2_REQUIRE(!a->bias[0] && !a->bias[1], M2_ERR_ARG,
             "m2_longconv_fwd: kind 4 takes the bias folded into the spectrum (m2_filter_spectrum_bias); pass bias = NULL");
  M2_REQUIRE(m2_aligned(a->xin, 16) && a->xin_sb % 8 == 0 && a->xin_sc % 8 == 0 && m2_aligned(a->out, 16) &&
             a->out_sb % 8 == 0 && a->out_sc % 8 == 0, M2_ERR_ALIGN,
             "m2_longconv_fwd: kind 4 needs 16-byte aligned rows of xin and out");
  M2_REQUIRE(a->n_filters == 1 || (m2_aligned(a->u, 16) && a->u_sb % 8 == 0 && a->u_sc % 8 == 0),
             M2_ERR_ALIGN, "m2_longconv_fwd: kind 4 needs 16-byte aligned rows of u");
  const int u_f16 = a->n_filters == 2 && a->u_dtype == M2_F16, yu_bf16 = a->n_filters == 2 && (a->u_dtype == M2_BF16 || a->yu_bf16);
  const Shape sh = shape_of(a->seq_len, a->batch);
  if (longconv_direct_us(a->batch, a->seq_len, a->d_model, a->n_filters) < bt_us(a->batch, a->seq_len, a->d_model, a->n_filters))
    return longconv_direct_launch(a, tap_count(sh.nb), 128 * sh.nb, u_f16, yu_bf16, st);
  Params P;
  P.B = a->batch; P.L = a->seq_len; P.D = a->d_model; P.nf = a->n_filters;
  P.NB = sh.nb; P.Bt = sh.bt;
  P.ntile = (P.B + P.Bt - 1) / P.Bt;
  P.tpad = tap_count(P.NB);
  const int most = 2 * m2_sm_count();                          // resident CTAs: two per SM by registers, tensor and shared memory
  P.G = group_of(sh, P.B, P.D, P.nf);
  P.cols = P.G * sh.cols;
  M2_REQUIRE((long long)P.ntile * P.D < (1LL << 30), M2_ERR_UNSUPPORTED, "m2_longconv_fwd: too many units");
  const long long reach = 3LL * P.D * a->xin_sc + (long long)P.B * a->xin_sb, ureach = (long long)P.D * a->u_sc + (long long)P.B * a->u_sb,
                  oreach = (long long)P.D * a->out_sc + (long long)P.B * a->out_sb;
  M2_REQUIRE(reach < REACH && ureach < REACH && oreach < REACH, M2_ERR_UNSUPPORTED, "m2_longconv_fwd: tensors too large for kind 4");
  P.units = P.ntile * ((P.D + P.G - 1) / P.G);
  P.ksteps = P.NB == 1 ? (P.L + 15) / 16 : 8;
  P.tcols = 32;
  while (P.tcols < P.nf * P.cols) P.tcols *= 2;
  P.u_f16 = u_f16; P.yu_bf16 = yu_bf16;
  P.xin = (const __nv_bfloat16*)a->xin; P.xsb = a->xin_sb; P.xsc = a->xin_sc;
  P.u = a->u; P.usb = a->u_sb; P.usc = a->u_sc;
  P.out = (__nv_bfloat16*)a->out; P.osb = a->out_sb; P.osc = a->out_sc;
  P.sw = a->short_w; P.sb = a->short_b;
  P.spec[0] = a->spec[0]; P.spec[1] = a->spec[1];
  const int smem = smem_of(sh, P.G, P.nf);
  // every CTA takes one contiguous range of units, so a channel's taps are fetched once per CTA
  const int grid = P.units < most ? P.units : most;
  M2_SMEM_ONCE(longconv_bt_kernel, SMEM_MAX);
  return m2_launch("longconv_bt_kernel", (long long)P.B * P.L * P.D, longconv_bt_kernel, grid, THREADS, smem, st, P);
}

}  // namespace m2
