// Block-diagonal bf16 GEMMs on the 5th-generation tensor cores (tcgen05), operands staged
// by TMA into 128-byte-swizzled shared memory, float32 accumulators in tensor memory.
//
//   plain: out[:, k*q + n] = x[:, k*p : (k+1)*p] . w[k][n, :]  (+ bias)            (wo)
//   GLU  : h[:, k*q + n]   = gelu(x_k . wg[k][n, :]) * (x_{k+nb/2} . wg[k+nb/2][n, :])
//          -- the gated GEMM with GELU and the product applied in the epilogue, so the
//          (m, 2*inter) pre-activation is never written.
//
// One persistent CTA per SM walks output tiles of 128 rows x BN columns.  Warp 0 issues TMA
// loads into a ring of shared-memory stages, warp 1 issues the MMAs (one thread) into one of
// two TMEM accumulator buffers, warps 2-17 drain the other buffer (tcgen05.ld), apply the
// epilogue with the reference's bf16 rounding points and store.  Every mbarrier wait is
// bounded; a wait that runs out sets the device status word and the CTA winds down.
//
// Computation replaced: bert/src/mm/blockdiag_multiply.py:49-60 (torch.bmm per block),
// bert/src/mm/structured_linear.py:67-70 (bias), bert/src/bert_layers.py:492-501 (GLU).
#include "tc_common.cuh"

namespace m2 {

int m2_get_encode_fn(m2_encode_tiled_fn* fn) {
  static m2_encode_tiled_fn cached = nullptr;
  if (!cached) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres);
    if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || !p)
      return m2_set_error(M2_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cached = reinterpret_cast<m2_encode_tiled_fn>(p);
  }
  *fn = cached;
  return M2_OK;
}

int m2_make_tmap_bf16_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                         uint32_t box_rows) {
  m2_encode_tiled_fn enc;
  int rc = m2_get_encode_fn(&enc);
  if (rc) return rc;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return m2_set_error(M2_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return M2_OK;
}

namespace gemm {


constexpr int BM = 128;
constexpr int BK = 64;                 // one 128-byte swizzle row of bf16
constexpr int EPI_WARPS = 16;              // four warps per TMEM lane quarter, each a quarter of the columns
constexpr int EPI_WARP0 = 3;               // warp 0: TMA producer, warps 1-2: MMA issuers, then the epilogue warps
constexpr int THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
constexpr int A_BYTES = BM * BK * 2;   // 16 KB
constexpr int SMEM_BUDGET = 200 * 1024;

struct Params {
  int M, p, q, nb_out, pair_off, ntn, ntm, ksteps, total_tiles, out_cols, wide_out;
  void* out; long long ldo;
  const float* bias;
};

template <int BN, bool GLU>
struct Cfg {
  static constexpr int NACC = GLU ? 2 : 1;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = NACC * (A_BYTES + B_BYTES);
  static constexpr int NSTAGES = (SMEM_BUDGET / STAGE_BYTES) > 8 ? 8 : (SMEM_BUDGET / STAGE_BYTES);
  static constexpr int ACC_COLS = NACC * BN;         // TMEM columns of one accumulator buffer
  static constexpr int TCOLS = (2 * ACC_COLS <= 32) ? 32 : (2 * ACC_COLS <= 64) ? 64 : (2 * ACC_COLS <= 128) ? 128
                               : (2 * ACC_COLS <= 256) ? 256 : 512;
  static constexpr int SMEM = NSTAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
  static_assert(2 * ACC_COLS <= 512, "accumulators exceed tensor memory");
  static_assert(NSTAGES >= 2, "need at least two stages");
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// GLU epilogue of one tile for one warp: columns [chalf*CW, (chalf+1)*CW) of the gate accumulator at
// `tacc` and of the linear accumulator BN columns further, as gelu(gate) (cast to bf16) * linear.
// All of the warp's columns are read into registers first and the accumulator buffer is handed back
// (`tempty`) before any arithmetic, so the next tile's MMAs never wait for a GELU.
template <int BN, int CW>
__device__ __forceinline__ void glu_epilogue_tile(uint32_t tacc, int chalf, __nv_bfloat16* orow, bool in_range, int wide_out,
                                                  uint64_t* tempty) {
  constexpr int NCH = CW / 16;
  uint32_t a[NCH][16], b[NCH][16];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    tc::tmem_ld16(tacc + chalf * CW + 16 * ch, a[ch]);
    tc::tmem_ld16(tacc + BN + chalf * CW + 16 * ch, b[ch]);
  }
  tc::tmem_ld_wait();
  tc::tc_fence_before();
  tc::mbar_arrive(tempty);
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    const int c0 = chalf * CW + 16 * ch;
    uint32_t packed[8];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const uint32_t g = pack_bf16(__uint_as_float(a[ch][j]), __uint_as_float(a[ch][j + 1]));
      const uint32_t n = pack_bf16(__uint_as_float(b[ch][j]), __uint_as_float(b[ch][j + 1]));
      float a0, a1;
      gelu_pair(__uint_as_float(g << 16), __uint_as_float(g & 0xFFFF0000u), a0, a1);
      packed[j >> 1] = bf2_mul(pack_bf16(a0, a1), n);   // GELU output cast to bf16, times the linear half
    }
    if (in_range) {
      if (wide_out) {                   // one full 32-byte sector per thread
        stg256(orow + c0, packed[0], packed[1], packed[2], packed[3], packed[4], packed[5], packed[6], packed[7]);
      } else {
        uint4* dst = reinterpret_cast<uint4*>(orow + c0);
        dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
      }
    }
  }
}

template <int BN, bool GLU>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Params P) {
  using C = Cfg<BN, GLU>;
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte alignment is what the 128-byte swizzle pattern is anchored to
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::NSTAGES * C::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::NSTAGES;
  uint64_t* tfull = bars + 2 * C::NSTAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = tc::uniform_warp_id(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::NSTAGES; ++s) { tc::mbar_init(full + s, 1); tc::mbar_init(empty + s, C::NACC); }
    for (int b = 0; b < 2; ++b) { tc::mbar_init(tfull + b, C::NACC); tc::mbar_init(tempty + b, 32 * EPI_WARPS); }
    *abort_flag = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tmA);
    tc::tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, C::TCOLS);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------
    if (tc::elect_one()) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const int nt = tile % P.ntn, kb = (tile / P.ntn) % P.nb_out, mt = tile / (P.ntn * P.nb_out);
        for (int ks = 0; ks < P.ksteps; ++ks) {
          if (!tc::mbar_wait(empty + stage, phase ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY)) { ok = false; break; }
          unsigned char* st = smem + stage * C::STAGE_BYTES;
          tc::mbar_expect_tx(full + stage, C::STAGE_BYTES);
          tc::tma_load_2d(st, &tmA, full + stage, kb * P.p + ks * BK, mt * BM);
          tc::tma_load_2d(st + A_BYTES, &tmB, full + stage, ks * BK, kb * P.q + nt * BN);
          if (GLU) {
            const int kn = kb + P.pair_off;
            tc::tma_load_2d(st + A_BYTES + C::B_BYTES, &tmA, full + stage, kn * P.p + ks * BK, mt * BM);
            tc::tma_load_2d(st + 2 * A_BYTES + C::B_BYTES, &tmB, full + stage, ks * BK, kn * P.q + nt * BN);
          }
          if (++stage == C::NSTAGES) { stage = 0; phase ^= 1; }
        }
      }
      tc::drain_loads(full, C::NSTAGES, tc::ring_parities(stage, phase));
    }
  } else if (warp >= 1 && warp <= C::NACC) {
    // ------------------------------- MMA issuers --------------------------------
    // The two accumulators of the gated product have one issuing thread each: warp 1 the gate block, warp 2 the
    // linear block.  Both wait for the same stage and both commit to its `empty` barrier and to the accumulator
    // buffer's `tfull` (count NACC).
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::make_idesc(BM, BN, 1);
      const int chain = warp - 1;
      const uint64_t dA0 = tc::smem_desc_k_sw128(tc::smem_u32(smem + chain * (A_BYTES + C::B_BYTES)));
      const uint64_t dB0 = tc::desc_advance(dA0, A_BYTES >> 4);
      int stage = 0; uint32_t phase = 0;
      int buf = 0; uint32_t bphase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        if (!tc::mbar_wait(tempty + buf, bphase ^ 1, abort_flag, tc::ST_TIMEOUT_MMA)) break;
        tc::tc_fence_after();
        const uint32_t acc = tmem_base + buf * C::ACC_COLS + chain * BN;
        for (int ks = 0; ks < P.ksteps; ++ks) {
          if (!tc::mbar_wait(full + stage, phase, abort_flag, tc::ST_TIMEOUT_TMA)) { ok = false; break; }
          tc::tc_fence_after();
          const uint32_t off = (uint32_t)(stage * (C::STAGE_BYTES >> 4));
          const uint64_t dA = tc::desc_advance(dA0, off), dB = tc::desc_advance(dB0, off);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            // 16 bf16 along K = 32 bytes = 2 units of the descriptor's 16-byte address field
            tc::mma_ss(acc, tc::desc_advance(dA, 2 * kk), tc::desc_advance(dB, 2 * kk), idesc, (ks | kk) ? 1u : 0u);
          }
          tc::mma_commit(empty + stage);        // stage reusable once these MMAs have read it
          if (++stage == C::NSTAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        tc::mma_commit(tfull + buf);            // accumulator complete
        if ((buf ^= 1) == 0) bphase ^= 1;
      }
    }
  } else if (warp >= EPI_WARP0) {
    // ------------------------------- epilogue -----------------------------------
    const int quarter = warp & 3;               // TMEM lanes this warp may touch: 32*quarter ..
    const int chalf = (warp - EPI_WARP0) >> 2;  // which slice of the tile's columns
    constexpr int CW = BN / (EPI_WARPS / 4);    // columns per warp
    static_assert(CW % 16 == 0, "column slice must be a multiple of 16");
    int buf = 0; uint32_t bphase = 0;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(P.out);
    for (int tile = blockIdx.x; tile < P.total_tiles; tile += gridDim.x) {
      const int nt = tile % P.ntn, kb = (tile / P.ntn) % P.nb_out, mt = tile / (P.ntn * P.nb_out);
      if (!tc::mbar_wait(tfull + buf, bphase, abort_flag, tc::ST_TIMEOUT_EPI)) break;
      tc::tc_fence_after();
      const int row = mt * BM + quarter * 32 + lane;
      const int col0 = kb * P.q + nt * BN;
      const uint32_t tacc = tmem_base + buf * C::ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      __nv_bfloat16* orow = out + (long long)row * P.ldo + col0;
      if constexpr (GLU) {
        glu_epilogue_tile<BN, CW>(tacc, chalf, orow, row < P.M, P.wide_out, tempty + buf);
      } else {
      // the warp's columns go to registers in one sweep and the buffer is handed back before the stores
      constexpr int NCH = CW / 16;
      uint32_t acc_r[NCH][16];
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) tc::tmem_ld16(tacc + chalf * CW + 16 * ch, acc_r[ch]);
      tc::tmem_ld_wait();
      tc::tc_fence_before();
      tc::mbar_arrive(tempty + buf);
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        const int c0 = chalf * CW + 16 * ch;
        const uint32_t (&a)[16] = acc_r[ch];
        uint32_t packed[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          float v0 = bf16r(__uint_as_float(a[j]));
          float v1 = bf16r(__uint_as_float(a[j + 1]));
          if (P.bias) {
            v0 += bf16r(__ldg(P.bias + col0 + c0 + j));
            v1 += bf16r(__ldg(P.bias + col0 + c0 + j + 1));
          }
          packed[j >> 1] = pack_bf16(v0, v1);
        }
        if (row < P.M) {
          if (P.wide_out) {                     // one full 32-byte sector per thread
            stg256(orow + c0, packed[0], packed[1], packed[2], packed[3], packed[4], packed[5], packed[6], packed[7]);
          } else {
            uint4* dst = reinterpret_cast<uint4*>(orow + c0);
#pragma unroll
            for (int v = 0; v < 2; ++v)
              dst[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
          }
        }
      }
      }
      if ((buf ^= 1) == 0) bphase ^= 1;
    }
  }

  // ------------------------------- teardown -------------------------------------
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, C::TCOLS);
  }
}





// ---------------------------------------------------------------------------------------
// GLU GEMM with the x slices resident in shared memory.  The kernel above brings 64 KB through TMA per
// K step (x and wg tiles of both blocks), and its TMA throughput -- about 38 bytes per clock and SM from
// L2, whatever the box shape and whether one or two threads issue the loads -- is what paces it.  When
// K = d_model / nblocks <= 192 the two K-slices of x one row tile needs (96 KB) stay put while the CTA
// walks over the column tiles of the block pair, and only wg rows (32 KB per K step) stream through the
// ring: 112 instead of 196 KB per tile.  A CTA
// owns a contiguous range of units (row tile, block pair, group of column tiles), so consecutive units
// mostly share their x; when they do not, the first tile of the new unit brings the x tiles in K step
// by K step, each as soon as the last MMAs reading the old one have completed (`a_empty`).
// Two issuing warps as above; same epilogue.
// ---------------------------------------------------------------------------------------
namespace res {
constexpr int BN = 128, MAX_KS = 3, NSTB = 4;
constexpr int B_STAGE = 2 * BN * BK * 2;                   // gate + linear wg rows of one K step: 32 KB
constexpr int OFF_B = 2 * MAX_KS * A_BYTES;                // after the resident x tiles: 96 KB
constexpr int OFF_BAR = OFF_B + NSTB * B_STAGE;
constexpr int NBARS = 2 * NSTB + MAX_KS + 4;
constexpr int SMEM = OFF_BAR + NBARS * 8 + 16 + 1024;
static_assert(SMEM <= 227 * 1024, "shared memory budget");
}  // namespace res

struct ResParams {
  int M, p, q, nb_half, ksteps, ntn, gs, ngroups, total_units, wide_out;
  void* out; long long ldo;
};

__global__ void __launch_bounds__(THREADS, 1)
glu_res_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const ResParams P) {
  using namespace res;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* b_full = bars;                   // [NSTB] wg rows (and, on a unit's first tile, x tiles) landed
  uint64_t* b_empty = b_full + NSTB;         // [NSTB] both issuers' MMAs have read the stage
  uint64_t* a_empty = b_empty + NSTB;        // [MAX_KS] both issuers are done with the x tiles of K step ks
  uint64_t* tfull = a_empty + MAX_KS;        // [2]
  uint64_t* tempty = tfull + 2;              // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = tc::uniform_warp_id(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTB; ++s) { tc::mbar_init(b_full + s, 1); tc::mbar_init(b_empty + s, 2); }
    for (int k = 0; k < MAX_KS; ++k) tc::mbar_init(a_empty + k, 2);
    for (int b = 0; b < 2; ++b) { tc::mbar_init(tfull + b, 2); tc::mbar_init(tempty + b, 32 * EPI_WARPS); }
    *abort_flag = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tmA);
    tc::tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  // this CTA's contiguous range of units; unit = (pair = row tile x block pair, group of column tiles)
  const int u0 = (int)((long long)blockIdx.x * P.total_units / gridDim.x);
  const int u1 = (int)((long long)(blockIdx.x + 1) * P.total_units / gridDim.x);
  auto decode = [&](int unit, int& pair, int& mt, int& kb, int& nt0, int& ntiles) {
    pair = unit / P.ngroups;
    const int g = unit % P.ngroups;
    mt = pair / P.nb_half; kb = pair % P.nb_half;
    nt0 = g * P.gs;
    ntiles = P.ntn - nt0 < P.gs ? P.ntn - nt0 : P.gs;
  };

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------
    if (tc::elect_one()) {
      int stage = 0; uint32_t phase = 0;
      int epoch = -1, prev_pair = -1;
      bool ok = true;
      for (int unit = u0; unit < u1 && ok; ++unit) {
        int pair, mt, kb, nt0, ntiles;
        decode(unit, pair, mt, kb, nt0, ntiles);
        const bool new_x = pair != prev_pair;
        if (new_x) { ++epoch; prev_pair = pair; }
        for (int t = 0; t < ntiles && ok; ++t) {
          const bool load_x = new_x && t == 0;
          for (int ks = 0; ks < P.ksteps; ++ks) {
            if (!tc::mbar_wait(b_empty + stage, phase ^ 1, abort_flag, tc::ST_TIMEOUT_EMPTY)) { ok = false; break; }
            if (load_x && epoch > 0 &&
                !tc::mbar_wait(a_empty + ks, (uint32_t)(epoch - 1) & 1u, abort_flag, tc::ST_TIMEOUT_EMPTY)) { ok = false; break; }
            unsigned char* st = smem + OFF_B + stage * B_STAGE;
            tc::mbar_expect_tx(b_full + stage, B_STAGE + (load_x ? 2 * A_BYTES : 0));
            if (load_x) {
              tc::tma_load_2d(smem + ks * A_BYTES, &tmA, b_full + stage, kb * P.p + ks * BK, mt * BM);
              tc::tma_load_2d(smem + (MAX_KS + ks) * A_BYTES, &tmA, b_full + stage, (kb + P.nb_half) * P.p + ks * BK, mt * BM);
            }
            const int row_g = kb * P.q + (nt0 + t) * BN;
            tc::tma_load_2d(st, &tmB, b_full + stage, ks * BK, row_g);
            tc::tma_load_2d(st + B_STAGE / 2, &tmB, b_full + stage, ks * BK, row_g + P.nb_half * P.q);
            if (++stage == NSTB) { stage = 0; phase ^= 1; }
          }
        }
      }
      tc::drain_loads(b_full, NSTB, tc::ring_parities(stage, phase));
    }
  } else if (warp == 1 || warp == 2) {
    // ------------------------------- MMA issuers: warp 1 gate, warp 2 linear ----------------------
    // Each thread issues every tile's MMAs of its accumulator in order, so its commit to `a_empty` after
    // the last tile that reads the old x covers all of its earlier MMAs as well.
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::make_idesc(BM, BN, 1);
      const int chain = warp - 1;
      const uint64_t dA0 = tc::smem_desc_k_sw128(tc::smem_u32(smem + chain * MAX_KS * A_BYTES));
      const uint64_t dB0 = tc::smem_desc_k_sw128(tc::smem_u32(smem + OFF_B + chain * (B_STAGE / 2)));
      int stage = 0; uint32_t phase = 0;
      int buf = 0; uint32_t bphase = 0;
      bool ok = true;
      for (int unit = u0; unit < u1 && ok; ++unit) {
        int pair, mt, kb, nt0, ntiles;
        decode(unit, pair, mt, kb, nt0, ntiles);
        const bool x_changes = unit + 1 < u1 && (unit + 1) / P.ngroups != pair;
        for (int t = 0; t < ntiles && ok; ++t) {
          if (!tc::mbar_wait(tempty + buf, bphase ^ 1, abort_flag, tc::ST_TIMEOUT_MMA)) { ok = false; break; }
          tc::tc_fence_after();
          const uint32_t acc = tmem_base + buf * 2 * BN + chain * BN;
          const bool release_x = x_changes && t == ntiles - 1;
          for (int ks = 0; ks < P.ksteps; ++ks) {
            if (!tc::mbar_wait(b_full + stage, phase, abort_flag, tc::ST_TIMEOUT_TMA)) { ok = false; break; }
            tc::tc_fence_after();
            const uint64_t dA = tc::desc_advance(dA0, ks * (A_BYTES >> 4)), dB = tc::desc_advance(dB0, stage * (B_STAGE >> 4));
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) tc::mma_ss(acc, tc::desc_advance(dA, 2 * kk), tc::desc_advance(dB, 2 * kk), idesc, (ks | kk) ? 1u : 0u);
            tc::mma_commit(b_empty + stage);
            if (release_x) tc::mma_commit(a_empty + ks);
            if (++stage == NSTB) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          tc::mma_commit(tfull + buf);
          if ((buf ^= 1) == 0) bphase ^= 1;
        }
      }
    }
  } else if (warp >= EPI_WARP0) {
    // ------------------------------- epilogue -----------------------------------
    const int quarter = warp & 3;
    const int chalf = (warp - EPI_WARP0) >> 2;
    constexpr int CW = BN / (EPI_WARPS / 4);
    int buf = 0; uint32_t bphase = 0;
    bool ok = true;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(P.out);
    for (int unit = u0; unit < u1 && ok; ++unit) {
      int pair, mt, kb, nt0, ntiles;
      decode(unit, pair, mt, kb, nt0, ntiles);
      const int row = mt * BM + quarter * 32 + lane;
      for (int t = 0; t < ntiles; ++t) {
        if (!tc::mbar_wait(tfull + buf, bphase, abort_flag, tc::ST_TIMEOUT_EPI)) { ok = false; break; }
        tc::tc_fence_after();
        const uint32_t tacc = tmem_base + buf * 2 * BN + ((uint32_t)(quarter * 32) << 16);
        __nv_bfloat16* orow = out + (long long)row * P.ldo + kb * P.q + (nt0 + t) * BN;
        glu_epilogue_tile<BN, CW>(tacc, chalf, orow, row < P.M, P.wide_out, tempty + buf);
        if ((buf ^= 1) == 0) bphase ^= 1;
      }
    }
  }

  // ------------------------------- teardown -------------------------------------
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, 512);
  }
}


template <int BN, bool GLU>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const Params& P, cudaStream_t st) {
  using C = Cfg<BN, GLU>;
  auto kern = gemm_tc_kernel<BN, GLU>;
  M2_SMEM_ONCE(kern, C::SMEM);
  int grid = P.total_tiles < m2_sm_count() ? P.total_tiles : m2_sm_count();
  return m2_launch("gemm_tc_kernel", (long long)P.M * P.out_cols, kern, grid, THREADS, C::SMEM, st, tmA, tmB, P);
}

// Column tile of a block-diagonal GEMM with q columns per block: the widest that divides q is the most efficient; with
// few row tiles narrower ones put more SMs to work (wo at 1024 rows: 32 tiles of 192 columns, or 96 of 64).  A K step
// brings 128 rows of A and n of B at about 50 bytes per clock and multiplies for 2 n clocks, a tile costs some 2500 more.
static int pick_bn(int q, long long row_tiles, int ksteps) {
  int best = 0;
  double least = 0;
  for (int n : {256, 192, 128, 64}) {
    if (q % n) continue;
    const long long tiles = row_tiles * (q / n), waves = (tiles + m2_sm_count() - 1) / m2_sm_count();
    const double load = (BM + n) * BK * 2 / 50.0, mma = 2.0 * n;
    const double cost = waves * (ksteps * (load > mma ? load : mma) + 2500.0);
    if (best == 0 || cost < 0.97 * least) { least = cost; best = n; }
  }
  return best;
}

}  // namespace gemm

bool blockdiag_tc_supported(const m2_blockdiag_args* a) {
  return a->dtype == M2_BF16 && a->p % 64 == 0 && a->q % 64 == 0 &&
         a->in_features == a->nblocks * a->p && a->out_features == a->nblocks * a->q &&
         a->ldx % 8 == 0 && a->ldo % 8 == 0 && m2_aligned(a->x, 16) && m2_aligned(a->w, 16) &&
         m2_aligned(a->out, 16) && a->m >= 1;
}

bool glu_tc_supported(const m2_glu_args* a) {
  const int p = a->d_model / a->nblocks, q = 2 * a->inter / a->nblocks;
  return a->dtype == M2_BF16 && p % 64 == 0 && q % 128 == 0 && a->ldx % 8 == 0 && a->ldh % 8 == 0 &&
         m2_aligned(a->x, 16) && m2_aligned(a->wg, 16) && m2_aligned(a->h, 16) && a->m >= 1;
}

int blockdiag_tc_launch(const m2_blockdiag_args* a, cudaStream_t st) {
  using namespace gemm;
  const int bn = pick_bn(a->q, (long long)((a->m + BM - 1) / BM) * a->nblocks, a->p / BK);
  CUtensorMap tmA, tmB;
  int rc = m2_make_tmap_bf16_2d(&tmA, a->x, a->m, a->in_features, a->ldx, BM);
  if (rc) return rc;
  rc = m2_make_tmap_bf16_2d(&tmB, a->w, (uint64_t)a->nblocks * a->q, a->p, a->p, bn);
  if (rc) return rc;
  Params P;
  P.M = a->m; P.p = a->p; P.q = a->q; P.nb_out = a->nblocks; P.pair_off = 0;
  P.ntn = a->q / bn; P.ntm = (a->m + BM - 1) / BM; P.ksteps = a->p / BK;
  P.total_tiles = P.ntm * P.nb_out * P.ntn; P.out_cols = a->out_features;
  P.out = a->out; P.ldo = a->ldo; P.bias = a->bias;
  P.wide_out = m2_aligned(a->out, 32) && a->ldo % 16 == 0 && a->q % 16 == 0;   // 32-byte stores are legal
  switch (bn) {
    case 256: return launch<256, false>(tmA, tmB, P, st);
    case 192: return launch<192, false>(tmA, tmB, P, st);
    case 128: return launch<128, false>(tmA, tmB, P, st);
    default: return launch<64, false>(tmA, tmB, P, st);
  }
}

int glu_tc_launch(const m2_glu_args* a, cudaStream_t st) {
  using namespace gemm;
  const int p = a->d_model / a->nblocks, q = 2 * a->inter / a->nblocks;
  CUtensorMap tmA, tmB;
  int rc = m2_make_tmap_bf16_2d(&tmA, a->x, a->m, a->d_model, a->ldx, BM);
  if (rc) return rc;
  rc = m2_make_tmap_bf16_2d(&tmB, a->wg, (uint64_t)a->nblocks * q, p, p, 128);
  if (rc) return rc;
  Params P;
  P.M = a->m; P.p = p; P.q = q; P.nb_out = a->nblocks / 2; P.pair_off = a->nblocks / 2;
  P.ntn = q / 128; P.ntm = (a->m + BM - 1) / BM; P.ksteps = p / BK;
  P.total_tiles = P.ntm * P.nb_out * P.ntn; P.out_cols = a->inter;
  P.out = a->h; P.ldo = a->ldh; P.bias = nullptr;
  P.wide_out = m2_aligned(a->h, 32) && a->ldh % 16 == 0 && q % 16 == 0;
  // K <= 192 per block: x slices resident in shared memory, unless the caller asks for the streaming
  // two-accumulator kernel (variant 1; the tests compare the two bit for bit).
  if (P.ksteps <= res::MAX_KS && a->variant != 1) {
    ResParams R;
    R.M = a->m; R.p = p; R.q = q; R.nb_half = a->nblocks / 2; R.ksteps = P.ksteps; R.ntn = q / res::BN;
    // column tiles per unit: about 6 units per SM, so that the contiguous ranges balance
    const long long pairs = (long long)P.ntm * R.nb_half;
    int gs = R.ntn;
    while (gs > 1 && pairs * ((R.ntn + gs - 1) / gs) < 6LL * m2_sm_count()) gs = (gs + 1) / 2;
    R.gs = gs; R.ngroups = (R.ntn + gs - 1) / gs;
    R.total_units = (int)(pairs * R.ngroups);
    R.wide_out = P.wide_out; R.out = a->h; R.ldo = a->ldh;
    M2_SMEM_ONCE(glu_res_kernel, res::SMEM);
    const int grid = R.total_units < m2_sm_count() ? R.total_units : m2_sm_count();
    return m2_launch("glu_res_kernel", (long long)a->m * a->d_model, glu_res_kernel, grid, THREADS, res::SMEM, st, tmA, tmB, R);
  }
  return launch<128, true>(tmA, tmB, P, st);
}

}  // namespace m2
