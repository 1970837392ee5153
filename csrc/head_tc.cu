// Logits of up to 64 rows on tcgen05: out[m, n] = x[m] . W[n], bf16 operands (kind::f16), fp32 accumulation and results.
//
// The product is a stream of the vocabulary matrix, read once.  The kernels it replaces load weights to registers, through L1: they
// had to wait until the projections before them had left the SMs (their shared memory leaves L1 too small), 9 to 16 rows cost half
// as much again as one (a second MMA tile, more activations beside the loads in flight), and from 17 rows on a library product
// rounded the logits to bf16.  Here copies go to shared memory, 160 KB an SM on their way, the first of them before the rows are
// known, and rows up to 64 are one operand: a tile is 128 vocabulary rows (the MMA's A: TMEM lanes) by 16, 32 or 64 activation rows
// (its B: TMEM columns), K in stages of 128 values.  The tensor cores' fp32 sums lose 6e-6 of the logits over 5120 terms in a row; so
// accumulators of 256 values of K each (of 5120 values with 17 to 32 rows 512, above that 640) share it, as the warps of the kernel for rows do, and are added up at the
// end: 2.5e-7 off 64 bits with 16 rows (3.0e-7 there), 6e-7 with 64 (1.7e-3 with results in bf16).  15 520 x 5120 with its norm, one after the other, us before and
// here (24 to read): 8 rows 31.6, 35.3; 12 and 16 rows 45.5, 35.6; 32 rows 40.6, 36.7; 64 rows 42.5, 39.5.  In a tick, where the kernel
// for rows waits: 8 sequences 432 both, 12 sequences 500 and 485, 2 x 8 rows 505 and 492.  The whole vocabulary, 248 320 x 5120 (394 to read), where a CTA goes
// through 13 tiles and there is no second accumulator: 8 rows 385, 386; 9 rows 541, 382; 16 rows 532, 387; 17 rows 410, 386; 32 rows 429, 395;
// 64 rows 505, 437; and 62 080 x 5120 8 rows 110, 117; 16 rows 147, 113; 64 rows 139, 126.
//
// Warp roles (192 threads): warp 0 = TMA producer, warp 1 = TMEM owner and MMA issuer, warps 2..5 = epilogue.  Every mbarrier wait is
// bounded (error word, abort flag, TMEM freed).
// In the place of the reference's dense head (tilerl_kernels/backend.py:559-1797, a library product there).
#include <cuda.h>

#include "tcgen05.cuh"

namespace {

constexpr int HT_M = 128, HT_BOX = 64;                        // vocabulary rows of a tile; values of a 128-byte row of a copy
constexpr int HT_THREADS = 192;

template <int BN>
struct HeadCfg {
  static constexpr int A_BOX = HT_M * 128, B_BOX = BN * 128, STAGE = 2 * (A_BOX + B_BOX);      // two boxes of 64 k each
  static constexpr int STAGES = 200 * 1024 / STAGE;
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int PARTS = 512 / BN;                       // accumulators of BN columns in TMEM
};

template <int BN>
__global__ void __launch_bounds__(HT_THREADS, 1)
head_bf16_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, float* out, long ldo, int M, int N, int nk) {
  using C = HeadCfg<BN>;
  constexpr int S = C::STAGES;
  extern __shared__ unsigned char ht_smem[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ht_smem) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * C::STAGE);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (S + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * S + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) mbar_init(full(s), 1), mbar_init(empty(s), 1);
    for (int b = 0; b < 2; ++b) mbar_init(acc_full(b), 1), mbar_init(acc_empty(b), 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents(67);
  const int tiles = (N + HT_M - 1) / HT_M, per = max(BN == 16 ? 2 : 4, (nk + C::PARTS - 1) / C::PARTS), parts = (nk + per - 1) / per;
  const int bufs = 2 * parts <= C::PARTS ? 2 : 1;             // a second tile's, where they fit

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      const uint32_t smem0 = smem_u32(smem);
      const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, units = mine * nk;
      auto load_w = [&](int u, int st) {
        const int tile = (int)blockIdx.x + u / nk * (int)gridDim.x, kt = u % nk;
        const uint32_t dst = smem0 + (uint32_t)st * C::STAGE;
        mbar_expect_tx(full(st), C::STAGE);
        tma_load_2d(dst, &map_w, kt * 2 * HT_BOX, tile * HT_M, full(st));
        tma_load_2d(dst + C::A_BOX, &map_w, kt * 2 * HT_BOX + HT_BOX, tile * HT_M, full(st));
      };
      const int pre = min(S, units);
      for (int u = 0; u < pre; ++u) load_w(u, u);             // weights do not depend on the kernel before
      pdl_wait();
      int st = 0;
      uint32_t ph = 0;
      for (int u = 0; u < units; ++u) {
        if (u >= pre) {
          if (!mbar_wait(empty(st), ph ^ 1u, abort_flag)) break;
          load_w(u, st);
        }
        const uint32_t dst = smem0 + (uint32_t)st * C::STAGE + 2 * C::A_BOX;
        tma_load_2d(dst, &map_x, u % nk * 2 * HT_BOX, 0, full(st));
        tma_load_2d(dst + C::B_BOX, &map_x, u % nk * 2 * HT_BOX + HT_BOX, 0, full(st));
        if (++st == S) st = 0, ph ^= 1u;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    pdl_wait();
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(HT_M >> 4) << 24);
      const uint64_t d0 = desc_sw128(smem_u32(smem));
      const uint32_t lo0 = (uint32_t)d0, hi = (uint32_t)(d0 >> 32);
      int st = 0, count = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, ++count) {
        const int buf = count % bufs;
        if (count >= bufs) {
          if (!(ok = mbar_wait(acc_empty(buf), (uint32_t)(count / bufs - 1) & 1u, abort_flag))) break;
          tc_fence_after();
        }
        for (int kt = 0; kt < nk; ++kt) {
          if (!(ok = mbar_wait(full(st), ph, abort_flag))) break;
          tc_fence_after();
          const uint32_t a = lo0 + (uint32_t)st * (uint32_t)(C::STAGE >> 4), b = a + (uint32_t)(2 * C::A_BOX >> 4);
#pragma unroll
          for (int i = 0; i < 8; ++i)                          // 16 k each, four to a box
            tc_mma_bf16_lh(tmem_base + (uint32_t)(buf * (512 / 2) + kt / per * BN), a + (i >> 2) * (C::A_BOX >> 4) + (i & 3) * 2, b + (i >> 2) * (C::B_BOX >> 4) + (i & 3) * 2, hi,
                           idesc, kt % per || i ? 1u : 0u);
          tc_commit(empty(st));
          if (++st == S) st = 0, ph ^= 1u;
        }
        if (ok) tc_commit(acc_full(buf));
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (warps 2..5): a thread a vocabulary row ----------------
    pdl_wait();                                               // (`out` may still be read by the kernel before)
    const int quad = warp & 3;
    int count = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++count) {
      const int buf = count % bufs, n = tile * HT_M + quad * 32 + lane;
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full(buf), (uint32_t)(count / bufs) & 1u, abort_flag))) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < BN; c += 16) {
        float v[16] = {};
        for (int q = 0; q < parts; ++q) {
          uint32_t r[32];
          tc_ld16(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * (512 / 2) + q * BN + c), r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(r[i]);
        }
        if (c + 16 == BN) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty(buf));
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c + i < M && n < N) out[(long)(c + i) * ldo + n] = v[i];
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    // give copies that are still in flight time to land before the CTA's memory goes away
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
  }
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}

typedef CUresult (*EncodeTiledFnH)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [rows, K] bf16, boxes of 64 values x `box` rows; what lies past either end reads as zero
bool head_map(CUtensorMap* m, const void* base, long rows, long K, int box) {
  static EncodeTiledFnH encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) return false;
    encode = (EncodeTiledFnH)fn;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t b[2] = {HT_BOX, (cuuint32_t)box}, estr[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
int launch_head(const CUtensorMap& mw, const CUtensorMap& mx, float* out, long ldo, int M, int N, int nk, int grid, cudaStream_t st) {
  auto kern = head_bf16_kernel<BN>;
  static TrlPerDevice<bool> set;
  bool& configured = set.here();
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, HeadCfg<BN>::SMEM) != cudaSuccess) return 3;
    configured = true;
  }
  return (int)trl_launch(kern, dim3(grid), dim3(HT_THREADS), (size_t)HeadCfg<BN>::SMEM, st, mw, mx, out, ldo, M, N, nk);
}

}  // namespace

// x [M, K] bf16 contiguous, w [N, K] bf16, out fp32 [M, ldo]; K % 8 == 0, both inputs 16-byte aligned, M up to 64.
TRL_API int trl_head_bf16(const void* x, const void* w, void* out, long ldo, int M, int N, int K, void* stream) {
  if (M < 1 || M > 64 || N < 1 || K < 8 || K % 8 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15))
    return (int)cudaErrorInvalidValue;
  const int bn = M <= 16 ? 16 : M <= 32 ? 32 : 64, tiles = (N + HT_M - 1) / HT_M;
  CUtensorMap mw, mx;
  if (!head_map(&mw, w, N, K, HT_M) || !head_map(&mx, x, M, K, bn)) return (int)cudaErrorInvalidValue;
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = min(tiles, sms), nk = (K + 2 * HT_BOX - 1) / (2 * HT_BOX);
  cudaStream_t st = (cudaStream_t)stream;
  switch (bn) {
    case 16: return launch_head<16>(mw, mx, (float*)out, ldo, M, N, nk, grid, st);
    case 32: return launch_head<32>(mw, mx, (float*)out, ldo, M, N, nk, grid, st);
    default: return launch_head<64>(mw, mx, (float*)out, ldo, M, N, nk, grid, st);
  }
}
