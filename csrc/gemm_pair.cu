// tcgen05 block-scaled NVFP4 GEMM on pairs of SMs: gemm_tc.cu's product for one, two or four NVFP4 terms a token, at every
// number of columns.
//
// What bounds the one-SM form there is shared memory and its epilogue: a k-tile of 128 x 256 x 256 writes 54 KB and its MMAs
// read 48 KB back, and the tensor cores stand still while the only accumulator that fits is read out (34 816 x 5120, 2000 rows:
// 402 us; 293 with the epilogue left out, 236 with the MMAs left out too).  Here two SMs work on 256 rows x BN columns
// (`cta_group::2`): each holds its own 128 weight rows, and HALF of the activation columns, which the MMA hands to both, so that
// a k-tile of 128 x 192 x 256 a SM writes 34 KB and reads 28.  192 columns leave room in TMEM for two accumulators (2 x 192)
// beside two buffers of scale factors (2 x 64): the epilogue of a tile runs beside the next one's MMAs.  Few columns take
// narrower tiles, which leave room for more stages of weights; where there are fewer tiles than pairs, two or three pairs of a
// cluster share a tile along K and add their parts through each other's shared memory, no scratch, no counters, in a fixed
// order (rules at gemm_tc.cu::plan_pair).  With the quantiser, one-SM form (behind elect.sync too) and here, us:
//     rows                 8          32          128          512         2000
//     34 816 x 5120   25.3 21.4   26.2 21.5   42.6  30.8   125  90.4   402  283   (2.5 PFLOP/s counted once a row)
//     5120 x 17 408   23.7 17.0   22.6 16.6   37.1  24.5   84.7 53.5   230  186
//     16 480 x 5120   20.1 13.4   20.2 13.7   30.6  18.3   52.3 46.6   169  142
//     5120 x 6144     14.8  9.7   15.5  9.8   28.3  12.1   45.1 23.6   117   60
//     1024 x 3072      8.4  7.4    8.5  6.9   23.3   7.8   29.6  9.8    29   19   (3, 16, 128, 512, 2000 rows; without
//                              the barriers round the TMEM allocation, which the rest has: 0.3 to 1 us a product)
//
// Roles (10 warps): warp 0 = TMA producer of its SM's operands (a stage = 256 k; both SMs' copies count on the even one's
// barrier), warp 1 = TMEM owner and, in the even SM, MMA issuer for both, warps 2-9 = epilogue: two groups of four, each
// half of the columns.  A warp turns 32 rows x 16 tokens round through its own piece of shared memory, so that results leave
// as 16-byte stores along a token's row (2 bytes a lane along the rows were 3.7 us a tile in the open), or as 8-byte ones or one by
// one where rows, strides or bases are no multiple (a rank's 2060 rows).  Before, those went to the one-SM kernel in whole tiles; that, here
// as 8-byte stores, and a multiple of eight beside it, us with the quantiser, plain and with a residual:
//     rows                    128                             512                             2000
//     2060 x 5120      16.3 10.7 10.6, 23.9 11.4 10.7   18.9 14.2 13.9, 27.1 14.2 14.2   39.6 33.2 32.5, 56.2 34.4 33.5
//     16 484 x 5120    20.7 18.3 18.1, 29.3 18.5 18.3   59.5 47.5 46.4, 104  49.6 51.4   209  151  142,  369  184  169
// (one by one 11.7, 22.5; 16.9, 20.3; 44.2, 57.9 and 23.0, 29.0; 64.2, 96.4; 204, 318, residuals not yet requested ahead).  Weights' and
// activations' scales come by tiled copies too, since only these may count on the other SM's barrier; none is multicast.
//
// In the reference's place: linear_fp4_fp8 / linear_fp4_mma8 (packages/tilerl-kernels/src/tilerl_kernels/kernels_linear.py:924-1687).
#include <cuda.h>
#include "common.cuh"
#include "tcgen05.cuh"
#include "gemm_pair.cuh"

namespace {

constexpr int GP_ROWS = 128;                      // weight rows an SM
constexpr int GP_KT = 128;                        // bytes of K a stage (256 e2m1)
constexpr int GP_THREADS = 320;
constexpr int GP_MAX_STAGES = 9;
constexpr int GP_TR_STRIDE = 36;                  // floats a token in a warp's turning piece: 32 rows, and 4 so that reads spread
constexpr int GP_TR_BYTES = 16 * GP_TR_STRIDE * 4 + 128;      // and the column scales of a chunk

enum { GP_STORE = 0, GP_RESIDUAL = 1, GP_SWIGLU = 2, GP_STORE_F32 = 3 };

template <int BN, int J>
struct PairCfg {
  static constexpr int A_BYTES = GP_ROWS * GP_KT, SFA_BYTES = 4 * TC_SF_ATOM;
  static constexpr int ATOMS = BN > 128 ? 2 : 1;  // of activation scales (128 columns each) that a tile touches
  static constexpr int B_BYTES = BN / 2 * GP_KT, SFB_BYTES = ATOMS * 4 * TC_SF_ATOM;
  static constexpr int STAGE = A_BYTES + SFA_BYTES + B_BYTES + SFB_BYTES;
  static constexpr int OFF_SFA = A_BYTES, OFF_B = A_BYTES + SFA_BYTES + (1024 - SFA_BYTES % 1024) % 1024, OFF_SFB = OFF_B + B_BYTES;
  static constexpr int STAGES = 208 * 1024 / STAGE < GP_MAX_STAGES ? 208 * 1024 / STAGE : GP_MAX_STAGES;
  // epilogue: chunks of CH columns (16 tokens of one or two terms, 8 of four), in one or two groups of four warps
  static constexpr int CH = J == 1 ? 16 : 32, HALVES = BN / 2 >= CH ? 2 : 1, COLS_WARP = BN / HALVES;
  static constexpr int SMEM = STAGES * STAGE + 8 * GP_TR_BYTES + 512 + 1024;
  // TMEM: accumulators at 0 and BN, two buffers of 64 columns of scale factors behind them
  static constexpr int TMEM_COLS = BN <= 64 ? 256 : 512, SF_COL0 = TMEM_COLS - 128;
  static_assert(OFF_SFB + SFB_BYTES == STAGE && STAGE % 1024 == 0 && SMEM <= 227 * 1024 && 2 * BN <= SF_COL0, "layout");
  static_assert(SMEM >= 208 * 1024, "no other kernel with TMEM fits beside it on an SM");
};

struct PairParams {
  const float* tscale;
  const float* rs;
  const bf16* residual;
  void* out;
  int N, tokens, cols, ldr, ldo, r_tiles, c_tiles, nk, w_tiled, epi;
  int vec;               // rows of a token that leave as one vector: 8, 4 or 1
  int parts;             // pairs that share a tile (a cluster), each a part of K; 1: a pair goes through whole tiles
};

__device__ __forceinline__ uint32_t gp_map(uint32_t addr, int cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ float4 gp_ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// What a CTA waits for without a limit, and why it ends.  A cluster barrier takes the place of __syncthreads for two to six CTAs
// that the hardware starts together; shared memory of another CTA may only be touched once one has been passed, and no CTA may
// leave before the last access to its own, so an mbarrier with a limit can stand in for neither the first nor the last.  Every thread
// comes to each of them: no path returns early, and all waits in between (the ring, the accumulators, the producers' tail) have
// a limit, after which they leave their loop.  The allocation of TMEM waits for the other CTA's, right behind the first barrier, and
// for columns to be free: a CTA leaves too little shared memory on its SM for any other kernel that holds some (each takes
// 190 KB or more, and gives its columns back on every path).  The release waits for the other CTA's, behind a barrier too.
// Not the .aligned forms: the warps come here from loops and branches that their lanes left at different times, and a warp
// that is not converged would count more than once.
__device__ __forceinline__ void gp_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void gp_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void gp_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void gp_commit(uint32_t bar, uint16_t both) {       // on this barrier of both SMs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(both) : "memory");
}
__device__ __forceinline__ void gp_cp_sf(uint32_t taddr, uint32_t lo, uint32_t hi) {
  asm volatile("{ .reg .b64 d; mov.b64 d, {%1, %2}; tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], d; }"
               ::"r"(taddr), "r"(lo), "r"(hi) : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc, uint32_t sfa,
                                       uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; .reg .b64 da, db;\n"
      "  mov.b64 da, {%1, %3}; mov.b64 db, {%2, %3};\n"
      "  setp.ne.b32 p, %5, 0;\n"
      "  tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %4, [%6], [%7], p; }\n"
      ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb) : "memory");
}

__device__ __forceinline__ float gp_swiglu(float g, float u, float s) { return __fdividef(g * s, 1.f + __expf(-(g * s))) * (u * s); }

// A value of a row and token, times s, out; SwiGLU (rows in (gate, up) pairs): the pair of an even row.
__device__ __forceinline__ void gp_store1(const PairParams& p, int tok, int row, float v, float up, float s, float res) {
  const size_t at = (size_t)tok * p.ldo;
  if (p.epi == GP_SWIGLU) {
    if (!(row & 1) && row + 1 < p.N) reinterpret_cast<bf16*>(p.out)[at + (row >> 1)] = __float2bfloat16(gp_swiglu(v, up, s));
  } else if (p.epi == GP_STORE_F32) {
    reinterpret_cast<float*>(p.out)[at + row] = fmaf(v, s, res);
  } else {
    reinterpret_cast<bf16*>(p.out)[at + row] = __float2bfloat16(fmaf(v, s, res));
  }
}
// Four of them.
__device__ __forceinline__ void gp_store4(const PairParams& p, int tok, int row, float4 v, float s, uint2 res) {
  const size_t at = (size_t)tok * p.ldo;
  if (p.epi == GP_SWIGLU) {
    *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(p.out) + at + (row >> 1)) = f2_to_bf162_bits(gp_swiglu(v.x, v.y, s), gp_swiglu(v.z, v.w, s));
    return;
  }
  const float2 a = bf162_bits_to_f2(res.x), b = bf162_bits_to_f2(res.y);
  v = make_float4(fmaf(v.x, s, a.x), fmaf(v.y, s, a.y), fmaf(v.z, s, b.x), fmaf(v.w, s, b.y));
  if (p.epi == GP_STORE_F32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at + row) = v;
  else *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(p.out) + at + row) = make_uint2(f2_to_bf162_bits(v.x, v.y), f2_to_bf162_bits(v.z, v.w));
}
// Eight values of a row block and token, times s, out.
__device__ __forceinline__ void gp_store8(const PairParams& p, int tok, int row, float4 lo, float4 hi, float s, uint4 res) {
  if (p.epi == GP_SWIGLU) {                          // rows in (gate, up) pairs
    *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(p.out) + (size_t)tok * p.ldo + (row >> 1)) =
        make_uint2(f2_to_bf162_bits(gp_swiglu(lo.x, lo.y, s), gp_swiglu(lo.z, lo.w, s)), f2_to_bf162_bits(gp_swiglu(hi.x, hi.y, s), gp_swiglu(hi.z, hi.w, s)));
    return;
  }
  const float2 a = bf162_bits_to_f2(res.x), b = bf162_bits_to_f2(res.y), c = bf162_bits_to_f2(res.z), d = bf162_bits_to_f2(res.w);
  lo = make_float4(fmaf(lo.x, s, a.x), fmaf(lo.y, s, a.y), fmaf(lo.z, s, b.x), fmaf(lo.w, s, b.y));      // (no residual: zeros)
  hi = make_float4(fmaf(hi.x, s, c.x), fmaf(hi.y, s, c.y), fmaf(hi.z, s, d.x), fmaf(hi.w, s, d.y));
  if (p.epi == GP_STORE_F32) {
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (size_t)tok * p.ldo + row);
    o[0] = lo, o[1] = hi;
  } else {
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.out) + (size_t)tok * p.ldo + row) =
        make_uint4(f2_to_bf162_bits(lo.x, lo.y), f2_to_bf162_bits(lo.z, lo.w), f2_to_bf162_bits(hi.x, hi.y), f2_to_bf162_bits(hi.z, hi.w));
  }
}
// Residuals of V rows from `row` on, one vector (V = 1: in the low half).
template <int V>
__device__ __forceinline__ uint4 gp_residual(const PairParams& p, int tok, int row) {
  uint4 r = make_uint4(0u, 0u, 0u, 0u);
  if (p.epi != GP_RESIDUAL || tok >= p.tokens || row >= p.N) return r;
  const bf16* src = p.residual + (size_t)tok * p.ldr + row;
  if constexpr (V == 8) {
    r = __ldcg(reinterpret_cast<const uint4*>(src));
  } else if constexpr (V == 4) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(src));
    r.x = v.x, r.y = v.y;
  } else {
    r.x = __ldcg(reinterpret_cast<const unsigned short*>(src));
  }
  return r;
}

// A warp's piece of 32 rows x T tokens, V rows a lane and vector: V tokens at a time, 64 bytes of each.  `res`: the residuals in the
// order in which the values leave.
template <int V, int T>
__device__ __forceinline__ void gp_piece_residual(const PairParams& p, int tok0, int n0, int lane, uint32_t (&res)[T / 2]) {
#pragma unroll
  for (int i = 0; i < T / V; ++i) {
    const uint4 r = gp_residual<V>(p, tok0 + i * V + lane / (32 / V), n0 + lane % (32 / V) * V);
    if constexpr (V == 8) res[i * 4] = r.x, res[i * 4 + 1] = r.y, res[i * 4 + 2] = r.z, res[i * 4 + 3] = r.w;
    else if constexpr (V == 4) res[i * 2] = r.x, res[i * 2 + 1] = r.y;
    else res[i / 2] = i % 2 ? res[i / 2] | r.x << 16 : r.x;
  }
}
template <int V, int T>
__device__ __forceinline__ void gp_piece_store(const PairParams& p, int tok0, int n0, int lane, const float* tr, float s, const uint32_t (&res)[T / 2]) {
#pragma unroll
  for (int i = 0; i < T / V; ++i) {
    const int t = i * V + lane / (32 / V), tok = tok0 + t, col = lane % (32 / V) * V, row = n0 + col;
    const float* v = tr + t * GP_TR_STRIDE + col;
    if (tok >= p.tokens || row >= p.N) continue;
    if constexpr (V == 8) {
      gp_store8(p, tok, row, reinterpret_cast<const float4*>(v)[0], reinterpret_cast<const float4*>(v)[1], s, make_uint4(res[i * 4], res[i * 4 + 1], res[i * 4 + 2], res[i * 4 + 3]));
    } else if constexpr (V == 4) {
      gp_store4(p, tok, row, *reinterpret_cast<const float4*>(v), s, make_uint2(res[i * 2], res[i * 2 + 1]));
    } else {
      gp_store1(p, tok, row, v[0], v[lane < 31], s, __uint_as_float(i % 2 ? res[i / 2] & 0xffff0000u : res[i / 2] << 16));
    }
  }
}

// V: p.vec where it is 8; else 0 (the branches on it cost a tick of 32 sequences 0.5 %, as one kernel for all).
template <int BN, int J, bool SPLIT, int V>
__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_nvfp4_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_sfw,
                       const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_sfx, const PairParams p) {
  using C = PairCfg<BN, J>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* turn = smem + STAGES * C::STAGE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(turn + 8 * GP_TR_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int part = SPLIT ? pair % p.parts : 0, even = 2 * part;          // even: the cluster's CTA that issues for this pair
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };                              // the even SM's counts both SMs' copies
  auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + b); };   // of the even SM: both SMs' epilogue warps

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(full(s), 1), mbar_init(empty(s), 1);
    for (int b = 0; b < 2; ++b) mbar_init(acc_full(b), 1), mbar_init(acc_empty(b), 8 * C::HALVES);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // TMEM of a pair is taken by both SMs together: only once both CTAs are known to run (and the other SM's barriers are there).
  // An allocation that waits for its other half has no limit on its wait, as the mbarriers have.
  gp_cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  gp_cluster_sync();                                // both halves are allocated
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  // whole tiles, an even share for each pair; columns run fastest, so that a pair's weight rows stay while they do
  const long long T = (long long)p.r_tiles * p.c_tiles;
  const int tile0 = SPLIT ? pair / p.parts : (int)(pair * T / pairs), tile1 = SPLIT ? tile0 + 1 : (int)((pair + 1) * T / pairs);
  const int k0 = SPLIT ? part * p.nk / p.parts : 0, k1 = SPLIT ? (part + 1) * p.nk / p.parts : p.nk;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      const uint32_t smem0 = smem_u32(smem);
      const int units = (tile1 - tile0) * (k1 - k0);
      auto load_w = [&](int rt, int kt, int st) {
        const uint32_t dst = smem0 + (uint32_t)st * C::STAGE, bar = gp_map(full(st), even);
        const int nt = rt * 2 + rank;
        if (rank == 0) mbar_expect_tx(full(st), 2u * C::STAGE);
        gp_load_2d(dst, &map_w, p.w_tiled ? 0 : kt * GP_KT, p.w_tiled ? (nt * p.nk + kt) * GP_ROWS : nt * GP_ROWS, bar);
        gp_load_2d(dst + C::OFF_SFA, &map_sfw, 0, (nt * p.nk + kt) * 16, bar);
      };
      auto load_x = [&](int ct, int kt, int st) {
        const uint32_t dst = smem0 + (uint32_t)st * C::STAGE, bar = gp_map(full(st), even);
        gp_load_2d(dst + C::OFF_B, &map_x, kt * GP_KT, ct * BN + rank * (BN / 2), bar);
        gp_load_3d(dst + C::OFF_SFB, &map_sfx, 0, kt * 16, ct * BN / 128, bar);
      };
      int w_rt = tile0 / p.c_tiles, w_ct = tile0 % p.c_tiles, w_kt = k0, x_ct = w_ct, x_kt = k0, st = 0;
      uint32_t ph = 0;
      auto next_w = [&] { if (++w_kt == k1) { w_kt = k0; if (++w_ct == p.c_tiles) w_ct = 0, ++w_rt; } };
      const int pre = min(STAGES, units);
      for (int u = 0; u < pre; ++u) load_w(w_rt, w_kt, u), next_w();       // weights do not depend on the previous kernel
      pdl_wait();
      for (int u = 0; u < units; ++u) {
        if (u >= pre) {
          if (!mbar_wait(empty(st), ph ^ 1u, abort_flag)) break;
          load_w(w_rt, w_kt, st), next_w();
        }
        load_x(x_ct, x_kt, st);
        if (++x_kt == k1) { x_kt = k0; if (++x_ct == p.c_tiles) x_ct = 0; }
        if (++st == STAGES) st = 0, ph ^= 1u;
      }
      // the last arrivals of the even SM's MMAs on this CTA's barriers, before its memory goes away
      for (int s = 0; s < pre; ++s) {
        const int u = units - pre + s;              // the last unit of its stage
        if (!mbar_wait(empty(u % STAGES), (uint32_t)(u / STAGES) & 1u, abort_flag)) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (for both SMs) ----------------
    pdl_wait();
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * GP_ROWS) >> 4) << 24);
      const uint64_t d_op = desc_sw128(smem_u32(smem)), d_sf = desc_sf(smem_u32(smem));
      const uint32_t op_lo = (uint32_t)d_op, op_hi = (uint32_t)(d_op >> 32), sf_lo = (uint32_t)d_sf, sf_hi = (uint32_t)(d_sf >> 32);
      int st = 0, it = 0, ct = tile0 % p.c_tiles;
      uint32_t ph = 0;
      const uint16_t both = (uint16_t)(3u << even);
      bool ok = true;
      for (int tile = tile0; ok && tile < tile1; ++tile) {
        const int n = tile - tile0, buf = n & 1;
        if (n >= 2) {
          ok = mbar_wait(acc_empty(buf), (uint32_t)((n >> 1) - 1) & 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
        }
        const uint32_t acc = tmem_base + (uint32_t)buf * BN;
        const uint32_t sfb_off = (uint32_t)(ct * BN % 128) / 32;        // a tile may start in the middle of an atom of scales
        for (int kt = k0; kt < k1; ++kt, ++it) {
          ok = mbar_wait(full(st), ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t off = (uint32_t)st * (uint32_t)(C::STAGE >> 4);
          const uint32_t sf = tmem_base + C::SF_COL0 + (uint32_t)(it & 1) * 64;
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            gp_cp_sf(sf + kb * 4, sf_lo + off + (C::OFF_SFA >> 4) + kb * (TC_SF_ATOM >> 4), sf_hi);
#pragma unroll
            for (int j = 0; j < C::ATOMS; ++j)
              gp_cp_sf(sf + 16 + kb * 8 + j * 4, sf_lo + off + (C::OFF_SFB >> 4) + (j * 4 + kb) * (TC_SF_ATOM >> 4), sf_hi);
          }
#pragma unroll
          for (int kb = 0; kb < 4; ++kb)
            gp_mma(acc, op_lo + off + kb * 2, op_lo + off + (C::OFF_B >> 4) + kb * 2, op_hi, idesc, sf + kb * 4,
                   sf + 16 + kb * 8 + sfb_off, kt > k0 || kb ? 1u : 0u);
          gp_commit(empty(st), both);
          if (++st == STAGES) st = 0, ph ^= 1u;
        }
        if (ok) gp_commit(acc_full(buf), both);
        if (++ct == p.c_tiles) ct = 0;
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    pdl_wait();
    const int quad = warp & 3, half = (warp - 2) >> 2;
    constexpr int CHUNKS = C::COLS_WARP / C::CH, TPC = C::CH / J;    // a chunk's tokens: 8 or 16
    float* tr = reinterpret_cast<float*>(turn + (warp - 2) * GP_TR_BYTES);
    float* rs_s = tr + 16 * GP_TR_STRIDE;
    float* sum = reinterpret_cast<float*>(smem);    // parts: [token][128 rows] of this CTA's, in the ring, which is through by then
    const float ts = *p.tscale;
    const uint32_t even_empty = gp_map(acc_empty(0), even);
    const int tile_end = half < C::HALVES ? tile1 : tile0;
    for (int tile = tile0; tile < tile_end; ++tile) {
      const int n = tile - tile0, buf = n & 1, rt = tile / p.c_tiles, ct = tile % p.c_tiles;
      const int n0 = (rt * 2 + rank) * GP_ROWS + quad * 32;          // this warp's rows, columns and tokens
      const int col0 = ct * BN + half * C::COLS_WARP, tok0 = col0 / J;
      // what the values need besides the accumulator, requested before it is waited for: column scales (a lane a column), and
      // the residuals as they will leave (vectors of 8 rows)
      float rs[CHUNKS];
      uint32_t res[CHUNKS][TPC / 2];
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        const int col = col0 + c * C::CH + lane;
        rs[c] = lane < C::CH && col < p.cols ? __ldcg(p.rs + col) : 0.f;
        if (!SPLIT) {
          if (V == 8) gp_piece_residual<8, TPC>(p, tok0 + c * TPC, n0, lane, res[c]);
          else if (p.vec == 4) gp_piece_residual<4, TPC>(p, tok0 + c * TPC, n0, lane, res[c]);
          else gp_piece_residual<1, TPC>(p, tok0 + c * TPC, n0, lane, res[c]);
        }
      }
      // (the warps of a group do not meet: each has its own barrier phase and its own piece of shared memory)
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full(buf), (uint32_t)(n >> 1) & 1u, abort_flag))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN + half * C::COLS_WARP);
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        uint32_t r[32];
        if (C::CH == 32) tc_ld32(taddr + (uint32_t)(c * 32), r); else tc_ld16(taddr + (uint32_t)(c * 16), r);
        rs_s[lane] = rs[c];
        __syncwarp();
        tc_wait_ld();
        if (c == CHUNKS - 1) {                       // read out: the accumulator goes back
          tc_fence_before();
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(even_empty + 8u * buf) : "memory");
        }
#pragma unroll
        for (int t = 0; t < TPC; ++t) {
          // a token's terms: two in their order, as the one-SM kernel adds them (whole tiles: the same bits), four the smallest first
          float a = 0.f;
#pragma unroll
          for (int i = 0; i < J; ++i) {
            const int j = J == 4 ? J - 1 - i : i;
            a = fmaf(__uint_as_float(r[t * J + j]), rs_s[t * J + j], a);
          }
          if (SPLIT || J == 4) a *= ts;
          if (SPLIT) sum[(size_t)(half * (C::COLS_WARP / J) + c * TPC + t) * GP_ROWS + quad * 32 + lane] = a;
          else tr[t * GP_TR_STRIDE + lane] = a;
        }
        __syncwarp();
        if (!SPLIT) {
          const float s = J == 4 ? 1.f : ts;
          if (V == 8) gp_piece_store<8, TPC>(p, tok0 + c * TPC, n0, lane, tr, s, res[c]);
          else if (p.vec == 4) gp_piece_store<4, TPC>(p, tok0 + c * TPC, n0, lane, tr, s, res[c]);
          else gp_piece_store<1, TPC>(p, tok0 + c * TPC, n0, lane, tr, s, res[c]);
          __syncwarp();
        }
      }
    }
  }

  if constexpr (SPLIT) {
    // each pair of the cluster sums its share of the tokens, in the order of the parts
    gp_cluster_sync();
    constexpr int TOKENS = BN / J;
    const int rt = tile0 / p.c_tiles, ct = tile0 % p.c_tiles, t0 = part * TOKENS / p.parts, t1 = (part + 1) * TOKENS / p.parts;
    for (int i = t0 * 16 + (int)threadIdx.x; i < t1 * 16; i += GP_THREADS) {
      const int t = i >> 4, r = (i & 15) * 8, tok = ct * TOKENS + t, row = (rt * 2 + rank) * GP_ROWS + r;
      if (tok >= p.tokens || row >= p.N) continue;
      const uint4 res = V == 8 ? gp_residual<8>(p, tok, row) : make_uint4(0u, 0u, 0u, 0u);
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      for (int q = 0; q < p.parts; ++q) {
        const uint32_t src = gp_map(smem_u32(smem) + (uint32_t)(t * GP_ROWS + r) * 4u, 2 * q + rank);
        const float4 a = gp_ld_cluster(src), b = gp_ld_cluster(src + 16);
        lo.x += a.x, lo.y += a.y, lo.z += a.z, lo.w += a.w;
        hi.x += b.x, hi.y += b.y, hi.z += b.z, hi.w += b.w;
      }
      if (V == 8) {
        gp_store8(p, tok, row, lo, hi, 1.f, res);
      } else if (p.vec == 4) {
        const uint4 a = gp_residual<4>(p, tok, row), b = gp_residual<4>(p, tok, row + 4);
        gp_store4(p, tok, row, lo, 1.f, make_uint2(a.x, a.y));
        if (row + 4 < p.N) gp_store4(p, tok, row + 4, hi, 1.f, make_uint2(b.x, b.y));
      } else {
        const float v[9] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w, 0.f};
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (row + e < p.N) gp_store1(p, tok, row + e, v[e], v[e + 1], 1.f, __uint_as_float(gp_residual<1>(p, tok, row + e).x << 16));
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before the CTAs' memory goes away
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
  }
  gp_cluster_sync();                                // nothing of the pair is in flight towards the other SM any more
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS) : "memory");
  gp_cluster_sync();                                // no CTA leaves while the other's half is being given back
}

typedef CUresult (*EncodeTiledFnP)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

bool gp_tensor(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
            CUtensorMapSwizzle swizzle) {
  static EncodeTiledFnP encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) return false;
    encode = (EncodeTiledFnP)fn;
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int J, bool SPLIT, int V>
int launch_pair(const CUtensorMap (&m)[4], const PairParams& p, int pairs, cudaStream_t stream) {
  auto kern = gemm_nvfp4_pair_kernel<BN, J, SPLIT, V>;
  static TrlPerDevice<bool> set;
  bool& configured = set.here();
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<BN, J>::SMEM) != cudaSuccess) return 3;
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs), cfg.blockDim = dim3(GP_THREADS), cfg.dynamicSmemBytes = PairCfg<BN, J>::SMEM, cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * p.parts, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = g_trl_use_pdl ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, m[0], m[1], m[2], m[3], p);
}

template <int BN, int J>
int launch_pair(const CUtensorMap (&m)[4], const PairParams& p, int pairs, cudaStream_t stream) {
  if (p.vec == 8) return p.parts > 1 ? launch_pair<BN, J, true, 8>(m, p, pairs, stream) : launch_pair<BN, J, false, 8>(m, p, pairs, stream);
  return p.parts > 1 ? launch_pair<BN, J, true, 0>(m, p, pairs, stream) : launch_pair<BN, J, false, 0>(m, p, pairs, stream);
}

template <int J>
int launch_pair(const CUtensorMap (&m)[4], const PairParams& p, int bn, int pairs, cudaStream_t stream) {
  switch (bn) {
    case 32: return launch_pair<32, J>(m, p, pairs, stream);
    case 64: return launch_pair<64, J>(m, p, pairs, stream);
    case 128: return launch_pair<128, J>(m, p, pairs, stream);
    default: return launch_pair<192, J>(m, p, pairs, stream);
  }
}

}  // namespace

int gemm_pair_clusters(int parts) {
  static TrlPerDevice<int> counts[4];
  if (parts < 1 || parts > 3) return 0;
  int& known = counts[parts].here();
  if (known == 0) {
    auto kern = gemm_nvfp4_pair_kernel<64, 2, true, 8>;
    constexpr int smem = PairCfg<64, 2>::SMEM;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * parts), cfg.blockDim = dim3(GP_THREADS), cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * parts, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known = n > 0 ? n : -1;
  }
  return known;
}

int gemm_pair_launch(const GemmPairArgs& a, int bn, cudaStream_t stream) {
  const int cols = a.tokens * a.J, nk = (a.K + 255) / 256, n_tiles = (a.N + GP_ROWS - 1) / GP_ROWS;
  CUtensorMap m[4];
  {
    const cuuint64_t rows = a.w_tiled ? (cuuint64_t)n_tiles * nk * GP_ROWS : (cuuint64_t)a.N, width = a.w_tiled ? GP_KT : (cuuint64_t)a.K / 2;
    const cuuint64_t dims[2] = {width, rows}, strides[1] = {width};
    const cuuint32_t box[2] = {GP_KT, GP_ROWS};
    if (!gp_tensor(&m[0], a.wq, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return (int)cudaErrorInvalidValue;
  }
  {
    const cuuint64_t dims[2] = {128, (cuuint64_t)n_tiles * nk * 16}, strides[1] = {128};
    const cuuint32_t box[2] = {128, 16};
    if (!gp_tensor(&m[1], a.sfw, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return (int)cudaErrorInvalidValue;
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)a.K / 2, (cuuint64_t)cols}, strides[1] = {(cuuint64_t)a.K / 2};
    const cuuint32_t box[2] = {GP_KT, (cuuint32_t)bn / 2};
    if (!gp_tensor(&m[2], a.xq, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return (int)cudaErrorInvalidValue;
  }
  {
    const cuuint64_t dims[3] = {128, (cuuint64_t)nk * 16, (cuuint64_t)(cols + 255) / 256 * 2}, strides[2] = {128, (cuuint64_t)nk * 2048};
    const cuuint32_t box[3] = {128, 16, (cuuint32_t)(bn > 128 ? 2 : 1)};
    if (!gp_tensor(&m[3], a.sfx, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return (int)cudaErrorInvalidValue;
  }
  PairParams p;
  p.tscale = a.tscale, p.rs = a.rs, p.residual = (const bf16*)a.residual, p.out = a.out;
  p.N = a.N, p.tokens = a.tokens, p.cols = cols, p.ldr = a.ldr, p.ldo = a.ldo;
  p.r_tiles = (n_tiles + 1) / 2, p.c_tiles = (cols + bn - 1) / bn, p.nk = nk, p.w_tiled = a.w_tiled, p.epi = a.epi, p.parts = a.parts, p.vec = a.vec;
  const long long tiles = (long long)p.r_tiles * p.c_tiles;
  const int pairs = a.parts > 1 ? (int)tiles * a.parts : (int)(tiles < a.pairs ? tiles : a.pairs);
  if (bn == 32 && p.c_tiles > 1) return (int)cudaErrorInvalidValue;      // (its scales would start on an odd column of TMEM)
  switch (a.J) {
    case 1: return launch_pair<1>(m, p, bn, pairs, stream);
    case 2: return launch_pair<2>(m, p, bn, pairs, stream);
    default: return launch_pair<4>(m, p, bn, pairs, stream);
  }
}
