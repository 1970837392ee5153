// Skinny (M <= 4 rows per pass) weight-streaming linears for the decode tick.
//
//   y[m, n] = epi( tscale * sum_k x'[m, k] * W[n, k] )
//
// * W is NVFP4 in the checkpoint layout: e2m1 nibbles [N, K/2] (low nibble = even
//   k), one e4m3 scale per 16 k [N, K/16], one fp32 tensor scale -- or bf16 [N, K].
// * x' = x, or RMSNorm(x) * norm_w when norm_w != nullptr: the norm is folded into
//   the prologue, every CTA recomputes it from the (L2-resident) activation row.
// * epi: plain store | + residual | SwiGLU on interleaved (gate, up) row pairs.
//
// The kernel is HBM-bound by construction: each warp owns R consecutive weight
// rows and walks K in 32-weight chunks with 128-bit streaming loads (R*U loads
// in flight per lane).  The activation lives in shared memory as f16, pre-scaled
// by a per-row power of two so that a 16-element block sum cannot overflow, in a
// chunk-interleaved layout that makes the four 16-byte reads per chunk
// bank-conflict free.  e2m1 -> f16x2 uses the native cvt; products accumulate in
// f16x2 within one 16-element scale block (exact products: 2-bit x 8-bit
// mantissas), then promote to fp32 with the block scale.
//
// Reference parity: `linear_fp4_gemv` / `linear_bf16_gemv` of
// packages/tilerl-kernels/src/tilerl_kernels/kernels_linear.py:924-1097.
#include <stdlib.h>

#include "common.cuh"

enum { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2, EPI_STORE_F32 = 3, EPI_PUSH = 4 };

namespace {

constexpr int GEMV_THREADS = 512;

// Stage x (bf16 [M, K], optional RMSNorm) into shared memory as scaled f16.
// Layout per row m: piece p (8 halves) of 32-element chunk c sits at
// ((p * nchunks + c) * 8) halves.  Returns nothing; xs_inv[m] = 1 / applied scale.
template <int M>
__device__ __forceinline__ void stage_x(const bf16* x, int ldx, int K,
                                        const float* __restrict__ norm_w, float eps,
                                        __half* xs, float* xs_inv, float* red) {
  const int nchunks = K >> 5;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const bf16* xr = x + (size_t)m * ldx;
    // one pass: sum of squares and max |x * w| together (the max of the normalised row is
    // rstd times the latter), one block reduction for both
    float rstd = 1.f;
    float ss = 0.f, amax = 0.f;
    for (int k = threadIdx.x * 2; k < K; k += blockDim.x * 2) {
      float2 v = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + k));
      ss += v.x * v.x + v.y * v.y;
      if (norm_w != nullptr) v.x *= norm_w[k], v.y *= norm_w[k + 1];
      amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
    }
    {
      const int lane_ = threadIdx.x & 31, w_ = threadIdx.x >> 5, nw_ = (blockDim.x + 31) >> 5;
      ss = warp_sum(ss);
      amax = warp_max(amax);
      __syncthreads();
      if (lane_ == 0) red[w_] = ss, red[32 + w_] = amax;
      __syncthreads();
      ss = warp_sum(lane_ < nw_ ? red[lane_] : 0.f);
      amax = warp_max(lane_ < nw_ ? red[32 + lane_] : 0.f);
    }
    if (norm_w != nullptr) {
      rstd = rsqrtf(ss / (float)K + eps);
      amax *= rstd * 1.01f;   // bf16 rounding of the normalised values can add < 0.4 %
    }
    // power-of-two scale s with amax * s <= 256: 16 products of |w| <= 6 stay < 65504
    int e = 0;
    if (amax > 0.f) {
      frexpf(amax, &e);  // amax = f * 2^e, f in [0.5, 1)
    }
    const float s = exp2f((float)(8 - e));
    if (threadIdx.x == 0) xs_inv[m] = exp2f((float)(e - 8));
    __half* dst = xs + (size_t)m * K;
    for (int k = threadIdx.x * 2; k < K; k += blockDim.x * 2) {
      float2 v = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + k));
      if (norm_w != nullptr) {
        v.x = __bfloat162float(__float2bfloat16(v.x * rstd * norm_w[k]));
        v.y = __bfloat162float(__float2bfloat16(v.y * rstd * norm_w[k + 1]));
      }
      const int c = k >> 5, p = (k >> 3) & 3, o = k & 7;
      *reinterpret_cast<__half2*>(dst + ((size_t)(p * nchunks + c) << 3) + o) =
          __floats2half2_rn(v.x * s, v.y * s);
    }
  }
  __syncthreads();
}

template <int M, int R, int EPI>
__global__ void __launch_bounds__(GEMV_THREADS, 1)
gemv_nvfp4_kernel(const bf16* x, int ldx, const uint8_t* __restrict__ wq,
                  const uint8_t* __restrict__ wscale, const float* __restrict__ tscale,
                  const float* __restrict__ norm_w, float eps, const bf16* residual,
                  int ldr, void* yout, int ldy, int N, int K, const TrlPushArgs push) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* xs = reinterpret_cast<__half*>(smem_raw);
  float* xs_inv = reinterpret_cast<float*>(smem_raw + (size_t)M * K * sizeof(__half));
  float* red = xs_inv + 8;
  // a pushing kernel lets the next kernel in only after its pushes (see allreduce_finish_kernel)
  pdl_enter();
  if (EPI != EPI_PUSH) pdl_trigger();
  pdl_wait();
  stage_x<M>(x, ldx, K, norm_w, eps, xs, xs_inv, red);

  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * (GEMV_THREADS / 32) + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * (GEMV_THREADS / 32);
  const int nchunks = K >> 5;
  const size_t row_bytes = (size_t)K >> 1, srow_bytes = (size_t)K >> 4;
  const float ts = *tscale;

  for (int r0 = warp * R; r0 < N; r0 += nwarps * R) {
    float acc[R][M];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
    const uint8_t* wrow[R];
    const uint8_t* srow[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int rr = min(r0 + r, N - 1);
      wrow[r] = wq + (size_t)rr * row_bytes;
      srow[r] = wscale + (size_t)rr * srow_bytes;
    }
    // D-deep register ring: while chunk c is consumed, the loads of the next D-1 chunks of
    // every row are in flight (the loop is bound by memory latency / D, not by latency)
    constexpr int D = (R * M <= 4) ? 4 : 2;
    uint4 wv[D][R];
    uint16_t sv[D][R];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int c = lane + 32 * d;
      if (c < nchunks) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          wv[d][r] = ldg_stream_16(wrow[r] + ((size_t)c << 4));
          sv[d][r] = ldg_stream_2(srow[r] + ((size_t)c << 1));
        }
      }
    }
    for (int base = lane; base < nchunks; base += 32 * D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int c = base + 32 * d;
        if (c < nchunks) {
#pragma unroll
          for (int m = 0; m < M; ++m) {
            uint32_t xh[16];
            const __half* xm = xs + (size_t)m * K;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              uint4 t = *reinterpret_cast<const uint4*>(xm + ((size_t)(p * nchunks + c) << 3));
              xh[p * 4 + 0] = t.x, xh[p * 4 + 1] = t.y, xh[p * 4 + 2] = t.z, xh[p * 4 + 3] = t.w;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float2 sc = h2_to_f2(cvt_e4m3x2_to_h2(sv[d][r]));
              const uint32_t w4[4] = {wv[d][r].x, wv[d][r].y, wv[d][r].z, wv[d][r].w};
#pragma unroll
              for (int blk = 0; blk < 2; ++blk) {
                uint32_t a = 0u;  // f16x2 zero
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                  uint32_t h[4];
                  cvt_e2m1x8_to_h2x4(w4[blk * 2 + q], h);
#pragma unroll
                  for (int i = 0; i < 4; ++i) a = hfma2_u(h[i], xh[(blk * 2 + q) * 4 + i], a);
                }
                const float2 af = h2_to_f2(a);
                acc[r][m] = fmaf(blk == 0 ? sc.x : sc.y, af.x + af.y, acc[r][m]);
              }
            }
          }
          const int cn = c + 32 * D;
          if (cn < nchunks) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              wv[d][r] = ldg_stream_16(wrow[r] + ((size_t)cn << 4));
              sv[d][r] = ldg_stream_2(srow[r] + ((size_t)cn << 1));
            }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = warp_sum(acc[r][m]) * ts * xs_inv[m];

    if (EPI == EPI_SWIGLU) {
      // rows (2j, 2j+1) = (gate_j, up_j); R is even and r0 is a multiple of R
      if (lane < (R / 2) * M) {
        const int j = lane / M, m = lane % M;
        float g = 0.f, u = 0.f;
#pragma unroll
        for (int r = 0; r < R; r += 2)
#pragma unroll
          for (int mm = 0; mm < M; ++mm)
            if (r / 2 == j && mm == m) g = acc[r][mm], u = acc[r + 1][mm];
        const int n = r0 + 2 * j;
        if (n + 1 < N)
          reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + (n >> 1)] = __float2bfloat16(silu_f(g) * u);
      }
    } else {
      if (lane < R * M) {
        const int r = lane / M, m = lane % M;
        float v = 0.f;
#pragma unroll
        for (int rr = 0; rr < R; ++rr)
#pragma unroll
          for (int mm = 0; mm < M; ++mm)
            if (rr == r && mm == m) v = acc[rr][mm];
        const int n = r0 + r;
        if (n < N) {
          if (EPI == EPI_PUSH) {
            // fp32 partial row straight into every rank's all-reduce slot (NVLink stores)
            // {value, epoch} in ONE 8-byte store per peer: the receiver polls the epoch half of
            // the word it needs, so no fence, counter or separate flag sits between the last
            // weight byte and the peer's sum
            const uint32_t epoch = *reinterpret_cast<const uint32_t*>(push.ws[push.rank]) + 1;
            const size_t off = 65536 + ((size_t)(((epoch & 1) * 8 + push.rank) * 8 + push.row0 + m) * push.hmax + n) * 8;
            const uint2 word = make_uint2(__float_as_uint(v), epoch);
            for (int p = 0; p < push.world; ++p) st_relaxed_sys_v2(push.ws[p] + off, word);
          } else {
            if (EPI == EPI_RESIDUAL) v += __bfloat162float(residual[(size_t)m * ldr + n]);
            if (EPI == EPI_STORE_F32)
              reinterpret_cast<float*>(yout)[(size_t)m * ldy + n] = v;
            else
              reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + n] = __float2bfloat16(v);
          }
        }
      }
    }
  }
  if (EPI == EPI_PUSH) pdl_trigger();
}

// Balanced variant.  A CTA owns a contiguous block of row PAIRS and its 16 warps split that
// block's (pair, 32-chunk step) units evenly, whatever the row count: a 5120-row projection
// on 148 x 16 warps no longer runs two rounds with the second almost empty.  A pair that is
// cut between warps is summed through shared-memory slots in a fixed order (bitwise
// reproducible); the epilogue then runs block-wide with coalesced stores.
__device__ __forceinline__ int sk_owner(int unit, int U, int W) {
  int w = (int)(((long long)unit * W) / U);
  while (w + 1 < W && (int)(((long long)(w + 1) * U) / W) <= unit) ++w;
  while (w > 0 && (int)(((long long)w * U) / W) > unit) --w;
  return w;
}

template <int M, int EPI>
__global__ void __launch_bounds__(GEMV_THREADS, 1)
gemv_nvfp4_sk_kernel(const bf16* x, int ldx, const uint8_t* __restrict__ wq,
                     const uint8_t* __restrict__ wscale, const float* __restrict__ tscale,
                     const float* __restrict__ norm_w, float eps, const bf16* residual,
                     int ldr, void* yout, int ldy, int N, int K, int nslot,
                     const TrlPushArgs push) {
  constexpr int W = GEMV_THREADS / 32;
  constexpr int D = 4;   // units in flight per lane: 4 x 2 rows x 16 B
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* xs = reinterpret_cast<__half*>(smem_raw);
  float* xs_inv = reinterpret_cast<float*>(smem_raw + (size_t)M * K * sizeof(__half));
  float* red = xs_inv + 8;
  float* slots = red + 64;   // [pairs_local][2 rows][nslot][M]
  pdl_enter();
  if (EPI != EPI_PUSH) pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npairs = N >> 1;
  const int p_lo = (int)(((long long)blockIdx.x * npairs) / gridDim.x);
  const int p_hi = (int)(((long long)(blockIdx.x + 1) * npairs) / gridDim.x);
  const int pl = p_hi - p_lo;
  for (int i = threadIdx.x; i < pl * 2 * nslot * M; i += GEMV_THREADS) slots[i] = 0.f;
  pdl_wait();
  stage_x<M>(x, ldx, K, norm_w, eps, xs, xs_inv, red);   // ends with a block barrier

  const int nchunks = K >> 5;
  const int nsteps = (nchunks + 31) >> 5;
  const size_t row_bytes = (size_t)K >> 1, srow_bytes = (size_t)K >> 4;
  const int U = pl * nsteps;
  const int u0 = (int)(((long long)warp * U) / W), u1 = (int)(((long long)(warp + 1) * U) / W);

  if (u0 < u1) {
    uint4 wv[D][2];
    uint16_t sv[D][2];
    // loader cursor
    // byte offsets from this CTA's first row (32-bit: a CTA's block is a few MB), advanced
    // incrementally: 32 chunks per step, two rows per pair
    int ls = u0 % nsteps;
    const uint8_t* wbase = wq + (size_t)p_lo * 2 * row_bytes;
    const uint8_t* sbase = wscale + (size_t)p_lo * 2 * srow_bytes;
    uint32_t woff = (uint32_t)(u0 / nsteps) * 2u * (uint32_t)row_bytes + (uint32_t)(ls * 32 + lane) * 16u;
    uint32_t soff = (uint32_t)(u0 / nsteps) * 2u * (uint32_t)srow_bytes + (uint32_t)(ls * 32 + lane) * 2u;
    const uint32_t wwrap = 2u * (uint32_t)row_bytes - (uint32_t)nsteps * 512u;
    const uint32_t swrap = 2u * (uint32_t)srow_bytes - (uint32_t)nsteps * 64u;
    auto load = [&](int d) {
      if (ls * 32 + lane < nchunks) {
        wv[d][0] = ldg_stream_16(wbase + woff);
        wv[d][1] = ldg_stream_16(wbase + woff + (uint32_t)row_bytes);
        sv[d][0] = ldg_stream_2(sbase + soff);
        sv[d][1] = ldg_stream_2(sbase + soff + (uint32_t)srow_bytes);
      }
      woff += 512u, soff += 64u;
      if (++ls == nsteps) ls = 0, woff += wwrap, soff += swrap;
    };
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (u0 + d < u1) load(d);
    // consumer cursor
    int cp = u0 / nsteps, cs = u0 % nsteps;
    float acc[2][M];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
    auto flush = [&](int pair_local) {
      // two-slot mode: slot 0 belongs to the warp that holds the pair's first unit
      const int slot = nslot == 2 ? (pair_local * nsteps >= u0 ? 0 : 1) : warp - sk_owner(pair_local * nsteps, U, W);
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const float v = warp_sum(acc[r][m]);
          if (lane == 0) slots[((size_t)(pair_local * 2 + r) * nslot + slot) * M + m] = v;
          acc[r][m] = 0.f;
        }
    };
    for (int ub = u0; ub < u1; ub += D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int uc = ub + d;
        if (uc < u1) {
          const int c = cs * 32 + lane;
          if (c < nchunks) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
              uint32_t xh[16];
              const __half* xm = xs + (size_t)m * K;
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                uint4 t = *reinterpret_cast<const uint4*>(xm + ((size_t)(p * nchunks + c) << 3));
                xh[p * 4 + 0] = t.x, xh[p * 4 + 1] = t.y, xh[p * 4 + 2] = t.z, xh[p * 4 + 3] = t.w;
              }
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const float2 sc = h2_to_f2(cvt_e4m3x2_to_h2(sv[d][r]));
                const uint32_t w4[4] = {wv[d][r].x, wv[d][r].y, wv[d][r].z, wv[d][r].w};
#pragma unroll
                for (int blk = 0; blk < 2; ++blk) {
                  uint32_t a = 0u;  // f16x2 zero
#pragma unroll
                  for (int q = 0; q < 2; ++q) {
                    uint32_t h[4];
                    cvt_e2m1x8_to_h2x4(w4[blk * 2 + q], h);
#pragma unroll
                    for (int i = 0; i < 4; ++i) a = hfma2_u(h[i], xh[(blk * 2 + q) * 4 + i], a);
                  }
                  const float2 af = h2_to_f2(a);
                  acc[r][m] = fmaf(blk == 0 ? sc.x : sc.y, af.x + af.y, acc[r][m]);
                }
              }
            }
          }
          if (uc + D < u1) load(d);
          if (++cs == nsteps) {
            flush(cp);
            cs = 0, ++cp;
          }
        }
      }
    }
    if (cs != 0) flush(cp);   // range ended inside a pair
  }
  __syncthreads();

  // block-wide epilogue over this CTA's rows
  const float ts = *tscale;
  if (EPI == EPI_SWIGLU) {
    for (int i = threadIdx.x; i < pl * M; i += GEMV_THREADS) {
      const int pr = i / M, m = i % M;
      float g = 0.f, u = 0.f;
      for (int sl = 0; sl < nslot; ++sl) {
        g += slots[((size_t)(pr * 2) * nslot + sl) * M + m];
        u += slots[((size_t)(pr * 2 + 1) * nslot + sl) * M + m];
      }
      const float sc = ts * xs_inv[m];
      const int n = (p_lo + pr) * 2;
      if (n + 1 < N)
        reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + (n >> 1)] = __float2bfloat16(silu_f(g * sc) * (u * sc));
    }
  } else {
    for (int i = threadIdx.x; i < pl * 2 * M; i += GEMV_THREADS) {
      const int rl = i / M, m = i % M;
      const int n = p_lo * 2 + rl;
      if (n >= N) continue;
      float v = 0.f;
      for (int sl = 0; sl < nslot; ++sl) v += slots[((size_t)rl * nslot + sl) * M + m];
      v *= ts * xs_inv[m];
      if (EPI == EPI_PUSH) {
        const uint32_t epoch = *reinterpret_cast<const uint32_t*>(push.ws[push.rank]) + 1;
        const size_t off = 65536 + ((size_t)(((epoch & 1) * 8 + push.rank) * 8 + push.row0 + m) * push.hmax + n) * 8;
        const uint2 word = make_uint2(__float_as_uint(v), epoch);
        for (int p = 0; p < push.world; ++p) st_relaxed_sys_v2(push.ws[p] + off, word);
      } else {
        if (EPI == EPI_RESIDUAL) v += __bfloat162float(residual[(size_t)m * ldr + n]);
        if (EPI == EPI_STORE_F32)
          reinterpret_cast<float*>(yout)[(size_t)m * ldy + n] = v;
        else
          reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + n] = __float2bfloat16(v);
      }
    }
  }
  if (EPI == EPI_PUSH) pdl_trigger();
}

// bf16 weights [N, K]: fp32 FMA, 8 weights per 16-byte load.  x staged as fp32.
template <int M, int R, int EPI>
__global__ void __launch_bounds__(GEMV_THREADS, 1)
gemv_bf16_kernel(const bf16* x, int ldx, const bf16* __restrict__ w,
                 const float* __restrict__ norm_w, float eps, const bf16* residual,
                 int ldr, void* yout, int ldy, int N, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* xs = reinterpret_cast<float*>(smem_raw);
  float* red = xs + (size_t)M * K;
  pdl_launch_dependents(6);
  pdl_wait();
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const bf16* xr = x + (size_t)m * ldx;
    float rstd = 1.f;
    if (norm_w != nullptr) {
      float ss = 0.f;
      for (int k = threadIdx.x; k < K; k += blockDim.x) {
        float v = __bfloat162float(xr[k]);
        ss += v * v;
      }
      ss = block_sum(ss, red);
      rstd = rsqrtf(ss / (float)K + eps);
    }
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      float v = __bfloat162float(xr[k]);
      if (norm_w != nullptr) v = __bfloat162float(__float2bfloat16(v * rstd * norm_w[k]));
      xs[(size_t)m * K + k] = v;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * (GEMV_THREADS / 32) + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * (GEMV_THREADS / 32);
  const int nvec = K >> 3;
  for (int r0 = warp * R; r0 < N; r0 += nwarps * R) {
    float acc[R][M];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
    for (int c = lane; c < nvec; c += 32) {
      uint4 wv[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
        wv[r] = ldg_stream_16(w + (size_t)min(r0 + r, N - 1) * K + ((size_t)c << 3));
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float4 x0 = *reinterpret_cast<const float4*>(xs + (size_t)m * K + (c << 3));
        const float4 x1 = *reinterpret_cast<const float4*>(xs + (size_t)m * K + (c << 3) + 4);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float2 a = bf162_bits_to_f2(wv[r].x), b = bf162_bits_to_f2(wv[r].y);
          float2 cc = bf162_bits_to_f2(wv[r].z), d = bf162_bits_to_f2(wv[r].w);
          float s = acc[r][m];
          s = fmaf(a.x, x0.x, s), s = fmaf(a.y, x0.y, s), s = fmaf(b.x, x0.z, s), s = fmaf(b.y, x0.w, s);
          s = fmaf(cc.x, x1.x, s), s = fmaf(cc.y, x1.y, s), s = fmaf(d.x, x1.z, s), s = fmaf(d.y, x1.w, s);
          acc[r][m] = s;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = warp_sum(acc[r][m]);
    if (lane < R * M) {
      const int r = lane / M, m = lane % M;
      float v = 0.f;
#pragma unroll
      for (int rr = 0; rr < R; ++rr)
#pragma unroll
        for (int mm = 0; mm < M; ++mm)
          if (rr == r && mm == m) v = acc[rr][mm];
      const int n = r0 + r;
      if (n < N) {
        if (EPI == EPI_RESIDUAL) v += __bfloat162float(residual[(size_t)m * ldr + n]);
        if (EPI == EPI_STORE_F32)
          reinterpret_cast<float*>(yout)[(size_t)m * ldy + n] = v;
        else
          reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + n] = __float2bfloat16(v);
      }
    }
  }
}

// bf16 weights [N, K] for 1..16 activation rows on the tensor cores (mma.sync m16n8k16, fp32 accumulation): the weight
// matrix is streamed once for all rows, which is what bounds the kernel.  KW of a block's 16 warps share the K of 16 weight
// rows, K / KW each, so that a head of a few thousand rows (small vocabularies, tensor-parallel slices) fills every SM.  With
// a warp per 16 whole rows, the split before this one, 15 520 rows were work for 61 of 148 SMs.  15 520 x 5120, launch included:
// 1 / 8 / 16 rows 48 / 90 / 152 us before, 40 / 41 / 56 here (16 rows: the activation rows' shared-memory reads show), inside a
// tick 40 / 69 / 194 before, 33 / 33 / 47 here; 128 256 x 4096: 192 / 229 / 283 before, 184 / 185 / 192 here.
// A warp needs its K range of the activation rows only: it loads, norms and keeps them as B fragments in its own part of shared
// memory, 16 bytes a lane and step, and the rows' square sums are all the block exchanges.  The weights of the next steps are
// in flight (registers, two sets) while those of this one are multiplied, across the block's reduction too.
//
// Lane (g, t) = (lane / 4, lane % 4) loads 16 bytes (8 consecutive k) of weight rows g and g + 8 per 32-wide step straight
// into A fragments.  A dot product does not care in which order k is summed, so the 8 loaded values serve two MMAs under a
// fixed permutation of k: fragment slots {2t, 2t+1, 2t+8, 2t+9} of the first MMA are elements 0..3 of the lane's chunk, of the
// second elements 4..7; the B fragment is the same chunk of activation row g, split the same way.  The 16 partial sums of an
// output are added in a fixed order.
constexpr int BR_WARPS = 16, BR_THREADS = BR_WARPS * 32;
template <int NT>
struct BrCfg {                                   // NT tiles of 8 activation rows
  static constexpr int RED_LD = NT * 128 + 1;    // floats of a warp's partial sums; odd: one bank apart from warp to warp
  static constexpr size_t red_bytes(int nbuf) { return (size_t)nbuf * BR_WARPS * RED_LD * sizeof(float); }
  static constexpr size_t x_bytes(int K, int kw) { return (size_t)BR_WARPS * ((K / 32 + kw - 1) / kw) * NT * 512; }
};
// BR_U: steps whose weight loads are in flight together (one set; 8 or 10 KB a warp with both)
template <int NT, int KW, int BR_U, int EPI>
__global__ void __launch_bounds__(BR_THREADS, 1)
gemv_bf16_rows_kernel(const bf16* x, int ldx, const bf16* __restrict__ w, const float* __restrict__ norm_w, float eps,
                      const bf16* residual, int ldr, void* yout, int ldy, int M, int N, int K, int nbuf, int aligned) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float ssp[BR_WARPS][NT * 8];
  constexpr int RED_LD = BrCfg<NT>::RED_LD;
  constexpr int RG = BR_WARPS / KW;              // groups of 16 rows a block works on at once
  const int steps = K >> 5, per = (steps + KW - 1) / KW;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint4* xs = reinterpret_cast<uint4*>(smem_raw) + (size_t)warp * per * NT * 32 + lane;      // [per][NT][32]
  float* red = reinterpret_cast<float*>(smem_raw + (size_t)BR_WARPS * per * NT * 512);        // [nbuf][warp][RED_LD]
  const int j0 = min((warp % KW) * per, steps), nj = min(per, steps - j0), j1 = max(1, j0 + nj);
  const int sub = (warp / KW) * 16;              // this warp's rows of a group
  const int groups = (N + RG * 16 - 1) / (RG * 16), chunks = max(1, (nj + BR_U - 1) / BR_U);
  pdl_launch_dependents(6);

  uint4 wa[2][BR_U], wb[2][BR_U];
  // chunk c of group gr into register set `set` (compile-time after unrolling)
  auto load = [&](uint4 (&a)[BR_U], uint4 (&b)[BR_U], int gr, int c) {
    const bf16* pa = w + (size_t)min(gr * (RG * 16) + sub + g, N - 1) * K + (t << 3);
    const bf16* pb = w + (size_t)min(gr * (RG * 16) + sub + g + 8, N - 1) * K + (t << 3);
#pragma unroll
    for (int u = 0; u < BR_U; ++u) {               // past the end: the last step again (its x is taken as zero below)
      const int j = min(j0 + c * BR_U + u, j1 - 1) << 5;
      a[u] = ldg_stream_16(pa + j), b[u] = ldg_stream_16(pb + j);
    }
  };
  int gr = blockIdx.x, c = 0;
  if (gr < groups) load(wa[0], wb[0], gr, 0);

  pdl_wait();                                      // (at once where the launch is not a programmatic one)
  {
    float ss[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) ss[i] = 0.f;
#pragma unroll 4
    for (int j = 0; j < nj; ++j) {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int m = i * 8 + g;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (m < M) {
          const bf16* xr = x + (size_t)m * ldx + ((size_t)(j0 + j) << 5) + (t << 3);
          if (aligned) {
            v = __ldcg(reinterpret_cast<const uint4*>(xr));
          } else {
            const unsigned short* h = reinterpret_cast<const unsigned short*>(xr);
            uint32_t e[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) e[k] = __ldcg(h + k);
            v = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
          }
        }
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = bf162_bits_to_f2(q[k]);
          ss[i] = fmaf(f.x, f.x, ss[i]), ss[i] = fmaf(f.y, f.y, ss[i]);
        }
        xs[(j * NT + i) * 32] = v;
      }
    }
    if (norm_w != nullptr) {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
        ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
        if (t == 0) ssp[warp][i * 8 + g] = ss[i];
      }
      __syncthreads();
      float rstd[NT];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < KW; ++k) v += ssp[(warp / KW) * KW + k][i * 8 + g];
        rstd[i] = rsqrtf(v / (float)K + eps);
      }
#pragma unroll 2
      for (int j = 0; j < nj; ++j) {
        float nw[8];
        const float* np = norm_w + ((size_t)(j0 + j) << 5) + (t << 3);
#pragma unroll
        for (int k = 0; k < 8; ++k) nw[k] = np[k];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const uint4 v = xs[(j * NT + i) * 32];
          const uint32_t q[4] = {v.x, v.y, v.z, v.w};
          uint32_t o[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 f = bf162_bits_to_f2(q[k]);
            o[k] = f2_to_bf162_bits(f.x * rstd[i] * nw[2 * k], f.y * rstd[i] * nw[2 * k + 1]);
          }
          xs[(j * NT + i) * 32] = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
  }

  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  int buf = 0;
  // one chunk: start the loads of the following one, multiply this one, and at the end of a group add up the block's sums
  auto chunk = [&](uint4 (&a)[BR_U], uint4 (&b)[BR_U], uint4 (&na)[BR_U], uint4 (&nb)[BR_U]) {
    const int cc = c, cg = gr;
    if (++c == chunks) c = 0, gr += gridDim.x;
    if (gr < groups) load(na, nb, gr, c);
#pragma unroll
    for (int u = 0; u < BR_U; ++u) {
      const int j = cc * BR_U + u;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        uint4 xv = xs[(min(j, max(nj, 1) - 1) * NT + i) * 32];
        if (j >= nj) xv = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(acc[i][0]), "+f"(acc[i][1]), "+f"(acc[i][2]), "+f"(acc[i][3])
                     : "r"(a[u].x), "r"(b[u].x), "r"(a[u].y), "r"(b[u].y), "r"(xv.x), "r"(xv.y));
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(acc[i][0]), "+f"(acc[i][1]), "+f"(acc[i][2]), "+f"(acc[i][3])
                     : "r"(a[u].z), "r"(b[u].z), "r"(a[u].w), "r"(b[u].w), "r"(xv.z), "r"(xv.w));
      }
    }
    if (cc + 1 < chunks) return;
    // accumulator of lane (g, t): weight rows g | g + 8, activation rows 2t | 2t + 1 of tile i
    float* rb = red + (size_t)buf * BR_WARPS * RED_LD;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) rb[warp * RED_LD + (i * 4 + e) * 32 + lane] = acc[i][e], acc[i][e] = 0.f;
    __syncthreads();
    constexpr int T = KW / (4 * NT) > 0 ? KW / (4 * NT) : 1;      // threads of an output
    constexpr int OPT = RG * 128 * NT * T / BR_THREADS;           // outputs of a thread
    static_assert(OPT >= 1 && OPT * BR_THREADS == RG * 128 * NT * T, "every partial sum is added once");
#pragma unroll
    for (int op = 0; op < OPT; ++op) {
      const int o = (threadIdx.x + op * BR_THREADS) / T, q = threadIdx.x % T;
      const int rg = o / (128 * NT), nl = o & 15, m = (o % (128 * NT)) >> 4, n = cg * (RG * 16) + rg * 16 + nl;
      const float* src = rb + rg * KW * RED_LD + ((m >> 3) * 4 + ((nl >> 3) << 1) + (m & 1)) * 32 + ((nl & 7) << 2) + ((m & 7) >> 1);
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < KW; k += T) v += src[(k + q) * RED_LD];
      if (T == 4) v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (T >= 2) v += __shfl_xor_sync(0xffffffffu, v, 1);
      if (q == 0 && n < N && m < M) {
        if (EPI == EPI_RESIDUAL) v += __bfloat162float(residual[(size_t)m * ldr + n]);
        if (EPI == EPI_STORE_F32)
          reinterpret_cast<float*>(yout)[(size_t)m * ldy + n] = v;
        else
          reinterpret_cast<bf16*>(yout)[(size_t)m * ldy + n] = __float2bfloat16(v);
      }
    }
    if (nbuf == 2) buf ^= 1;                       // the other buffer was last read before the barrier above
    else __syncthreads();
  };
  while (gr < groups) {                            // every warp of the block runs through the same groups; those with fewer
    chunk(wa[0], wb[0], wa[1], wb[1]);             // chunks than others (a short last range of K) only wait longer
    if (gr >= groups) break;
    chunk(wa[1], wb[1], wa[0], wb[0]);
  }
}

int g_num_sms = 0;
int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_num_sms;
}

template <int M, int R, int EPI>
cudaError_t launch_nvfp4(const bf16* x, int ldx, const uint8_t* wq, const uint8_t* ws, const float* ts,
                         const float* norm_w, float eps, const bf16* res, int ldr, void* y, int ldy,
                         int N, int K, cudaStream_t st, const TrlPushArgs& push) {
  const size_t smem = (size_t)M * K * sizeof(__half) + 8 * sizeof(float) + 64 * sizeof(float);
  auto kern = gemv_nvfp4_kernel<M, R, EPI>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    configured = true;
  }
  const int warps_needed = (N + R - 1) / R;
  int grid = min(num_sms(), (warps_needed + GEMV_THREADS / 32 - 1) / (GEMV_THREADS / 32));
  return trl_launch(kern, dim3(grid), dim3(GEMV_THREADS), smem, st, x, ldx, wq, ws, ts, norm_w, eps,
                    res, ldr, y, ldy, N, K, push);
}

template <int M, int EPI>
cudaError_t launch_nvfp4_sk(const bf16* x, int ldx, const uint8_t* wq, const uint8_t* ws, const float* ts,
                            const float* norm_w, float eps, const bf16* res, int ldr, void* y, int ldy,
                            int N, int K, cudaStream_t st, const TrlPushArgs& push) {
  constexpr int W = GEMV_THREADS / 32;
  if (N % 2 != 0) return cudaErrorInvalidValue;   // the older kernel handles odd row counts
  const int npairs = N / 2;
  const int grid = min(num_sms(), npairs);
  const int pl_max = (npairs + grid - 1) / grid;
  // a pair is shared by at most two warps once every CTA's warp share is at least one pair
  const int nslot = (npairs / grid) >= W ? 2 : W;
  const size_t smem = (size_t)M * K * sizeof(__half) + 8 * sizeof(float) + 64 * sizeof(float) +
                      (size_t)pl_max * 2 * nslot * M * sizeof(float);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  auto kern = gemv_nvfp4_sk_kernel<M, EPI>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    configured = true;
  }
  return trl_launch(kern, dim3(grid), dim3(GEMV_THREADS), smem, st, x, ldx, wq, ws, ts, norm_w, eps,
                    res, ldr, y, ldy, N, K, nslot, push);
}

template <int M, int EPI>
cudaError_t dispatch_r(const bf16* x, int ldx, const uint8_t* wq, const uint8_t* ws, const float* ts,
                       const float* norm_w, float eps, const bf16* res, int ldr, void* y, int ldy,
                       int N, int K, cudaStream_t st, const TrlPushArgs& push) {
  // The balanced kernel pays a block-wide epilogue; it wins where whole-row rounds leave warps
  // idle: rounds * R row-times against the ideal N / warps.
  static const char* mode = getenv("TRL_GEMV_BALANCED");   // "0" never, "1" always, unset: by shape
  const int all_warps = num_sms() * (GEMV_THREADS / 32);
  const int R0 = (M > 2 && N >= all_warps * 4 * 2) ? 4 : 2;
  const float ideal = (float)N / (float)all_warps;
  const float rounds = (float)(((N + R0 - 1) / R0 + all_warps - 1) / all_warps) * (float)R0;
  const bool balanced = mode ? (mode[0] == '1') : (ideal / rounds < 0.7f);
  if (balanced) {
    const cudaError_t e = launch_nvfp4_sk<M, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
    if (e != cudaErrorInvalidValue) return e;
  }
  // enough row blocks to give every warp of a full grid at least two -> R = 4
  const int full_warps = num_sms() * (GEMV_THREADS / 32);
  if (M > 2 && N >= full_warps * 4 * 2)
    return launch_nvfp4<M, 4, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
  return launch_nvfp4<M, 2, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
}

template <int EPI>
cudaError_t dispatch_m(int M, const bf16* x, int ldx, const uint8_t* wq, const uint8_t* ws,
                       const float* ts, const float* norm_w, float eps, const bf16* res, int ldr,
                       void* y, int ldy, int N, int K, cudaStream_t st, const TrlPushArgs& push = TrlPushArgs()) {
  switch (M) {
    case 1: return dispatch_r<1, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
    case 2: return dispatch_r<2, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
    case 3: return dispatch_r<3, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
    case 4: return dispatch_r<4, EPI>(x, ldx, wq, ws, ts, norm_w, eps, res, ldr, y, ldy, N, K, st, push);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

// y: bf16 (or fp32 for EPI_STORE_F32).  M up to 4 per pass; larger M is looped.
// K must be a multiple of 32 and M*K*2 bytes must fit in shared memory (<= ~190 KB).
TRL_API int trl_gemv_nvfp4(const void* x, int ldx, const void* wq, const void* wscale, const void* tscale,
                           const void* norm_w, float eps, const void* residual, int ldr, void* y, int ldy,
                           int M, int N, int K, int epi, void* stream) {
  if (K % 32 != 0 || N <= 0 || M <= 0) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t ysz = (epi == EPI_STORE_F32) ? 4 : 2;
  int per = 4;
  while (per > 1 && (size_t)per * K * 2 > 190 * 1024) --per;
  for (int m0 = 0; m0 < M; m0 += per) {
    const int mm = min(per, M - m0);
    const bf16* xp = (const bf16*)x + (size_t)m0 * ldx;
    const bf16* rp = residual ? (const bf16*)residual + (size_t)m0 * ldr : nullptr;
    void* yp = (char*)y + (size_t)m0 * ldy * ysz;
    cudaError_t e;
    switch (epi) {
      case EPI_STORE: e = dispatch_m<EPI_STORE>(mm, xp, ldx, (const uint8_t*)wq, (const uint8_t*)wscale, (const float*)tscale, (const float*)norm_w, eps, rp, ldr, yp, ldy, N, K, st); break;
      case EPI_RESIDUAL: e = dispatch_m<EPI_RESIDUAL>(mm, xp, ldx, (const uint8_t*)wq, (const uint8_t*)wscale, (const float*)tscale, (const float*)norm_w, eps, rp, ldr, yp, ldy, N, K, st); break;
      case EPI_SWIGLU: e = dispatch_m<EPI_SWIGLU>(mm, xp, ldx, (const uint8_t*)wq, (const uint8_t*)wscale, (const float*)tscale, (const float*)norm_w, eps, rp, ldr, yp, ldy, N, K, st); break;
      case EPI_STORE_F32: e = dispatch_m<EPI_STORE_F32>(mm, xp, ldx, (const uint8_t*)wq, (const uint8_t*)wscale, (const float*)tscale, (const float*)norm_w, eps, rp, ldr, yp, ldy, N, K, st); break;
      default: return (int)cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

// 1: trl_gemv_bf16 shares K between warps (up to 16 rows in one launch), 0: a warp for two whole rows, up to four a launch.
// The activation rows (8 or 16, as MMA tiles go) and one reduction buffer have to fit shared memory: K up to 13 824 with
// 8 rows, 6 656 with 16.
constexpr size_t BR_SMEM = 226 * 1024 - 512;
TRL_API int trl_gemv_bf16_one_pass(int M, int K) {
  if (M < 1 || M > 16 || K % 32 != 0 || K < 32) return 0;
  if (M == 1 && K < 2048) return 0;                // a short row for a warp of its own: 32 768 x 1024 22.6 us, 24.6 with K shared
  return (M <= 8 ? BrCfg<1>::x_bytes(K, BR_WARPS) + BrCfg<1>::red_bytes(1) : BrCfg<2>::x_bytes(K, BR_WARPS) + BrCfg<2>::red_bytes(1)) <= BR_SMEM;
}

TRL_API int trl_gemv_bf16(const void* x, int ldx, const void* w, const void* norm_w, float eps,
                          const void* residual, int ldr, void* y, int ldy, int M, int N, int K, int epi,
                          void* stream) {
  if (K % 8 != 0 || N <= 0 || M <= 0) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t ysz = (epi == EPI_STORE_F32) ? 4 : 2;
  if (trl_gemv_bf16_one_pass(M, K) && (epi == EPI_STORE || epi == EPI_STORE_F32 || epi == EPI_RESIDUAL)) {
    // up to 16 rows: one pass over the weights on the tensor cores
    const int nt = M <= 8 ? 1 : 2;
    // Warps that share K.  A barrier a group costs about as much as five steps of a warp, so K up to 2560 is shared by 8 and up
    // to 1280 by 4 (10 steps a warp at most) as long as there are two rounds of blocks; the
    // activation rows are then kept once for each group of rows, which fits at these K.  The set of loads is 4 or 5 steps,
    // whichever leaves less of the last one unused (128 256 x 4096, 16 rows: 192 us with 4, 235 with 5).
    int kw = BR_WARPS;
    while (kw > 4 && K / 32 <= 10 * (kw / 2) && (N + 15) / 16 >= 2 * num_sms() * (BR_WARPS / (kw / 2))) kw /= 2;
    const size_t xb = nt == 1 ? BrCfg<1>::x_bytes(K, kw) : BrCfg<2>::x_bytes(K, kw);
    int nbuf = 2;                                  // one reduction buffer (and a second barrier a group) where two do not fit
    size_t smem = xb + (nt == 1 ? BrCfg<1>::red_bytes(2) : BrCfg<2>::red_bytes(2));
    if (smem > BR_SMEM) nbuf = 1, smem = xb + (nt == 1 ? BrCfg<1>::red_bytes(1) : BrCfg<2>::red_bytes(1));
    const int rows = 16 * (BR_WARPS / kw), grid = min(num_sms(), (N + rows - 1) / rows);
    const int aligned = ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    cudaError_t e = cudaErrorInvalidValue;
    // Logits (fp32) are not a programmatic launch: loads in flight to registers need L1, and a block that comes to an SM while the kernel before
    // it leaves finds L1 as small as that kernel's shared memory made it.  In a decode tick, after projections with 228 KB of
    // shared memory, most blocks took 8 us a round of rows instead of 4.5: 15 520 x 5120, 1 or 8 rows, 62 us after the last
    // projection, 33 with the SMs empty first; 12 rows 45 to 68 from run to run (single slow SMs), 48 now; 16 rows 45.5, 47.5.
    // bf16 projections follow kernels of their own kind, which leave L1 as it should be, and keep the overlap.
    const int per = (K / 32 + kw - 1) / kw, u = (per + 3) / 4 * 4 < (per + 4) / 5 * 5 ? 4 : 5;
#define BR_CASE(NTT, KWW, U, EP)                                                                          \
  if (nt == NTT && kw == KWW && u == U && epi == EP) {                                                    \
    auto kern = gemv_bf16_rows_kernel<NTT, KWW, U, EP>;                                                    \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BR_SMEM);                \
    if (EP == EPI_STORE_F32) {                                                                            \
      kern<<<dim3(grid), dim3(BR_THREADS), smem, st>>>((const bf16*)x, ldx, (const bf16*)w,               \
          (const float*)norm_w, eps, (const bf16*)residual, ldr, y, ldy, M, N, K, nbuf, aligned);         \
      e = cudaGetLastError();                                                                             \
    } else {                                                                                              \
      e = trl_launch(kern, dim3(grid), dim3(BR_THREADS), smem, st, (const bf16*)x, ldx, (const bf16*)w,   \
                     (const float*)norm_w, eps, (const bf16*)residual, ldr, y, ldy, M, N, K, nbuf, aligned); \
    }                                                                                                     \
  }
#define BR_CASES(NTT, KWW)                                                                                          \
  BR_CASE(NTT, KWW, 4, EPI_STORE) BR_CASE(NTT, KWW, 4, EPI_STORE_F32) BR_CASE(NTT, KWW, 4, EPI_RESIDUAL)            \
  BR_CASE(NTT, KWW, 5, EPI_STORE) BR_CASE(NTT, KWW, 5, EPI_STORE_F32) BR_CASE(NTT, KWW, 5, EPI_RESIDUAL)
    BR_CASES(1, 4) BR_CASES(1, 8) BR_CASES(1, 16) BR_CASES(2, 4) BR_CASES(2, 8) BR_CASES(2, 16)
#undef BR_CASES
#undef BR_CASE
    return (int)e;
  }
  // one short row, rows too long for shared memory, K not a multiple of 32, more than 16 rows: fp32 FMA, up to four rows a pass
  int per = 4;
  while (per > 1 && (size_t)per * K * 4 > 190 * 1024) --per;
  for (int m0 = 0; m0 < M; m0 += per) {
    const int mm = min(per, M - m0);
    const bf16* xp = (const bf16*)x + (size_t)m0 * ldx;
    const bf16* rp = residual ? (const bf16*)residual + (size_t)m0 * ldr : nullptr;
    void* yp = (char*)y + (size_t)m0 * ldy * ysz;
    // at least half of an SM's shared memory: the blocks start while the kernel before them is still leaving (programmatic
    // launch), and without it the SMs that empty first take three or four of them and the last ones none (32 768 x 1024 in a
    // decode tick: 22.0 us after the last projection, 15.5 with one block an SM)
    const size_t smem = max((size_t)mm * K * 4 + 32 * 4, (size_t)116 * 1024);
    const int grid = min(num_sms(), (N / 2 + GEMV_THREADS / 32 - 1) / (GEMV_THREADS / 32) + 1);
    cudaError_t e = cudaErrorInvalidValue;
#define BF16_CASE(MM, EP)                                                                          \
  if (mm == MM && epi == EP) {                                                                     \
    auto kern = gemv_bf16_kernel<MM, 2, EP>;                                                       \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);           \
    e = trl_launch(kern, dim3(grid), dim3(GEMV_THREADS), smem, st, xp, ldx, (const bf16*)w,        \
                   (const float*)norm_w, eps, rp, ldr, yp, ldy, N, K);                             \
  }
    BF16_CASE(1, EPI_STORE) BF16_CASE(2, EPI_STORE) BF16_CASE(3, EPI_STORE) BF16_CASE(4, EPI_STORE)
    BF16_CASE(1, EPI_STORE_F32) BF16_CASE(2, EPI_STORE_F32) BF16_CASE(3, EPI_STORE_F32) BF16_CASE(4, EPI_STORE_F32)
    BF16_CASE(1, EPI_RESIDUAL) BF16_CASE(2, EPI_RESIDUAL) BF16_CASE(3, EPI_RESIDUAL) BF16_CASE(4, EPI_RESIDUAL)
#undef BF16_CASE
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

// Row-parallel GEMV whose epilogue pushes fp32 partial rows into every rank's one-shot
// all-reduce slot (see comm.cu); trl_allreduce_finish completes the sum on each rank.
TRL_API int trl_gemv_nvfp4_push(const void* x, int ldx, const void* wq, const void* wscale, const void* tscale,
                                void* const* ws, int rank, int world, int hmax, int M, int N, int K, void* stream) {
  if (K % 32 != 0 || N <= 0 || M <= 0 || M > 8 || N > hmax) return (int)cudaErrorInvalidValue;
  int per = 4;
  while (per > 1 && (size_t)per * K * 2 > 190 * 1024) --per;
  for (int m0 = 0; m0 < M; m0 += per) {
    const int mm = min(per, M - m0);
    TrlPushArgs push;
    for (int i = 0; i < 8; ++i) push.ws[i] = i < world ? (unsigned char*)ws[i] : nullptr;
    push.rank = rank, push.world = world, push.hmax = hmax, push.row0 = m0;
    const int last = (m0 + mm >= M) ? 1 : 0;
    cudaError_t e = dispatch_m<EPI_PUSH>(mm, (const bf16*)x + (size_t)m0 * ldx, ldx, (const uint8_t*)wq,
                                         (const uint8_t*)wscale, (const float*)tscale, nullptr, 0.f, nullptr, 0,
                                         nullptr, last, N, K, (cudaStream_t)stream, push);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
