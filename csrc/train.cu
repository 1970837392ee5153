// Elementwise and low-rank parts of a training step, in fp32: RMSNorm, SwiGLU, adapters, the attention block's norms, rotation,
// softmax and gate, cross-entropy, AdamW over many tensors, each with its gradient.
//
// As torch ops each of these was four to forty launches that pass over the rows once apiece, and a step waited for the host.  All
// are bound by memory: a kernel reads its rows once and keeps them in registers between the passes; norms, SwiGLU, gate, loss and AdamW
// move 16 bytes a lane, softmax, the attention's preparation and the outer products 4.  The adapters are bound by what their products read from shared memory.
// (The dense products beside them stay library GEMMs.)  Sums are in a fixed order; nothing is added with atomics.
//
// In the place of the reference's tape handlers and optimizer (src/tilerl/autograd.py:113-301, :466, :661) and its loss
// (tilerl_kernels/reference.py:1511-1603).
#include "common.cuh"

namespace {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + expf(-x)); }

// ---- RMSNorm: a block a row, up to 8192 values ---------------------------------------------------------------------
// kept (or null): a copy of the rows for the gradient, since the caller may write into x between the passes.
template <int RN_V>                                 // vectors a thread keeps
__global__ void __launch_bounds__(256) tr_rmsnorm_kernel(const float* x, const float* w, float* out, float* kept, int h, float eps) {
  __shared__ float red[32];
  const float* row = x + (size_t)blockIdx.x * h;
  float4 v[RN_V];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < RN_V; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c < h) v[i] = ld4(row + c), ss += dot4(v[i], v[i]);
  }
  const float r = 1.f / sqrtf(block_sum(ss, red) / (float)h + eps);
#pragma unroll
  for (int i = 0; i < RN_V; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c >= h) continue;
    if (kept) st4(kept + (size_t)blockIdx.x * h + c, v[i]);
    const float4 g = ld4(w + c);
    st4(out + (size_t)blockIdx.x * h + c, make_float4(v[i].x * r * g.x, v[i].y * r * g.y, v[i].z * r * g.z, v[i].w * r * g.w));
  }
}
template <int RN_V>
__global__ void __launch_bounds__(256) tr_rmsnorm_grad_kernel(const float* x, const float* w, const float* up, float* dx, int h, float eps) {
  __shared__ float red[32];
  const size_t at = (size_t)blockIdx.x * h;
  float4 v[RN_V], e[RN_V];
  float ss = 0.f, se = 0.f;
#pragma unroll
  for (int i = 0; i < RN_V; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c >= h) continue;
    const float4 g = ld4(w + c), u = ld4(up + at + c);
    v[i] = ld4(x + at + c), e[i] = make_float4(u.x * g.x, u.y * g.y, u.z * g.z, u.w * g.w);
    ss += dot4(v[i], v[i]), se += dot4(v[i], e[i]);
  }
  const float r = 1.f / sqrtf(block_sum(ss, red) / (float)h + eps);
  const float m = block_sum(se, red) / (float)h * r * r * r;
#pragma unroll
  for (int i = 0; i < RN_V; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c < h) st4(dx + at + c, make_float4(r * e[i].x - v[i].x * m, r * e[i].y - v[i].y * m, r * e[i].z - v[i].z * m, r * e[i].w - v[i].w * m));
  }
}

// ---- SwiGLU of interleaved (gate, up) pairs: four results a thread -------------------------------------------------
__global__ void __launch_bounds__(256) tr_swiglu_kernel(const float* gu, float* out, long n4) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const float4 a = ld4(gu + i * 8), b = ld4(gu + i * 8 + 4);
  st4(out + i * 4, make_float4(a.x * sigm(a.x) * a.y, a.z * sigm(a.z) * a.w, b.x * sigm(b.x) * b.y, b.z * sigm(b.z) * b.w));
}
__device__ __forceinline__ float2 swiglu_grad(float g, float u, float up) {
  const float s = sigm(g);
  return make_float2(up * u * s * (1.f + g * (1.f - s)), up * g * s);
}
__global__ void __launch_bounds__(256) tr_swiglu_grad_kernel(const float* gu, const float* up, float* d, long n4) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const float4 a = ld4(gu + i * 8), b = ld4(gu + i * 8 + 4), e = ld4(up + i * 4);
  const float2 p = swiglu_grad(a.x, a.y, e.x), q = swiglu_grad(a.z, a.w, e.y), r = swiglu_grad(b.x, b.y, e.z), s = swiglu_grad(b.z, b.w, e.w);
  st4(d + i * 8, make_float4(p.x, p.y, q.x, q.y)), st4(d + i * 8 + 4, make_float4(r.x, r.y, s.x, s.y));
}

// ---- adapters of rank up to 32 ---------------------------------------------------------------------------------------
// out [M, R] = scale * x [M, K] . A, A(k, r) = a[r][k] or (by_k) a[k][r].  Sixteen rows a block: four rows a warp, two groups of four
// warps that take every other 128 k and are added up at the end, the lanes share K; 16 ranks a block's y, their factors staged,
// rows and factors of a group's next 128 on their way meanwhile.  2048 x 6144 with 16 ranks: 100 us with the loads in the open, 45 with
// one group, 31 so; the rows take 8 to read, the products 5.4 at the rate of fp32 FMAs, their factors twice that from shared memory; 32 ranks 56.
constexpr int LR = 16, LR_T = 128, LR_S = LR_T + 4;
__global__ void __launch_bounds__(256) tr_lowrank_kernel(const float* x, const float* a, float* out, int M, int K, int R, int by_k, float scale) {
  __shared__ __align__(16) float s[2][2][LR][LR_S];
  const int group = threadIdx.x >> 7, tid = threadIdx.x & 127, lane = tid & 31, row0 = blockIdx.x * 16 + (tid >> 5) * 4, r0 = blockIdx.y * LR;
  // the factors this thread stages: by_k, 4 ranks of four k (R % 4 == 0), else 4 k of four ranks
  const int fr = by_k ? (tid & 3) * 4 : tid >> 5, fk = by_k ? tid >> 2 : lane * 4;
  float4 v[4], f[4];
  float acc[4][LR] = {};
  auto fetch = [&](int k0) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      v[m] = row0 + m < M && k0 + lane * 4 < K ? ld4(x + (size_t)(row0 + m) * K + k0 + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      const int k = by_k ? k0 + fk + 32 * m : k0 + fk, q = r0 + (by_k ? fr : fr + 4 * m);
      f[m] = q < R && k < K ? ld4(a + (by_k ? (size_t)k * R + q : (size_t)q * K + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (group * LR_T < K) fetch(group * LR_T);
  for (int k0 = group * LR_T, b = 0; k0 < K; k0 += 2 * LR_T, b ^= 1) {
    float4 now[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      now[m] = v[m];
      if (by_k) {
        float* d = &s[group][b][fr][fk + 32 * m];
        d[0] = f[m].x, d[LR_S] = f[m].y, d[2 * LR_S] = f[m].z, d[3 * LR_S] = f[m].w;
      } else {
        st4(&s[group][b][fr + 4 * m][fk], f[m]);
      }
    }
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");     // (the other half was read before the barrier of the tile before)
    if (k0 + 2 * LR_T < K) fetch(k0 + 2 * LR_T);
#pragma unroll
    for (int r = 0; r < LR; ++r) {
      const float4 w = ld4(&s[group][b][r][lane * 4]);
#pragma unroll
      for (int m = 0; m < 4; ++m) acc[m][r] += dot4(now[m], w);
    }
  }
  __syncthreads();
  float* other = &s[0][0][0][0];                    // the second group's sums: [16 rows][16 ranks]
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int r = 0; r < LR; ++r) {
      acc[m][r] = warp_sum(acc[m][r]);
      if (group == 1 && lane == r) other[((tid >> 5) * 4 + m) * LR + r] = acc[m][r];
    }
  __syncthreads();
  if (group == 1) return;
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int r = 0; r < LR; ++r)
      if (lane == r && row0 + m < M && r0 + r < R) out[(size_t)(row0 + m) * R + r0 + r] = (acc[m][r] + other[((tid >> 5) * 4 + m) * LR + r]) * scale;
}

// out [M, N] = base + scale * z [M, R] . b, b(r, n) = b[n][r] or (by_r) b[r][n]; base may be null, or bf16 (a dense product's result).
// A thread four columns (two from rank 32 on), their factors in registers, 16 rows a block, four of them on their way.  Measured
// against it and slower: eight rows on their way and 32 a block (29.6 us a call of a training step, 23.5 here), factors in shared memory.
constexpr int EX_ROWS = 16;
template <int R>
__global__ void __launch_bounds__(128) tr_expand_kernel(const float* base, const bf16* base16, const float* z, const float* b, float* out, int M, int N,
                                                        int by_r, float scale) {
  constexpr int W = R > 16 ? 2 : 4;
  __shared__ __align__(16) float s[EX_ROWS][R];
  const int n = (blockIdx.x * 128 + threadIdx.x) * W, m0 = blockIdx.y * EX_ROWS, rows = min(EX_ROWS, M - m0);
  for (int i = threadIdx.x; i < rows * R; i += 128) s[i / R][i % R] = z[(size_t)m0 * R + i];
  float f[W][R];
  if (!by_r) {
#pragma unroll
    for (int w = 0; w < W; ++w)
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 v = n < N ? ld4(b + (size_t)(n + w) * R + r) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[w][r] = v.x, f[w][r + 1] = v.y, f[w][r + 2] = v.z, f[w][r + 3] = v.w;
      }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (n < N && W == 4) v = ld4(b + (size_t)r * N + n);
      else if (n < N) v.x = b[(size_t)r * N + n], v.y = b[(size_t)r * N + n + 1];
      f[0][r] = v.x, f[1][r] = v.y;
      if (W == 4) f[2 % W][r] = v.z, f[3 % W][r] = v.w;
    }
  }
  __syncthreads();
  if (n >= N) return;
  for (int m = 0; m < rows; m += 4) {
    float y[4][W];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const size_t at = (size_t)(m0 + m + q) * N + n;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m + q < rows && base) {
        if (W == 4) v = ld4(base + at);
        else v.x = base[at], v.y = base[at + 1];
      } else if (m + q < rows && base16) {
        const uint2 u = W == 4 ? *reinterpret_cast<const uint2*>(base16 + at) : make_uint2(*reinterpret_cast<const uint32_t*>(base16 + at), 0u);
        const float2 lo = bf162_bits_to_f2(u.x), hi = bf162_bits_to_f2(u.y);
        v = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
      y[q][0] = v.x, y[q][1] = v.y;
      if (W == 4) y[q][2 % W] = v.z, y[q][3 % W] = v.w;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (m + q >= rows) break;
      float t[W] = {};
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 v = ld4(&s[m + q][r]);
#pragma unroll
        for (int w = 0; w < W; ++w)
          t[w] = fmaf(v.x, f[w][r], t[w]), t[w] = fmaf(v.y, f[w][r + 1], t[w]), t[w] = fmaf(v.z, f[w][r + 2], t[w]), t[w] = fmaf(v.w, f[w][r + 3], t[w]);
      }
#pragma unroll
      for (int w = 0; w < W; ++w) t[w] = fmaf(t[w], scale, y[q][w]);
      float* o = out + (size_t)(m0 + m + q) * N + n;
      if (W == 4) st4(o, make_float4(t[0], t[1], t[2 % W], t[3 % W]));
      else *reinterpret_cast<float2*>(o) = make_float2(t[0], t[1]);
    }
  }
}

// Gradients of the factors: part [blockIdx.y] of sum_m z[m][r] v[m][n], then the parts added up.
template <int R>
__global__ void __launch_bounds__(128) tr_outer_kernel(const float* v, const float* z, float* part, int M, int N, int rows) {
  __shared__ float s[32][R];
  const int n = blockIdx.x * 128 + threadIdx.x, lo = blockIdx.y * rows, hi = min(M, lo + rows);
  float acc[R] = {};
  for (int m0 = lo; m0 < hi; m0 += 32) {
    const int cnt = min(32, hi - m0);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt * R; i += 128) s[i / R][i % R] = z[(size_t)m0 * R + i];
    __syncthreads();
    if (n < N)
#pragma unroll 16
      for (int m = 0; m < cnt; ++m) {
        const float x = v[(size_t)(m0 + m) * N + n];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = fmaf(x, s[m][r], acc[r]);
      }
  }
  if (n < N)
#pragma unroll
    for (int r = 0; r < R; ++r) part[((size_t)blockIdx.y * R + r) * N + n] = acc[r];
}
__global__ void __launch_bounds__(256) tr_outer_sum_kernel(const float* part, float* out, int N, int R, int parts, int by_r, float scale) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= N * R) return;
  const int r = i / N, n = i % N;
  float t = 0.f;
  for (int p = 0; p < parts; ++p) t += part[(size_t)p * R * N + i];
  out[by_r ? (size_t)i : (size_t)n * R + r] = t * scale;
}

// ---- attention block --------------------------------------------------------------------------------------------------
struct AttnRows {
  const float *qkv, *qw, *kw, *cs, *sn;             // cs, sn: [positions, half], row (b % pos_rows) * T + t
  int B, T, nq, nkv, d, half, gated, pos_rows;
  float eps;
  __device__ int rows() const { return nq * d * (gated ? 2 : 1) + 2 * nkv * d; }
  __device__ int at(int h) const {                  // a q head's, then a k head's, then a v head's values in a row
    return h < nq ? h * d * (gated ? 2 : 1) : nq * d * (gated ? 2 : 1) + (h - nq) * d;
  }
};

// A warp a (token, head): norm and rotation of q and k, v as it is; out [B, heads, T, d], so that the products are plain batched ones
// with a group's query heads as rows.
template <int AR_V>                                 // values a lane
__global__ void __launch_bounds__(256) tr_attn_prep_kernel(const AttnRows a, float* q, float* k, float* v) {
  const int lane = threadIdx.x & 31, heads = a.nq + 2 * a.nkv;
  const long x = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (x >= (long)a.B * a.T * heads) return;
  const int h = (int)(x % heads), t = (int)(x / heads % a.T), b = (int)(x / heads / a.T);
  const float* src = a.qkv + ((size_t)b * a.T + t) * a.rows() + a.at(h);
  if (h >= a.nq + a.nkv) {
    for (int c = lane; c < a.d; c += 32) v[(((size_t)b * a.nkv + h - a.nq - a.nkv) * a.T + t) * a.d + c] = src[c];
    return;
  }
  const float* w = h < a.nq ? a.qw : a.kw;
  const float *cs = a.cs + ((size_t)(b % a.pos_rows) * a.T + t) * a.half, *sn = a.sn + ((size_t)(b % a.pos_rows) * a.T + t) * a.half;
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < AR_V; ++i) {
    const int c = lane + 32 * i;
    if (c < a.d) ss += src[c] * src[c];
  }
  const float r = 1.f / sqrtf(warp_sum(ss) / (float)a.d + a.eps);
  float* dst = h < a.nq ? q + (((size_t)b * a.nq + h) * a.T + t) * a.d : k + (((size_t)b * a.nkv + h - a.nq) * a.T + t) * a.d;
#pragma unroll
  for (int i = 0; i < AR_V; ++i) {
    const int c = lane + 32 * i;
    if (c >= a.d) continue;
    float y = src[c] * r * w[c];
    if (c < a.half) y = y * cs[c] - src[c + a.half] * r * w[c + a.half] * sn[c];
    else if (c < 2 * a.half) y = y * cs[c - a.half] + src[c - a.half] * r * w[c - a.half] * sn[c - a.half];
    dst[c] = y;
  }
}

// Its gradient into dqkv, the gate's beside it: dq, dk, dv, o by head as above, up [B, T, nq, d].
template <int AR_V>
__global__ void __launch_bounds__(256) tr_attn_prep_grad_kernel(const AttnRows a, const float* dq, const float* dk, const float* dv, const float* o,
                                                                const float* up, float* dqkv) {
  const int lane = threadIdx.x & 31, heads = a.nq + 2 * a.nkv;
  const long x = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (x >= (long)a.B * a.T * heads) return;
  const int h = (int)(x % heads), t = (int)(x / heads % a.T), b = (int)(x / heads / a.T);
  const size_t tok = (size_t)b * a.T + t, row = tok * a.rows();
  if (h >= a.nq + a.nkv) {
    const int hv = h - a.nq - a.nkv;
    for (int c = lane; c < a.d; c += 32) dqkv[row + a.at(h) + c] = dv[(((size_t)b * a.nkv + hv) * a.T + t) * a.d + c];
    return;
  }
  const float* src = a.qkv + row + a.at(h);
  const float* w = h < a.nq ? a.qw : a.kw;
  const float* g = h < a.nq ? dq + (((size_t)b * a.nq + h) * a.T + t) * a.d : dk + (((size_t)b * a.nkv + h - a.nq) * a.T + t) * a.d;
  const float *cs = a.cs + ((size_t)(b % a.pos_rows) * a.T + t) * a.half, *sn = a.sn + ((size_t)(b % a.pos_rows) * a.T + t) * a.half;
  float e[AR_V], v[AR_V], ss = 0.f, se = 0.f;
#pragma unroll
  for (int i = 0; i < AR_V; ++i) {
    const int c = lane + 32 * i;
    e[i] = v[i] = 0.f;
    if (c >= a.d) continue;
    v[i] = src[c];
    float y = g[c];
    if (c < a.half) y = y * cs[c] + g[c + a.half] * sn[c];
    else if (c < 2 * a.half) y = y * cs[c - a.half] - g[c - a.half] * sn[c - a.half];
    e[i] = y * w[c];
    ss += v[i] * v[i], se += v[i] * e[i];
  }
  const float r = 1.f / sqrtf(warp_sum(ss) / (float)a.d + a.eps), m = warp_sum(se) / (float)a.d * r * r * r;
  float* dst = dqkv + row + a.at(h);
#pragma unroll
  for (int i = 0; i < AR_V; ++i) {
    const int c = lane + 32 * i;
    if (c < a.d) dst[c] = r * e[i] - v[i] * m;
  }
  if (h < a.nq && a.gated)
    for (int c = lane; c < a.d; c += 32) {
      const float s = sigm(src[a.d + c]);
      dst[a.d + c] = up[(tok * a.nq + h) * a.d + c] * o[(((size_t)b * a.nq + h) * a.T + t) * a.d + c] * s * (1.f - s);
    }
}

// out = o * sigmoid(gate), or o: from [B, nq, T, d] to [B, T, nq, d], or (back) the other way; four values a thread.
__global__ void __launch_bounds__(256) tr_attn_gate_kernel(const float* o, const float* qkv, float* out, long n4, int T, int nq, int d, int rows, int gated,
                                                           int back) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const int c = (int)(i * 4 % d), h = (int)(i * 4 / d % nq);
  const long tok = i * 4 / d / nq, by_head = ((tok / T * nq + h) * T + tok % T) * d + c;
  const float4 v = ld4(o + (back ? i * 4 : by_head)), g = gated ? ld4(qkv + tok * rows + h * 2 * d + d + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  st4(out + (back ? by_head : i * 4), gated ? make_float4(v.x * sigm(g.x), v.y * sigm(g.y), v.z * sigm(g.z), v.w * sigm(g.w)) : v);
}

// Rows of scores [B, heads, T, S] in place: softmax(scale * s) over the keys whose position is not later.  A block a row, up to
// 4096 keys.
template <int SM_V>                                 // values a thread
__global__ void __launch_bounds__(256) tr_softmax_kernel(float* s, const long long* pos, int pos_rows, int heads, int T, float scale) {
  __shared__ float red[32];
  const long row = blockIdx.x;
  const int t = (int)(row % T), b = (int)(row / T / heads);
  const long long* p = pos + (size_t)(b % pos_rows) * T;
  const long long mine = p[t];
  float* x = s + row * T;
  float v[SM_V], m = -INFINITY;
#pragma unroll
  for (int i = 0; i < SM_V; ++i) {
    const int c = threadIdx.x + 256 * i;
    v[i] = c < T && p[c] <= mine ? x[c] * scale : -INFINITY;
    m = fmaxf(m, v[i]);
  }
  m = block_max(m, red);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < SM_V; ++i) v[i] = expf(v[i] - m), sum += v[i];
  const float inv = 1.f / block_sum(sum, red);
#pragma unroll
  for (int i = 0; i < SM_V; ++i) {
    const int c = threadIdx.x + 256 * i;
    if (c < T) x[c] = v[i] * inv;
  }
}
// Gradient of the scores, in place of that of the weights p: scale * p (dp - sum dp p).
template <int SM_V>
__global__ void __launch_bounds__(256) tr_softmax_grad_kernel(const float* p, float* dp, int T, float scale) {
  __shared__ float red[32];
  const long at = (long)blockIdx.x * T;
  float v[SM_V], e[SM_V], sum = 0.f;
#pragma unroll
  for (int i = 0; i < SM_V; ++i) {
    const int c = threadIdx.x + 256 * i;
    v[i] = c < T ? p[at + c] : 0.f, e[i] = c < T ? dp[at + c] : 0.f;
    sum = fmaf(v[i], e[i], sum);
  }
  sum = block_sum(sum, red);
#pragma unroll
  for (int i = 0; i < SM_V; ++i) {
    const int c = threadIdx.x + 256 * i;
    if (c < T) dp[at + c] = v[i] * (e[i] - sum) * scale;
  }
}

// ---- cross-entropy -------------------------------------------------------------------------------------------------------
// A row's largest value, sum of exponentials below it and log-sum-exp, [3, rows]; read once.  As torch for rows with infinities
// and NaN.
__global__ void __launch_bounds__(512) tr_lse_kernel(const float* lg, float* out, long V) {
  __shared__ float red[32];
  const float* x = lg + (size_t)blockIdx.x * V;
  float m = -INFINITY, s = 0.f;
  bool nan = false;
#pragma unroll 4
  for (long c = threadIdx.x * 4; c < V; c += 2048) {
    const float4 v = ld4(x + c);
    const float n = fmaxf(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)), m);
    nan |= v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
    if (n > m) s *= expf(m - n), m = n;
    if (fabsf(n) < INFINITY) s += expf(v.x - m) + expf(v.y - m) + expf(v.z - m) + expf(v.w - m);
  }
  const float all = block_max(m, red);
  s = block_sum(fabsf(m) < INFINITY ? s * expf(m - all) : 0.f, red);
  nan = __syncthreads_or(nan);
  if (threadIdx.x == 0) {
    if (nan || !(fabsf(all) < INFINITY)) s = NAN;
    out[blockIdx.x] = all, out[gridDim.x + blockIdx.x] = s;
    out[2 * gridDim.x + blockIdx.x] = nan ? NAN : fabsf(all) < INFINITY ? all + logf(s) : all;
  }
}
// grad = (exp(lg - max) / sum - [c == target]) * weight, in the forward pass: the caller may write into the logits before the other.  (Not exp(lg - lse): an lse of 20 is rounded to 1e-6, and so would
// every probability be.)
__global__ void __launch_bounds__(256) tr_ce_grad_kernel(const float* lg, const float* stats, const long long* target, const float* weight,
                                                         float* grad, long V) {
  const size_t at = (size_t)blockIdx.x * V;
  const float m = stats[blockIdx.x], inv = 1.f / stats[gridDim.x + blockIdx.x], w = weight[blockIdx.x];
  const long long t = target[blockIdx.x];
#pragma unroll 4
  for (long c = threadIdx.x * 4; c < V; c += 1024) {
    const float4 v = ld4(lg + at + c);
    float e[4] = {expf(v.x - m) * inv, expf(v.y - m) * inv, expf(v.z - m) * inv, expf(v.w - m) * inv};
    if (t >= c && t < c + 4) e[t - c] -= 1.f;
    st4(grad + at + c, make_float4(e[0] * w, e[1] * w, e[2] * w, e[3] * w));
  }
}

// x times *up; no pass over the values where that is 1, as it is for a loss that is differentiated itself.
__global__ void __launch_bounds__(256) tr_scale_by_kernel(float* x, const float* up, long n4) {
  const float u = *up;
  if (u == 1.f) return;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < n4; i += (long)gridDim.x * 256) {
    const float4 v = ld4(x + i * 4);
    st4(x + i * 4, make_float4(v.x * u, v.y * u, v.z * u, v.w * u));
  }
}

// ---- many tensors at a time -------------------------------------------------------------------------------------------------
// Tensors of a launch may be as unlike as a bias and an embedding: each has blocks by its own length, 2048 values a block.  (64 blocks a
// tensor whatever its length: AdamW of 248 320 x 1024 values 17.4 ms, of 5120 x 34 816 12.1; torch 4.1 and 2.9,
// here 1.04 and 0.74, seven passes over the values at 6.7 TB/s.)
constexpr int MT = 32;                              // tensors a launch
constexpr int MT_BLOCK = 2048;
struct Tensors {
  float *p[MT], *m[MT], *v[MT];
  const float* g[MT];
  long n[MT];
  float decay[MT], c1[MT], c2[MT];                  // 1 - lr * weight decay, bias corrections
  int first[MT + 1];                                // blocks before a tensor's
};
// This block's tensor and its first value; every vector of four in turn (the last one may be cut short).
template <typename F>
__device__ __forceinline__ void each_vector(const Tensors& t, F f) {
  int k = 0;
  while ((int)blockIdx.x >= t.first[k + 1]) ++k;
  const long at = (long)((int)blockIdx.x - t.first[k]) * MT_BLOCK;
#pragma unroll
  for (int i = 0; i < MT_BLOCK; i += 1024) {
    const long c = at + i + threadIdx.x * 4;
    if (c < t.n[k]) f(k, c, (int)(t.n[k] - c < 4 ? t.n[k] - c : 4));
  }
}
__device__ __forceinline__ float4 ld4(const float* p, int cnt) {
  return cnt == 4 ? ld4(p) : make_float4(p[0], cnt > 1 ? p[1] : 0.f, cnt > 2 ? p[2] : 0.f, 0.f);
}
__device__ __forceinline__ void st4(float* p, float4 v, int cnt) {
  if (cnt == 4) return st4(p, v);
  p[0] = v.x;
  if (cnt > 1) p[1] = v.y;
  if (cnt > 2) p[2] = v.z;
}
// b2m, b1m: 1 - beta as the caller's doubles round
__global__ void __launch_bounds__(256) tr_adamw_kernel(const __grid_constant__ Tensors t, float lr, float b1, float b1m, float b2, float b2m, float eps) {
  each_vector(t, [&](int k, long c, int cnt) {
    const float4 g = ld4(t.g[k] + c, cnt);
    float4 p = ld4(t.p[k] + c, cnt), m = ld4(t.m[k] + c, cnt), v = ld4(t.v[k] + c, cnt);
    const float decay = t.decay[k], c1 = t.c1[k], c2 = t.c2[k];
    auto one = [&](float& p, float& m, float& v, float g) {
      m = fmaf(g, b1m, m * b1), v = fmaf(g * g, b2m, v * b2);
      p = p * decay - lr * (m / c1) / (sqrtf(v / c2) + eps);
    };
    one(p.x, m.x, v.x, g.x), one(p.y, m.y, v.y, g.y), one(p.z, m.z, v.z, g.z), one(p.w, m.w, v.w, g.w);
    st4(t.m[k] + c, m, cnt), st4(t.v[k] + c, v, cnt), st4(t.p[k] + c, p, cnt);
  });
}
// Sums of squares in 64 bits: part [tensor][block]; added up by the caller.  Every tensor has the blocks of the longest.
__global__ void __launch_bounds__(256) tr_squares_kernel(const __grid_constant__ Tensors t, double* part) {
  __shared__ double red[256];
  const int k = blockIdx.y;
  const float* g = t.g[k];
  double s = 0.0;
#pragma unroll 4
  for (long c = ((long)blockIdx.x * 256 + threadIdx.x) * 4; c < t.n[k]; c += (long)gridDim.x * 1024) {
    const float4 v = ld4(g + c, (int)(t.n[k] - c < 4 ? t.n[k] - c : 4));
    s += (double)v.x * (double)v.x + (double)v.y * (double)v.y + ((double)v.z * (double)v.z + (double)v.w * (double)v.w);
  }
  red[threadIdx.x] = s;
  for (int o = 128; o > 0; o >>= 1) {
    __syncthreads();
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
  }
  if (threadIdx.x == 0) part[(long)k * gridDim.x + blockIdx.x] = red[0];
}
__global__ void __launch_bounds__(256) tr_scale_kernel(const __grid_constant__ Tensors t, float c) {
  each_vector(t, [&](int k, long at, int cnt) {
    const float4 v = ld4(t.p[k] + at, cnt);
    st4(t.p[k] + at, make_float4(v.x * c, v.y * c, v.z * c, v.w * c), cnt);
  });
}
// Blocks of a launch (0: too many), and each tensor's first.
int blocks_of(Tensors& t, int count) {
  long at = 0;
  for (int i = 0; i < MT; ++i) {
    t.first[i] = (int)at;
    if (i < count) at += (t.n[i] + MT_BLOCK - 1) / MT_BLOCK;
    if (at >= 1l << 31) return 0;
  }
  t.first[MT] = (int)at;
  return (int)at;
}

AttnRows rows_of(const void* qkv, const void* qw, const void* kw, const void* cs, const void* sn, int B, int T, int nq, int nkv, int d, int half,
                 int gated, int pos_rows, float eps) {
  return AttnRows{(const float*)qkv, (const float*)qw, (const float*)kw, (const float*)cs, (const float*)sn, B, T, nq, nkv, d, half, gated, pos_rows, eps};
}

}  // namespace

// Rows of h values (h % 4 == 0, up to 8192), 16-byte aligned; so are all buffers below.
TRL_API int trl_train_rmsnorm(const void* x, const void* w, void* out, void* kept, int rows, int h, float eps, void* stream) {
  if (h % 4 || h > 8192 || rows < 1) return (int)cudaErrorInvalidValue;
  (h <= 1024 ? tr_rmsnorm_kernel<1> : h <= 2048 ? tr_rmsnorm_kernel<2> : tr_rmsnorm_kernel<8>)<<<rows, 256, 0, (cudaStream_t)stream>>>((const float*)x, (const float*)w, (float*)out, (float*)kept, h, eps);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_rmsnorm_grad(const void* x, const void* w, const void* up, void* dx, int rows, int h, float eps, void* stream) {
  if (h % 4 || h > 8192 || rows < 1) return (int)cudaErrorInvalidValue;
  (h <= 1024 ? tr_rmsnorm_grad_kernel<1> : h <= 2048 ? tr_rmsnorm_grad_kernel<2> : tr_rmsnorm_grad_kernel<8>)<<<rows, 256, 0, (cudaStream_t)stream>>>((const float*)x, (const float*)w, (const float*)up, (float*)dx, h, eps);
  return (int)cudaGetLastError();
}
// n results (n % 4 == 0); up null: forward into out, else the gradient of gu.
TRL_API int trl_train_swiglu(const void* gu, const void* up, void* out, long n, void* stream) {
  if (n % 4 || n < 1) return (int)cudaErrorInvalidValue;
  const int grid = (int)((n / 4 + 255) / 256);
  if (up) tr_swiglu_grad_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)gu, (const float*)up, (float*)out, n / 4);
  else tr_swiglu_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)gu, (float*)out, n / 4);
  return (int)cudaGetLastError();
}

#define BY_RANK(CALL)                                   \
  switch (R) {                                          \
    case 4: { constexpr int RR = 4; CALL; break; }      \
    case 8: { constexpr int RR = 8; CALL; break; }      \
    case 16: { constexpr int RR = 16; CALL; break; }    \
    case 32: { constexpr int RR = 32; CALL; break; }    \
    default: return (int)cudaErrorInvalidValue;         \
  }
TRL_API int trl_train_lowrank(const void* x, const void* a, void* out, int M, int K, int R, int by_k, float scale, void* stream) {
  if (M < 1 || K < 4 || K % 4 || R < 4 || R % 4) return (int)cudaErrorInvalidValue;
  tr_lowrank_kernel<<<dim3((M + 15) / 16, (R + LR - 1) / LR), 256, 0, (cudaStream_t)stream>>>((const float*)x, (const float*)a, (float*)out, M, K, R, by_k, scale);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_expand(const void* base, int bf16_base, const void* z, const void* b, void* out, int M, int N, int R, int by_r, float scale, void* stream) {
  if (M < 1 || N < 4 || N % 4 || (M + EX_ROWS - 1) / EX_ROWS > 65535) return (int)cudaErrorInvalidValue;
  BY_RANK((tr_expand_kernel<RR><<<dim3((N / (RR > 16 ? 2 : 4) + 127) / 128, (M + EX_ROWS - 1) / EX_ROWS), 128, 0, (cudaStream_t)stream>>>(bf16_base ? nullptr : (const float*)base, bf16_base ? (const bf16*)base : nullptr, (const float*)z, (const float*)b,
                                                                                                        (float*)out, M, N, by_r, scale)))
  return (int)cudaGetLastError();
}
// part: at least trl_train_outer_parts(M, N) * R * N floats.
TRL_API int trl_train_outer_parts(int M, int N) {
  const int cols = (N + 127) / 128, want = (4 * 148 + cols - 1) / cols, most = (M + 63) / 64;
  return want < most ? want : most;
}
TRL_API int trl_train_outer(const void* v, const void* z, void* part, void* out, int M, int N, int R, int by_r, float scale, void* stream) {
  if (M < 1 || N < 1) return (int)cudaErrorInvalidValue;
  const int parts = trl_train_outer_parts(M, N), rows = (M + parts - 1) / parts;
  BY_RANK((tr_outer_kernel<RR><<<dim3((N + 127) / 128, parts), 128, 0, (cudaStream_t)stream>>>((const float*)v, (const float*)z, (float*)part, M, N, rows)))
  tr_outer_sum_kernel<<<(N * R + 255) / 256, 256, 0, (cudaStream_t)stream>>>((const float*)part, (float*)out, N, R, parts, by_r, scale);
  return (int)cudaGetLastError();
}

TRL_API int trl_train_attn_prep(const void* qkv, const void* qw, const void* kw, const void* cs, const void* sn, void* q, void* k, void* v, int B, int T, int nq,
                                int nkv, int d, int half, int gated, int pos_rows, float eps, void* stream) {
  if (d > 512 || 2 * half > d || B < 1 || T < 1) return (int)cudaErrorInvalidValue;
  const AttnRows a = rows_of(qkv, qw, kw, cs, sn, B, T, nq, nkv, d, half, gated, pos_rows, eps);
  auto kern = d <= 128 ? tr_attn_prep_kernel<4> : d <= 256 ? tr_attn_prep_kernel<8> : tr_attn_prep_kernel<16>;
  kern<<<(int)(((long)B * T * (nq + 2 * nkv) + 7) / 8), 256, 0, (cudaStream_t)stream>>>(a, (float*)q, (float*)k, (float*)v);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_attn_prep_grad(const void* qkv, const void* qw, const void* kw, const void* cs, const void* sn, const void* dq, const void* dk,
                                     const void* dv, const void* o, const void* up, void* dqkv, int B, int T, int nq, int nkv, int d, int half, int gated,
                                     int pos_rows, float eps, void* stream) {
  if (d > 512 || 2 * half > d || B < 1 || T < 1) return (int)cudaErrorInvalidValue;
  const AttnRows a = rows_of(qkv, qw, kw, cs, sn, B, T, nq, nkv, d, half, gated, pos_rows, eps);
  auto kern = d <= 128 ? tr_attn_prep_grad_kernel<4> : d <= 256 ? tr_attn_prep_grad_kernel<8> : tr_attn_prep_grad_kernel<16>;
  kern<<<(int)(((long)B * T * (nq + 2 * nkv) + 7) / 8), 256, 0, (cudaStream_t)stream>>>(
      a, (const float*)dq, (const float*)dk, (const float*)dv, (const float*)o, (const float*)up, (float*)dqkv);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_attn_gate(const void* o, const void* qkv, void* out, int B, int T, int nq, int d, int rows, int gated, int back, void* stream) {
  if (d % 4 || rows % 4 || B < 1 || T < 1) return (int)cudaErrorInvalidValue;
  const long n4 = (long)B * T * nq * d / 4;
  tr_attn_gate_kernel<<<(int)((n4 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const float*)o, (const float*)qkv, (float*)out, n4, T, nq, d, rows, gated, back);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_softmax(void* s, const void* pos, int pos_rows, int B, int heads, int T, float scale, void* stream) {
  if (T < 1 || T > 4096 || (long)B * heads * T >= 1l << 31) return (int)cudaErrorInvalidValue;
  auto kern = T <= 512 ? tr_softmax_kernel<2> : T <= 2048 ? tr_softmax_kernel<8> : tr_softmax_kernel<16>;
  kern<<<B * heads * T, 256, 0, (cudaStream_t)stream>>>((float*)s, (const long long*)pos, pos_rows, heads, T, scale);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_softmax_grad(const void* p, void* dp, long rows, int T, float scale, void* stream) {
  if (T < 1 || T > 4096 || rows < 1 || rows >= 1l << 31) return (int)cudaErrorInvalidValue;
  auto kern = T <= 512 ? tr_softmax_grad_kernel<2> : T <= 2048 ? tr_softmax_grad_kernel<8> : tr_softmax_grad_kernel<16>;
  kern<<<(int)rows, 256, 0, (cudaStream_t)stream>>>((const float*)p, (float*)dp, T, scale);
  return (int)cudaGetLastError();
}

TRL_API int trl_train_lse(const void* lg, void* stats, long rows, long V, void* stream) {
  if (rows < 1 || rows >= 1l << 31 || V < 4 || V % 4) return (int)cudaErrorInvalidValue;
  tr_lse_kernel<<<(int)rows, 512, 0, (cudaStream_t)stream>>>((const float*)lg, (float*)stats, V);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_ce_grad(const void* lg, const void* stats, const void* target, const void* weight, void* grad, long rows, long V, void* stream) {
  if (rows < 1 || rows >= 1l << 31 || V < 4 || V % 4) return (int)cudaErrorInvalidValue;
  tr_ce_grad_kernel<<<(int)rows, 256, 0, (cudaStream_t)stream>>>((const float*)lg, (const float*)stats, (const long long*)target, (const float*)weight,
                                                                (float*)grad, V);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_scale_by(void* x, const void* up, long n, void* stream) {
  if (n < 4 || n % 4) return (int)cudaErrorInvalidValue;
  const long blocks = (n / 4 + 1023) / 1024;
  tr_scale_by_kernel<<<(int)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>((float*)x, (const float*)up, n / 4);
  return (int)cudaGetLastError();
}

// Up to 32 tensors: tables of pointers and lengths on the host.
TRL_API int trl_train_adamw(void* const* p, void* const* m, void* const* v, const void* const* g, const long* n, const float* decay, const float* c1,
                            const float* c2, int count, float lr, float b1, float b1m, float b2, float b2m, float eps, void* stream) {
  if (count < 1 || count > MT) return (int)cudaErrorInvalidValue;
  Tensors t{};
  for (int i = 0; i < count; ++i)
    t.p[i] = (float*)p[i], t.m[i] = (float*)m[i], t.v[i] = (float*)v[i], t.g[i] = (const float*)g[i], t.n[i] = n[i], t.decay[i] = decay[i], t.c1[i] = c1[i],
    t.c2[i] = c2[i];
  const int blocks = blocks_of(t, count);
  if (blocks < 1) return (int)cudaErrorInvalidValue;
  tr_adamw_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(t, lr, b1, b1m, b2, b2m, eps);
  return (int)cudaGetLastError();
}
// Blocks a tensor for the longest of a launch's: part is [count, blocks] doubles.  16 up to 262 144 values, then one for every
// 16 384, up to 1184.  (16 whatever the length: clipping 5120 x 34 816 values 1921 us, 32 x 1024 x 6144 214; here
// 213 and 229.)
TRL_API int trl_train_squares_blocks(long n) { return (int)(n <= 16 * 16384 ? 16 : n >= 1184l * 16384 ? 1184 : (n + 16383) / 16384); }
TRL_API int trl_train_squares(const void* const* g, const long* n, int count, int blocks, void* part, void* stream) {
  if (count < 1 || count > MT || blocks < 1) return (int)cudaErrorInvalidValue;
  Tensors t{};
  for (int i = 0; i < count; ++i) t.g[i] = (const float*)g[i], t.n[i] = n[i];
  tr_squares_kernel<<<dim3(blocks, count), 256, 0, (cudaStream_t)stream>>>(t, (double*)part);
  return (int)cudaGetLastError();
}
TRL_API int trl_train_scale(void* const* p, const long* n, int count, float c, void* stream) {
  if (count < 1 || count > MT) return (int)cudaErrorInvalidValue;
  Tensors t{};
  for (int i = 0; i < count; ++i) t.p[i] = (float*)p[i], t.n[i] = n[i];
  const int blocks = blocks_of(t, count);
  if (blocks < 1) return (int)cudaErrorInvalidValue;
  tr_scale_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(t, c);
  return (int)cudaGetLastError();
}
