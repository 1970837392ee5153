// Gated delta rule over whole sequences for training: forward, and its gradient, in fp32.
//
// The tape's op used to run the chunked form as torch ops and differentiate it with autograd: over a thousand launches of a few
// microseconds a layer and step, bound by the host.  Here a forward is four launches and a gradient eight.  Chunks of 32 tokens: the
// products within a chunk grow with its length, what goes from chunk to chunk is a [128, 128] state, and a warp has a lane a
// token for everything that is one number a token.  Per chunk, head, with S the state before it, G the running sum of the log
// decays, D_ij = exp(G_i - G_j):
//
//     A_ij = beta_i D_ij k_i.k_j (j < i)     T = (I + A)^-1      P_ij = D_ij q_i.k_j (j <= i)
//     U = T beta (V - e^G K S) = U0 - W S,   U0 = T beta V,  W = T beta e^G K
//     O = e^G Q S + P U                      S' = e^{G_last} S + Kd^T U,   Kd_j = exp(G_last - G_j) k_j
//
// and, with dS' the gradient of the state after it:
//
//     dU = P^T dO + Kd dS'       dR = T^T dU         dS = e^{G_last} dS' + (e^G Q)^T dO - W^T dU
//     dA = -dR U^T (j < i)       dP = dO U^T (j <= i)
//     dV = beta dR               dQ = e^G dO S^T + (dP D) K
//     dK = -beta e^G dR S^T + exp(G_last - G) U dS'^T + (M + M^T) K + (dP D)^T Q,   M = beta dA D
//     dG: every term's exponent collects term x gradient; dg is its sum from the token to the chunk's end.
//
// Kernels: prep (convolution, SiLU, norms, gates; a warp a head and token) -> chunks (A, T, P, U0, W: a block a chunk and head) ->
// scan (from chunk to chunk; a state's columns never mix, so four blocks a head have 32 each) -> norm.  Gradient: the same with states
// kept, then norm, scan backwards, everything of a chunk that needs both states (a block a chunk and head), and prep's gradient
// in two steps.  All fp32 on the CUDA cores, as the torch ops were; products go through shared memory in tiles of 4 x 4 or
// 2 x 4 a thread, rows padded by four floats.  Sums over heads and tokens are in a fixed order.
//
// In the place of the reference's tape handlers of the block (src/tilerl/autograd.py:113-301).
#include "common.cuh"

namespace {

constexpr int D = 128, C = 32;                     // head width, tokens a chunk
constexpr int LD = D + 4;                          // floats a padded row
constexpr int SLICE = 32, LS = SLICE + 4;          // state columns a block of the scans, padded
constexpr int LC = C + 1;

struct GdnTrain {
  const float *inp, *conv, *dt_bias, *a_log, *norm_w;
  int B, T, nk, nv, kw, n;                         // n: chunks a sequence
  float eps;
  // [sequence, head, chunk, token, 128] unless said otherwise; tokens past the end are zeros
  float *q, *k, *v;                                // q, k by key head: normed (q times 1 / sqrt(128))
  float *g, *beta;                                 // [sequence, value head, chunk, token]: log decays' running sum, gates
  float *w, *u0, *qg, *kd;                         // by value head
  float *p, *t;                                    // [.., 32, 32]
  float *o, *u, *s;                                // s: [sequence, value head, chunk, 128, 128], states before the chunks
};

__device__ __forceinline__ float silu(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float silu_grad(float x) {
  const float s = 1.f / (1.f + expf(-x));
  return s * (1.f + x * (1.f - s));
}
__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ void fma4(float4& d, float a, float4 b) {
  d.x = fmaf(a, b.x, d.x), d.y = fmaf(a, b.y, d.y), d.z = fmaf(a, b.z, d.z), d.w = fmaf(a, b.w, d.w);
}
__device__ __forceinline__ float4 mul4(float4 a, float b) { return make_float4(a.x * b, a.y * b, a.z * b, a.w * b); }

// A run of RUN tokens, a warp a head of 128 channels: taps and the window of rows stay in registers (a token alone read four taps of
// four channels again for each row: 74 us at 4 x 512 tokens of 16 heads).  Convolutions of up to four taps; longer ones reread.
constexpr int RUN = 8, TAPS = 4;
struct Conv {
  float4 tap[TAPS];                                 // of four channels: tap[j].x is channel c's
  __device__ __forceinline__ void load(const GdnTrain& a, int c) {
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
      const int at = j - (TAPS - a.kw);             // shorter ones: zeros in front
      tap[j] = at >= 0 && a.kw <= TAPS ? make_float4(a.conv[c * a.kw + at], a.conv[(c + 1) * a.kw + at], a.conv[(c + 2) * a.kw + at], a.conv[(c + 3) * a.kw + at])
                                       : f4(0.f);
    }
  }
};
__device__ __forceinline__ void fma44(float4& d, float4 a, float4 b) {
  d.x = fmaf(a.x, b.x, d.x), d.y = fmaf(a.y, b.y, d.y), d.z = fmaf(a.z, b.z, d.z), d.w = fmaf(a.w, b.w, d.w);
}
// Its four channels at tokens t0 .. t0 + RUN - 1 of a sequence (zeros before its beginning and from its end on).
__device__ __forceinline__ void conv_run(const GdnTrain& a, const float* seq, int ld, int t0, int c, float4 (&y)[RUN]) {
  Conv cv;
  cv.load(a, c);
  if (a.kw <= TAPS) {
    float4 x[RUN + TAPS - 1];
#pragma unroll
    for (int i = 0; i < RUN + TAPS - 1; ++i) {
      const int t = t0 + i - (TAPS - 1);
      x[i] = t >= 0 && t < a.T ? ld4(seq + (size_t)t * ld + c) : f4(0.f);
    }
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      y[i] = f4(0.f);
#pragma unroll
      for (int j = 0; j < TAPS; ++j) fma44(y[i], x[i + j], cv.tap[j]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < RUN; ++i) {
    y[i] = f4(0.f);
    for (int j = 0; j < a.kw; ++j) {
      const int t = t0 + i - (a.kw - 1) + j;
      if (t < 0 || t0 + i >= a.T) continue;
      fma44(y[i], ld4(seq + (size_t)t * ld + c), make_float4(a.conv[c * a.kw + j], a.conv[(c + 1) * a.kw + j], a.conv[(c + 2) * a.kw + j], a.conv[(c + 3) * a.kw + j]));
    }
  }
}

// ---- prep: a block a run of tokens (of the padded sequence) and eight heads ---------------------------------------------
__global__ void __launch_bounds__(256) gt_prep_kernel(const GdnTrain a) {
  const int lane = threadIdx.x & 31;
  const int runs = a.n * C / RUN, b = blockIdx.x / runs, t0 = blockIdx.x % runs * RUN, ck = t0 / C, i0 = t0 % C;
  const int ch = (2 * a.nk + a.nv) * D, ld = ch + a.nv * D + 2 * a.nv;
  const float* seq = a.inp + (size_t)b * a.T * ld;
  const int h = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (h < 2 * a.nk + a.nv) {
    float4 x[RUN];
    conv_run(a, seq, ld, t0, h * D + lane * 4, x);
    float* dst = h < a.nk ? a.q + ((size_t)(b * a.nk + h) * a.n + ck) * C * D
                 : h < 2 * a.nk ? a.k + ((size_t)(b * a.nk + h - a.nk) * a.n + ck) * C * D
                                : a.v + ((size_t)(b * a.nv + h - 2 * a.nk) * a.n + ck) * C * D;
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      x[i] = t0 + i < a.T ? make_float4(silu(x[i].x), silu(x[i].y), silu(x[i].z), silu(x[i].w)) : f4(0.f);
      if (h < 2 * a.nk) {
        const float inv = 1.f / sqrtf(warp_sum(dot4(x[i], x[i])) + 1e-12f);
        x[i] = mul4(x[i], h < a.nk ? inv * rsqrtf((float)D) : inv);
      }
      st4(dst + (i0 + i) * D + lane * 4, x[i]);
    }
  }
  if (blockIdx.y == 0)
    for (int e = threadIdx.x; e < a.nv * RUN; e += blockDim.x) {
      const int hv = e / RUN, i = e % RUN, t = t0 + i;
      float g = 0.f, be = 0.f;
      if (t < a.T) {
        const float* row = seq + (size_t)t * ld + ch + a.nv * D;
        const float x = row[hv] + a.dt_bias[hv];
        g = -expf(a.a_log[hv]) * (x > 20.f ? x : log1pf(expf(x)));
        be = 1.f / (1.f + expf(-row[a.nv + hv]));
      }
      const size_t at = ((size_t)(b * a.nv + hv) * a.n + ck) * C + i0 + i;
      a.g[at] = g, a.beta[at] = be;                // (the chunk kernel makes sums of the decays)
    }
}

// Rows 4 rg .. 4 rg + 3 against row `lane` of two padded [32, 128] tiles: acc[r] += x_r . y_lane
__device__ __forceinline__ void rows_dot(const float* x, const float* y, int rg, int lane, float (&acc)[4]) {
#pragma unroll 4
  for (int c = 0; c < D; c += 4) {
    const float4 v = ld4(y + lane * LD + c);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 u = ld4(x + (rg * 4 + r) * LD + c);
      acc[r] = fmaf(u.x, v.x, acc[r]), acc[r] = fmaf(u.y, v.y, acc[r]), acc[r] = fmaf(u.z, v.z, acc[r]), acc[r] = fmaf(u.w, v.w, acc[r]);
    }
  }
}
__device__ __forceinline__ void load_tile(float* dst, const float* src, int threads) {      // [32, 128], padded
  for (int x = threadIdx.x; x < C * D / 4; x += threads) st4(dst + (x >> 5) * LD + (x & 31) * 4, ld4(src + x * 4));
}

// ---- chunks: what does not need the state ------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gt_chunk_kernel(const GdnTrain a) {
  extern __shared__ __align__(16) float sm[];
  float *sk = sm, *sq = sk + C * LD, *sv = sq + C * LD, *sa = sv + C * LD, *st = sa + C * LC, *sg = st + C * LC, *sb = sg + C;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ck = blockIdx.x % a.n, bh = blockIdx.x / a.n, b = bh / a.nv, h = bh % a.nv, hk = h / (a.nv / a.nk);
  const size_t kc = ((size_t)(b * a.nk + hk) * a.n + ck) * C, vc = ((size_t)bh * a.n + ck) * C;
  load_tile(sk, a.k + kc * D, 256), load_tile(sq, a.q + kc * D, 256), load_tile(sv, a.v + vc * D, 256);
  if (warp == 0) {
    float g = a.g[vc + lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) g += up;
    }
    sg[lane] = g, sb[lane] = a.beta[vc + lane];
    a.g[vc + lane] = g;
  }
  __syncthreads();
  {
    float kk[4] = {}, qk[4] = {};
    rows_dot(sk, sk, warp, lane, kk);
    rows_dot(sq, sk, warp, lane, qk);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = warp * 4 + r;
      const float d = lane <= i ? expf(sg[i] - sg[lane]) : 0.f;
      sa[i * LC + lane] = lane < i ? sb[i] * d * kk[r] : 0.f;
      a.p[(vc + i) * C + lane] = d * qk[r];
    }
  }
  __syncthreads();
  if (warp == 0) {                                 // T by forward substitution: a lane a column
    float col[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
      float x0 = lane == i ? 1.f : 0.f, x1 = 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) {
        const float v = sa[i * LC + m];
        if (m & 1) x1 = fmaf(-v, col[m], x1); else x0 = fmaf(-v, col[m], x0);
      }
      col[i] = x0 + x1;
      st[i * LC + lane] = col[i];
    }
  }
  __syncthreads();
  for (int x = tid; x < C * C; x += 256) a.t[vc * C + x] = st[(x >> 5) * LC + (x & 31)];
  float4 w[4], u[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) w[r] = u[r] = f4(0.f);
  for (int m = 0; m < warp * 4 + 4; ++m) {         // T is lower triangular
    const float be = sb[m];
    const float4 kv = mul4(ld4(sk + m * LD + lane * 4), be * expf(sg[m])), vv = mul4(ld4(sv + m * LD + lane * 4), be);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float c = st[(warp * 4 + r) * LC + m];
      fma4(w[r], c, kv), fma4(u[r], c, vv);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = warp * 4 + r;
    const size_t at = (vc + i) * D + lane * 4;
    st4(a.w + at, w[r]), st4(a.u0 + at, u[r]);
    st4(a.qg + at, mul4(ld4(sq + i * LD + lane * 4), expf(sg[i])));
    st4(a.kd + at, mul4(ld4(sk + i * LD + lane * 4), expf(sg[C - 1] - sg[i])));
  }
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One chunk's operands of a scan: three [32, 128] tiles, one [32, 32] slice of rows of 128 and P.
struct ScanStage {
  float x[3][C * LD];
  float y[C * LS], p[C * LS];
};
__device__ __forceinline__ void scan_load(ScanStage& s, const float* x0, const float* x1, const float* x2, const float* y, const float* p,
                                          size_t row0, int c0) {
  for (int x = threadIdx.x; x < C * D / 4; x += 256) {
    const int r = x >> 5, c = (x & 31) * 4;
    const size_t at = (row0 + r) * D + c;
    cp16(&s.x[0][r * LD + c], x0 + at), cp16(&s.x[1][r * LD + c], x1 + at), cp16(&s.x[2][r * LD + c], x2 + at);
  }
  const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 4;
  cp16(&s.y[r * LS + c], y + (row0 + r) * D + c0 + c);
  cp16(&s.p[r * LS + c], p + (row0 + r) * C + c);
}

// ---- scan: blocks (sequence and head, slice of columns) ------------------------------------------------------------
// 2.2 us a chunk (W S and Q S 1.1, the state's update 0.5, P U 0.2), loads a chunk ahead.
__global__ void __launch_bounds__(256) gt_scan_kernel(const GdnTrain a, int keep) {
  extern __shared__ __align__(16) float sm[];
  ScanStage* stage = reinterpret_cast<ScanStage*>(sm);
  float *ss = reinterpret_cast<float*>(stage + 2), *su = ss + D * LS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bh = blockIdx.x, c0 = blockIdx.y * SLICE;
  const int cg = (lane & 7) * 4, rp = (lane >> 3) + 4 * warp;       // columns; a pair of rows, or four rows of the state
  for (int x = tid; x < D * LS; x += 256) ss[x] = 0.f;
  scan_load(stage[0], a.w, a.qg, a.kd, a.u0, a.p, (size_t)bh * a.n * C, c0);
  cp_commit();
  for (int ck = 0; ck < a.n; ++ck) {
    const size_t row0 = ((size_t)bh * a.n + ck) * C;
    if (ck + 1 < a.n) scan_load(stage[(ck + 1) & 1], a.w, a.qg, a.kd, a.u0, a.p, row0 + C, c0);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    const ScanStage& s = stage[ck & 1];
    const float decay = expf(a.g[row0 + C - 1]);
    if (keep)
      for (int x = tid; x < D * SLICE / 4; x += 256)
        st4(a.s + (((size_t)bh * a.n + ck) * D + (x >> 3)) * D + c0 + (x & 7) * 4, ld4(ss + (x >> 3) * LS + (x & 7) * 4));
    // rows 0..31: W S, 32..63: e^G Q S
    const int row = 2 * rp;
    const float* xr = row < C ? &s.x[0][row * LD] : &s.x[1][(row - C) * LD];
    float4 acc[2] = {f4(0.f), f4(0.f)};
#pragma unroll 4
    for (int k = 0; k < D; k += 4) {
      const float4 x0 = ld4(xr + k), x1 = ld4(xr + LD + k);
      const float4 s0 = ld4(ss + k * LS + cg), s1 = ld4(ss + (k + 1) * LS + cg), s2 = ld4(ss + (k + 2) * LS + cg), s3 = ld4(ss + (k + 3) * LS + cg);
      fma4(acc[0], x0.x, s0), fma4(acc[1], x1.x, s0), fma4(acc[0], x0.y, s1), fma4(acc[1], x1.y, s1);
      fma4(acc[0], x0.z, s2), fma4(acc[1], x1.z, s2), fma4(acc[0], x0.w, s3), fma4(acc[1], x1.w, s3);
    }
    if (row < C) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float4 u0 = ld4(s.y + (row + r) * LS + cg);
        const float4 u = make_float4(u0.x - acc[r].x, u0.y - acc[r].y, u0.z - acc[r].z, u0.w - acc[r].w);
        st4(su + (row + r) * LS + cg, u);
        if (keep) st4(a.u + (row0 + row + r) * D + c0 + cg, u);
      }
    }
    __syncthreads();
    if (row >= C) {
      const int i0 = row - C;
      for (int j = 0; j <= i0 + 1; ++j) {          // (P is zero above its diagonal)
        const float4 u = ld4(su + j * LS + cg);
        fma4(acc[0], s.p[i0 * LS + j], u), fma4(acc[1], s.p[(i0 + 1) * LS + j], u);
      }
      st4(a.o + (row0 + i0) * D + c0 + cg, acc[0]), st4(a.o + (row0 + i0 + 1) * D + c0 + cg, acc[1]);
    }
    float4 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = mul4(ld4(ss + (rp * 4 + r) * LS + cg), decay);
#pragma unroll 4
    for (int i = 0; i < C; ++i) {
      const float4 kd = ld4(&s.x[2][i * LD + rp * 4]), u = ld4(su + i * LS + cg);
      fma4(v[0], kd.x, u), fma4(v[1], kd.y, u), fma4(v[2], kd.z, u), fma4(v[3], kd.w, u);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) st4(ss + (rp * 4 + r) * LS + cg, v[r]);       // (read by its owner only since the barrier)
    __syncthreads();
  }
}

// ---- gated norm: a warp a (token, head) ------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gt_norm_kernel(const GdnTrain a, float* out) {
  const int lane = threadIdx.x & 31, x = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (x >= a.B * a.T * a.nv) return;
  const int h = x % a.nv, t = x / a.nv % a.T, b = x / a.nv / a.T;
  const int ch = (2 * a.nk + a.nv) * D, ld = ch + a.nv * D + 2 * a.nv;
  const float4 o = ld4(a.o + (((size_t)(b * a.nv + h) * a.n + t / C) * C + t % C) * D + lane * 4);
  const float4 z = ld4(a.inp + ((size_t)b * a.T + t) * ld + ch + h * D + lane * 4), w = ld4(a.norm_w + lane * 4);
  const float r = rsqrtf(warp_sum(dot4(o, o)) * (1.f / D) + a.eps);
  st4(out + (size_t)x * D + lane * 4, make_float4(o.x * r * w.x * silu(z.x), o.y * r * w.y * silu(z.y), o.z * r * w.z * silu(z.z), o.w * r * w.w * silu(z.w)));
}

// ---- gradients ---------------------------------------------------------------------------------------------------------
struct GdnTrainGrad {
  const float* dout;       // [B, T, nv, 128]
  float* dinp;             // [B, T, rows]
  float *d_o, *du, *ds;    // ds: gradients of the states after the chunks
  float *dq, *dk, *dv;     // by value head
  float *dg, *dbeta;       // [sequence, value head, chunk, token]
  float* dy;               // [B, T, channels]: gradient of the convolution
};

__global__ void __launch_bounds__(256) gt_norm_grad_kernel(const GdnTrain a, const GdnTrainGrad d) {
  const int lane = threadIdx.x & 31, x = blockIdx.x * 8 + (threadIdx.x >> 5), tp = a.n * C;
  if (x >= a.B * tp * a.nv) return;
  const int h = x % a.nv, t = x / a.nv % tp, b = x / a.nv / tp;
  const size_t at = (((size_t)(b * a.nv + h) * a.n + t / C) * C + t % C) * D + lane * 4;
  if (t >= a.T) {
    st4(d.d_o + at, f4(0.f));
    return;
  }
  const int ch = (2 * a.nk + a.nv) * D, ld = ch + a.nv * D + 2 * a.nv;
  const size_t zat = ((size_t)b * a.T + t) * ld + ch + h * D + lane * 4;
  const float4 o = ld4(a.o + at), z = ld4(a.inp + zat), w = ld4(a.norm_w + lane * 4);
  const float4 g = ld4(d.dout + (((size_t)b * a.T + t) * a.nv + h) * D + lane * 4);
  const float r = rsqrtf(warp_sum(dot4(o, o)) * (1.f / D) + a.eps);
  const float4 e = make_float4(g.x * w.x * silu(z.x), g.y * w.y * silu(z.y), g.z * w.z * silu(z.z), g.w * w.w * silu(z.w));
  const float m = warp_sum(dot4(o, e)) * (1.f / D) * r * r * r;
  st4(d.d_o + at, make_float4(r * e.x - o.x * m, r * e.y - o.y * m, r * e.z - o.z * m, r * e.w - o.w * m));
  st4(d.dinp + zat, make_float4(g.x * o.x * r * w.x * silu_grad(z.x), g.y * o.y * r * w.y * silu_grad(z.y),
                                g.z * o.z * r * w.z * silu_grad(z.z), g.w * o.w * r * w.w * silu_grad(z.w)));
}

// The scan backwards: dU, and the gradients of the states.
__global__ void __launch_bounds__(256) gt_scan_grad_kernel(const GdnTrain a, const GdnTrainGrad d) {
  extern __shared__ __align__(16) float sm[];
  ScanStage* stage = reinterpret_cast<ScanStage*>(sm);
  float *ss = reinterpret_cast<float*>(stage + 2), *su = ss + D * LS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bh = blockIdx.x, c0 = blockIdx.y * SLICE;
  const int cg = (lane & 7) * 4, rp = (lane >> 3) + 4 * warp;       // columns; a row of dU, or four rows of the state
  for (int x = tid; x < D * LS; x += 256) ss[x] = 0.f;
  scan_load(stage[(a.n - 1) & 1], a.w, a.qg, a.kd, d.d_o, a.p, ((size_t)bh * a.n + a.n - 1) * C, c0);
  cp_commit();
  for (int ck = a.n - 1; ck >= 0; --ck) {
    const size_t row0 = ((size_t)bh * a.n + ck) * C;
    if (ck > 0) scan_load(stage[(ck - 1) & 1], a.w, a.qg, a.kd, d.d_o, a.p, row0 - C, c0);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    const ScanStage& s = stage[ck & 1];
    const float decay = expf(a.g[row0 + C - 1]);
    for (int x = tid; x < D * SLICE / 4; x += 256)
      st4(d.ds + (((size_t)bh * a.n + ck) * D + (x >> 3)) * D + c0 + (x & 7) * 4, ld4(ss + (x >> 3) * LS + (x & 7) * 4));
    float4 acc = f4(0.f);
#pragma unroll 4
    for (int k = 0; k < D; k += 4) {
      const float4 x = ld4(&s.x[2][rp * LD + k]);
      fma4(acc, x.x, ld4(ss + k * LS + cg)), fma4(acc, x.y, ld4(ss + (k + 1) * LS + cg));
      fma4(acc, x.z, ld4(ss + (k + 2) * LS + cg)), fma4(acc, x.w, ld4(ss + (k + 3) * LS + cg));
    }
    for (int i = rp; i < C; ++i) fma4(acc, s.p[i * LS + rp], ld4(s.y + i * LS + cg));
    st4(su + rp * LS + cg, acc);
    st4(d.du + (row0 + rp) * D + c0 + cg, acc);
    __syncthreads();
    float4 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = mul4(ld4(ss + (rp * 4 + r) * LS + cg), decay);
#pragma unroll 4
    for (int i = 0; i < C; ++i) {
      const float4 q = ld4(&s.x[1][i * LD + rp * 4]), w = ld4(&s.x[0][i * LD + rp * 4]), o = ld4(s.y + i * LS + cg), u = ld4(su + i * LS + cg);
      fma4(v[0], q.x, o), fma4(v[1], q.y, o), fma4(v[2], q.z, o), fma4(v[3], q.w, o);
      fma4(v[0], -w.x, u), fma4(v[1], -w.y, u), fma4(v[2], -w.z, u), fma4(v[3], -w.w, u);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) st4(ss + (rp * 4 + r) * LS + cg, v[r]);
    __syncthreads();
  }
}

// Everything of a chunk and head that both of its states are known for.  24 warps: three products side by side, four rows a warp.
constexpr int GC_T = 768;
struct ChunkGradSmem {
  float k[C * LD], q[C * LD], d_o[C * LD], u[C * LD], dr[C * LD], s[C * LD], ds[C * LD];
  float t[C * LC], p[C * LC], kk[C * LC], pd[C * LC], m[C * LC], ef[C * LC], y[C * LC];
  float g[C], beta[C], eg[C], ed[C], rv[C], row_ef[C], row_db[C], qd[C], ky[C], wz[C], ss[GC_T / 32];
};
__global__ void __launch_bounds__(GC_T) gt_chunk_grad_kernel(const GdnTrain a, const GdnTrainGrad d) {
  extern __shared__ __align__(16) float smf[];
  ChunkGradSmem& sm = *reinterpret_cast<ChunkGradSmem*>(smf);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, prod = warp >> 3, rg = warp & 7;
  const int ck = blockIdx.x % a.n, bh = blockIdx.x / a.n, b = bh / a.nv, h = bh % a.nv, hk = h / (a.nv / a.nk);
  const size_t kc = ((size_t)(b * a.nk + hk) * a.n + ck) * C, vc = ((size_t)bh * a.n + ck) * C;
  load_tile(sm.k, a.k + kc * D, GC_T), load_tile(sm.q, a.q + kc * D, GC_T), load_tile(sm.d_o, d.d_o + vc * D, GC_T);
  load_tile(sm.u, a.u + vc * D, GC_T), load_tile(sm.s, d.du + vc * D, GC_T);
  for (int x = tid; x < C * C; x += GC_T) sm.t[(x >> 5) * LC + (x & 31)] = a.t[vc * C + x], sm.p[(x >> 5) * LC + (x & 31)] = a.p[vc * C + x];
  if (warp == 0) {
    const float g = a.g[vc + lane], last = __shfl_sync(0xffffffffu, g, C - 1);
    sm.g[lane] = g, sm.beta[lane] = a.beta[vc + lane], sm.eg[lane] = expf(g), sm.ed[lane] = expf(last - g);
  }
  __syncthreads();
  for (int i = warp; i < C; i += GC_T / 32) {      // dR = T^T dU, dV, and dR . V
    float4 r = f4(0.f);
    for (int m = i; m < C; ++m) fma4(r, sm.t[m * LC + i], ld4(sm.s + m * LD + lane * 4));
    st4(sm.dr + i * LD + lane * 4, r);
    st4(d.dv + (vc + i) * D + lane * 4, mul4(r, sm.beta[i]));
    const float x = warp_sum(dot4(r, ld4(a.v + (vc + i) * D + lane * 4)));
    if (lane == 0) sm.rv[i] = x;
  }
  __syncthreads();
  {
    float acc[4] = {};
    rows_dot(prod == 0 ? sm.k : prod == 1 ? sm.d_o : sm.dr, prod == 0 ? sm.k : sm.u, rg, lane, acc);
    float* dst = prod == 0 ? sm.kk : prod == 1 ? sm.pd : sm.m;
#pragma unroll
    for (int r = 0; r < 4; ++r) dst[(rg * 4 + r) * LC + lane] = acc[r];
  }
  __syncthreads();
  for (int i = warp; i < C; i += GC_T / 32) {
    const int at = i * LC + lane;
    const float dec = lane <= i ? expf(sm.g[i] - sm.g[lane]) : 0.f;
    const float dp = lane <= i ? sm.pd[at] : 0.f, da = lane < i ? -sm.m[at] : 0.f, kk = sm.kk[at];
    const float ef = dp * sm.p[at] + da * sm.beta[i] * dec * kk;
    sm.pd[at] = dp * dec, sm.m[at] = da * sm.beta[i] * dec, sm.ef[at] = ef;
    const float re = warp_sum(ef), rb = warp_sum(da * dec * kk);
    if (lane == 0) sm.row_ef[i] = re, sm.row_db[i] = rb;
  }
  float dot[4] = {}, both = 0.f;                   // this warp's rows: Q . (dO S^T), K . (dR S^T) or K . (U dS'^T); <S, dS'>
  for (int kq = 0; kq < D / C; ++kq) {
    __syncthreads();
    const size_t s0 = (((size_t)bh * a.n + ck) * D + kq * C) * D;
    for (int x = tid; x < C * D / 4; x += GC_T) {
      const float4 s = ld4(a.s + s0 + x * 4), e = ld4(d.ds + s0 + x * 4);
      st4(sm.s + (x >> 5) * LD + (x & 31) * 4, s), st4(sm.ds + (x >> 5) * LD + (x & 31) * 4, e);
      both += dot4(s, e);
    }
    __syncthreads();
    float acc[4] = {};
    rows_dot(prod == 0 ? sm.d_o : prod == 1 ? sm.dr : sm.u, prod == 2 ? sm.ds : sm.s, rg, lane, acc);
    const int col = kq * C + lane;
    if (prod == 0) {
#pragma unroll
      for (int r = 0; r < 4; ++r) dot[r] = fmaf(sm.q[(rg * 4 + r) * LD + col], acc[r], dot[r]), acc[r] *= sm.eg[rg * 4 + r];
      for (int j = 0; j < rg * 4 + 4; ++j) {
        const float k = sm.k[j * LD + col];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = fmaf(sm.pd[(rg * 4 + r) * LC + j], k, acc[r]);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) d.dq[(vc + rg * 4 + r) * D + col] = acc[r];
    } else if (prod == 1) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = rg * 4 + r;
        dot[r] = fmaf(sm.k[i * LD + col], acc[r], dot[r]), acc[r] *= -sm.beta[i] * sm.eg[i];
      }
      for (int j = 0; j < C; ++j) {
        const float k = sm.k[j * LD + col];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = fmaf(sm.m[(rg * 4 + r) * LC + j] + sm.m[j * LC + rg * 4 + r], k, acc[r]);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) sm.y[(rg * 4 + r) * LC + lane] = acc[r];
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = rg * 4 + r;
        acc[r] *= sm.ed[i], dot[r] = fmaf(sm.k[i * LD + col], acc[r], dot[r]);
      }
      for (int i = rg * 4; i < C; ++i) {
        const float q = sm.q[i * LD + col];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = fmaf(sm.pd[i * LC + rg * 4 + r], q, acc[r]);
      }
    }
    __syncthreads();
    if (prod == 2) {
#pragma unroll
      for (int r = 0; r < 4; ++r) d.dk[(vc + rg * 4 + r) * D + col] = acc[r] + sm.y[(rg * 4 + r) * LC + lane];
    }
  }
  float* dots = prod == 0 ? sm.qd : prod == 1 ? sm.ky : sm.wz;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float x = warp_sum(dot[r]);
    if (lane == 0) dots[rg * 4 + r] = x;
  }
  both = warp_sum(both);
  if (lane == 0) sm.ss[warp] = both;
  __syncthreads();
  if (warp == 0) {                                 // a lane a token
    float cols = 0.f;
    for (int i = lane; i < C; ++i) cols += sm.ef[i * LC + lane];
    const float w = sm.wz[lane], all_w = warp_sum(w), eg = sm.eg[lane], ky = sm.ky[lane];
    float dg = sm.row_ef[lane] - cols + eg * sm.qd[lane] - sm.beta[lane] * eg * ky - w;
    const float st = warp_sum(lane < GC_T / 32 ? sm.ss[lane] : 0.f);
    if (lane == C - 1) dg += all_w + eg * st;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float down = __shfl_down_sync(0xffffffffu, dg, o);
      if (lane + o < 32) dg += down;
    }
    d.dg[vc + lane] = dg;
    d.dbeta[vc + lane] = sm.rv[lane] - eg * ky + sm.row_db[lane];
  }
}

// Gradients of norms, SiLU and gates: a block a run of tokens and eight heads.
__global__ void __launch_bounds__(256) gt_prep_grad_kernel(const GdnTrain a, const GdnTrainGrad d) {
  const int lane = threadIdx.x & 31, rep = a.nv / a.nk;
  const int runs = a.n * C / RUN, b = blockIdx.x / runs, t0 = blockIdx.x % runs * RUN, ck = t0 / C, i0 = t0 % C;
  if (t0 >= a.T) return;
  const int ch = (2 * a.nk + a.nv) * D, ld = ch + a.nv * D + 2 * a.nv;
  const float* seq = a.inp + (size_t)b * a.T * ld;
  const int h = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (h < 2 * a.nk + a.nv) {
    float4 y[RUN];
    conv_run(a, seq, ld, t0, h * D + lane * 4, y);
    const bool is_v = h >= 2 * a.nk, is_q = h < a.nk;
    const int first = is_v ? h - 2 * a.nk : (is_q ? h : h - a.nk) * rep, heads = is_v ? 1 : rep;
    const float* src = (is_v ? d.dv : is_q ? d.dq : d.dk) + (((size_t)(b * a.nv + first) * a.n + ck) * C + i0) * D + lane * 4;
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      if (t0 + i >= a.T) break;
      float4 e = f4(0.f);
      for (int r = 0; r < heads; ++r) {
        const float4 x = ld4(src + ((size_t)r * a.n * C + i) * D);
        e.x += x.x, e.y += x.y, e.z += x.z, e.w += x.w;
      }
      if (!is_v) {
        const float4 c = make_float4(silu(y[i].x), silu(y[i].y), silu(y[i].z), silu(y[i].w));
        const float inv = 1.f / sqrtf(warp_sum(dot4(c, c)) + 1e-12f), sc = is_q ? inv * rsqrtf((float)D) : inv;
        const float m = warp_sum(dot4(c, e)) * inv * inv;
        e = make_float4(sc * (e.x - c.x * m), sc * (e.y - c.y * m), sc * (e.z - c.z * m), sc * (e.w - c.w * m));
      }
      st4(d.dy + ((size_t)b * a.T + t0 + i) * ch + h * D + lane * 4,
          make_float4(e.x * silu_grad(y[i].x), e.y * silu_grad(y[i].y), e.z * silu_grad(y[i].z), e.w * silu_grad(y[i].w)));
    }
  }
  if (blockIdx.y == 0)
    for (int e = threadIdx.x; e < a.nv * RUN; e += blockDim.x) {
      const int hv = e / RUN, i = e % RUN, t = t0 + i;
      if (t >= a.T) continue;
      const size_t at = ((size_t)(b * a.nv + hv) * a.n + ck) * C + i0 + i, row = ((size_t)b * a.T + t) * ld + ch + a.nv * D;
      const float x = a.inp[row + hv] + a.dt_bias[hv], be = a.beta[at];
      d.dinp[row + hv] = -d.dg[at] * expf(a.a_log[hv]) / (1.f + expf(-x));
      d.dinp[row + a.nv + hv] = d.dbeta[at] * be * (1.f - be);
    }
}

// The convolution backwards: a run of tokens and eight heads' channels a block.
__global__ void __launch_bounds__(256) gt_conv_grad_kernel(const GdnTrain a, const GdnTrainGrad d) {
  const int ch = (2 * a.nk + a.nv) * D, ld = ch + a.nv * D + 2 * a.nv;
  const int runs = (a.T + RUN - 1) / RUN, b = blockIdx.x / runs, t0 = blockIdx.x % runs * RUN, c = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (c >= ch) return;
  const float* dy = d.dy + (size_t)b * a.T * ch + c;
  float* dst = d.dinp + ((size_t)b * a.T + t0) * ld + c;
  Conv cv;
  cv.load(a, c);
  if (a.kw <= TAPS) {
    float4 y[RUN + TAPS - 1];
#pragma unroll
    for (int i = 0; i < RUN + TAPS - 1; ++i) y[i] = t0 + i < a.T ? ld4(dy + (size_t)(t0 + i) * ch) : f4(0.f);
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      if (t0 + i >= a.T) break;
      float4 e = f4(0.f);
#pragma unroll
      for (int j = 0; j < TAPS; ++j) fma44(e, y[i + TAPS - 1 - j], cv.tap[j]);
      st4(dst + (size_t)i * ld, e);
    }
    return;
  }
  for (int i = 0; i < RUN && t0 + i < a.T; ++i) {
    float4 e = f4(0.f);
    for (int j = 0; j < a.kw; ++j) {
      const int t = t0 + i + a.kw - 1 - j;
      if (t >= a.T) continue;
      fma44(e, ld4(dy + (size_t)t * ch), make_float4(a.conv[c * a.kw + j], a.conv[(c + 1) * a.kw + j], a.conv[(c + 2) * a.kw + j], a.conv[(c + 3) * a.kw + j]));
    }
    st4(dst + (size_t)i * ld, e);
  }
}

// Pieces of the workspace, in order; `grad`: those of a gradient too.  Returns the floats used.
long carve(GdnTrain& a, GdnTrainGrad* d, float* ws, bool grad) {
  long at = 0;
  auto take = [&](long n) {
    float* p = ws + at;
    at += n;
    return p;
  };
  const long kt = (long)a.B * a.nk * a.n * C, vt = (long)a.B * a.nv * a.n * C;
  a.q = take(kt * D), a.k = take(kt * D), a.v = take(vt * D), a.g = take(vt), a.beta = take(vt);
  a.w = take(vt * D), a.u0 = take(vt * D), a.qg = take(vt * D), a.kd = take(vt * D), a.p = take(vt * C), a.t = take(vt * C), a.o = take(vt * D);
  a.u = a.s = nullptr;
  if (grad) {
    a.u = take(vt * D), a.s = take(vt / C * D * D);
    d->d_o = take(vt * D), d->du = take(vt * D), d->ds = take(vt / C * D * D);
    d->dg = take(vt), d->dbeta = take(vt), d->dy = take((long)a.B * a.T * (2 * a.nk + a.nv) * D);
    d->dq = a.w, d->dk = a.qg, d->dv = a.u0;       // read for the last time before these are written
  }
  return at;
}

constexpr int CHUNK_SMEM = (3 * C * LD + 2 * C * LC + 2 * C) * 4;
constexpr int SCAN_SMEM = (int)(2 * sizeof(ScanStage)) + (D * LS + C * LS) * 4;

int shared_memory() {
  static TrlPerDevice<bool> set;
  bool& ok = set.here();
  if (!ok)
    ok = cudaFuncSetAttribute(gt_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHUNK_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(gt_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(gt_scan_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(gt_chunk_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkGradSmem)) == cudaSuccess;
  return ok ? 0 : 3;
}

bool fits(int B, int T, int nk, int nv, int kw) {
  return B > 0 && T > 0 && nk > 0 && nv > 0 && nv % nk == 0 && nv % 2 == 0 && kw > 0 && (long)B * ((T + C - 1) / C) * C * (nv + 2 * nk) < (1l << 31) / 4;
}

int run_forward(const GdnTrain& a, int keep, cudaStream_t st) {
  gt_prep_kernel<<<dim3(a.B * a.n * (C / RUN), (2 * a.nk + a.nv + 7) / 8), 256, 0, st>>>(a);
  gt_chunk_kernel<<<a.B * a.nv * a.n, 256, CHUNK_SMEM, st>>>(a);
  gt_scan_kernel<<<dim3(a.B * a.nv, D / SLICE), 256, SCAN_SMEM, st>>>(a, keep);
  return (int)cudaGetLastError();
}

}  // namespace

// Floats of workspace for B sequences of T tokens (forward, or forward and gradient).
TRL_API long trl_gdn_train_workspace(int B, int T, int nk, int nv, int grad) {
  GdnTrain a{};
  GdnTrainGrad d{};
  a.B = B, a.T = T, a.nk = nk, a.nv = nv, a.n = (T + C - 1) / C;
  return carve(a, &d, nullptr, grad != 0);
}

// out [B, T, nv * 128] = block(inp [B, T, (2 nk + 2 nv) * 128 + 2 nv]), zero state and history before each sequence; fp32, heads of
// 128, an even number of value heads (rows of whole 16-byte pieces), 16-byte aligned.
TRL_API int trl_gdn_train_forward(const void* inp, const void* conv, const void* dt_bias, const void* a_log, const void* norm_w, void* out,
                                  void* ws, int B, int T, int nk, int nv, int kw, float eps, void* stream) {
  if (!fits(B, T, nk, nv, kw)) return (int)cudaErrorInvalidValue;
  if (shared_memory()) return 3;
  GdnTrain a{(const float*)inp, (const float*)conv, (const float*)dt_bias, (const float*)a_log, (const float*)norm_w, B, T, nk, nv, kw, (T + C - 1) / C, eps};
  carve(a, nullptr, (float*)ws, false);
  cudaStream_t st = (cudaStream_t)stream;
  if (const int rc = run_forward(a, 0, st)) return rc;
  gt_norm_kernel<<<(B * T * nv + 7) / 8, 256, 0, st>>>(a, (float*)out);
  return (int)cudaGetLastError();
}

// dinp [B, T, rows]: gradient of inp for dout [B, T, nv * 128].  Left for the caller in the workspace, at the offsets written to
// `where` (floats): o, gradients of the log decays by token, gradients of the convolution's outputs.
TRL_API int trl_gdn_train_backward(const void* inp, const void* conv, const void* dt_bias, const void* a_log, const void* norm_w, const void* dout,
                                   void* dinp, void* ws, long* where, int B, int T, int nk, int nv, int kw, float eps, void* stream) {
  if (!fits(B, T, nk, nv, kw)) return (int)cudaErrorInvalidValue;
  if (shared_memory()) return 3;
  GdnTrain a{(const float*)inp, (const float*)conv, (const float*)dt_bias, (const float*)a_log, (const float*)norm_w, B, T, nk, nv, kw, (T + C - 1) / C, eps};
  GdnTrainGrad d{};
  carve(a, &d, (float*)ws, true);
  d.dout = (const float*)dout, d.dinp = (float*)dinp;
  cudaStream_t st = (cudaStream_t)stream;
  if (const int rc = run_forward(a, 1, st)) return rc;
  gt_norm_grad_kernel<<<(B * a.n * C * nv + 7) / 8, 256, 0, st>>>(a, d);
  gt_scan_grad_kernel<<<dim3(B * nv, D / SLICE), 256, SCAN_SMEM, st>>>(a, d);
  gt_chunk_grad_kernel<<<B * nv * a.n, GC_T, sizeof(ChunkGradSmem), st>>>(a, d);
  gt_prep_grad_kernel<<<dim3(B * a.n * (C / RUN), (2 * nk + nv + 7) / 8), 256, 0, st>>>(a, d);
  gt_conv_grad_kernel<<<dim3(B * ((T + RUN - 1) / RUN), ((2 * nk + nv) * D / 4 + 255) / 256), 256, 0, st>>>(a, d);
  where[0] = a.o - (float*)ws, where[1] = d.dg - (float*)ws, where[2] = d.dy - (float*)ws;
  return (int)cudaGetLastError();
}
