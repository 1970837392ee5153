// Gated GQA attention over an fp8 (e4m3) paged KV pool.
//
// Pool layout per layer: values [blocks, hkv, 16, D] e4m3, scales [blocks, hkv, 16] fp32 with
// scale = amax(|row|) / 448 over the head dim of one (token, kv head); K is quantised after
// RoPE.  The pool holds half the bytes of the bf16 pool, so a decode tick at long context reads
// half as much and twice the context fits.
//
//   attn_prep_fp8  : q/k per-head RMSNorm + partial RoPE, normalised Q out in bf16, K / V rows
//                    quantised and scattered with their scales (one warp per head).
//   attn_decode_fp8: head dim 256: split-KV on the tensor cores straight from the e4m3 rows (mma.sync, f16 operands, which
//                    hold e4m3 exactly); the row scales go into the score and into the output weights.
//   attn_split_fp8 : head dims 64 and 128, and rows off a 16-byte boundary: one key a warp, fp32 FMAs.
//   attn_combine   : merge of the split partials + sigmoid gate (same maths as the bf16 path).
//
// Reference parity: kernels_mma.py:89-166,247-366 (fp8 write / attn_prep_fp8) and the `_fp8`
// variants of kernels_attn.py:151-334 of packages/tilerl-kernels/src/tilerl_kernels; format
// definition reference.py:382-402.
#include <cuda_fp8.h>

#include "common.cuh"

namespace {

constexpr int KVB = 16;
constexpr int MAXG = 8;
constexpr float E4M3_MAX = 448.f;

__device__ __forceinline__ unsigned char to_e4m3(float v) {
  return (unsigned char)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

__global__ void __launch_bounds__(256)
attn_prep_fp8_kernel(const bf16* qkv, int ld, const float* __restrict__ qw,
                     const float* __restrict__ kw, const int* positions,
                     const int* slot_mapping, bf16* q_out,
                     unsigned char* kcache, unsigned char* vcache,
                     float* kscale, float* vscale, int n_q, int n_kv, int D,
                     int rotary, float log2_theta, float eps, int gated) {
  extern __shared__ float sm[];
  float* cs = sm;                 // [rotary/2] cos
  float* sn = sm + rotary / 2;    // [rotary/2] sin
  float* buf = sn + rotary / 2;   // [warps][D]
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int pos = positions[t];
  const int half = rotary >> 1;
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const double inv = exp2(-(double)(2 * i) / (double)rotary * (double)log2_theta);
    double s, c;
    sincos((double)pos * inv, &s, &c);
    cs[i] = (float)c, sn[i] = (float)s;
  }
  __syncthreads();
  const bf16* row = qkv + (size_t)t * ld;
  const int per_q = gated ? 2 * D : D;
  const int slot = slot_mapping[t];
  float* hb = buf + (size_t)warp * D;
  for (int h = warp; h < n_q + 2 * n_kv; h += nw) {
    const bool is_q = h < n_q, is_k = !is_q && h < n_q + n_kv;
    const bf16* src = is_q ? row + (size_t)h * per_q
                           : row + (size_t)n_q * per_q + (size_t)(h - n_q) * D;
    if (!is_q && slot < 0) continue;
    float ss = 0.f;
    for (int d = lane; d < D; d += 32) {
      const float v = __bfloat162float(src[d]);
      hb[d] = v;
      ss += v * v;
    }
    __syncwarp();
    if (is_q || is_k) {
      ss = warp_sum(ss);
      const float rstd = rsqrtf(ss / (float)D + eps);
      const float* w = is_q ? qw : kw;
      for (int d = lane; d < D; d += 32) hb[d] = hb[d] * rstd * w[d];
      __syncwarp();
      // rotate in place: each lane reads the pair it needs before anyone overwrites it
      for (int d = lane; d < half; d += 32) {
        const float a = hb[d], b = hb[d + half];
        hb[d] = a * cs[d] - b * sn[d];
        hb[d + half] = b * cs[d] + a * sn[d];
      }
      __syncwarp();
    }
    if (is_q) {
      bf16* dst = q_out + ((size_t)t * n_q + h) * D;
      for (int d = lane; d < D; d += 32) dst[d] = __float2bfloat16(hb[d]);
    } else {
      const int kvh = is_k ? h - n_q : h - n_q - n_kv;
      const size_t ridx = ((size_t)(slot / KVB) * n_kv + kvh) * KVB + (slot % KVB);
      float amax = 0.f;
      for (int d = lane; d < D; d += 32) amax = fmaxf(amax, fabsf(hb[d]));
      amax = warp_max(amax);
      const float sc = fmaxf(amax, 1e-30f) / E4M3_MAX;
      unsigned char* dst = (is_k ? kcache : vcache) + ridx * D;
      for (int d = lane; d < D; d += 32) dst[d] = to_e4m3(hb[d] / sc);
      if (lane == 0) (is_k ? kscale : vscale)[ridx] = sc;
    }
    __syncwarp();
  }
}

template <int VEC>
__device__ __forceinline__ void load_e4m3_row(const unsigned char* p, float (&f)[VEC]) {
  if constexpr (VEC == 8) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const uint32_t u[2] = {w.x, w.y};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 a = h2_to_f2(cvt_e4m3x2_to_h2((uint16_t)(u[i] & 0xFFFFu)));
      const float2 b = h2_to_f2(cvt_e4m3x2_to_h2((uint16_t)(u[i] >> 16)));
      f[4 * i] = a.x, f[4 * i + 1] = a.y, f[4 * i + 2] = b.x, f[4 * i + 3] = b.y;
    }
  } else if constexpr (VEC == 4) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
    const float2 a = h2_to_f2(cvt_e4m3x2_to_h2((uint16_t)(u & 0xFFFFu)));
    const float2 b = h2_to_f2(cvt_e4m3x2_to_h2((uint16_t)(u >> 16)));
    f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y;
  } else {
    static_assert(VEC == 2, "head dim must be 64, 128 or 256");
    const float2 a = h2_to_f2(cvt_e4m3x2_to_h2(*reinterpret_cast<const uint16_t*>(p)));
    f[0] = a.x, f[1] = a.y;
  }
}

// One CTA per (split, kv head, token).  VEC = D / 32 elements per lane.
template <int VEC>
__global__ void __launch_bounds__(256)
attn_split_fp8_kernel(const bf16* q, const bf16* gate_src, int gate_ld,
                      const unsigned char* kcache, const unsigned char* vcache,
                      const float* kscale, const float* vscale,
                      const int* block_table, int max_blocks,
                      const int* seq_ids, const int* positions,
                      float* po, float* pm, float* pl,
                      bf16* out, int n_q, int n_kv, int n_splits, float scale_log2e,
                      int gated) {
  constexpr int D = VEC * 32;
  __shared__ float s_m[8][MAXG], s_l[8][MAXG];
  extern __shared__ float s_acc[];  // [8 warps][MAXG][D]
  pdl_launch_dependents();
  pdl_wait();
  const int split = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = n_q / n_kv;
  const int pos = positions[t];
  const int kv_len = pos + 1;
  const int* table = block_table + (size_t)seq_ids[t] * max_blocks;
  const int pages = (kv_len + KVB - 1) / KVB;
  const int pps = (pages + n_splits - 1) / n_splits;
  const int lo = split * pps * KVB, hi = min(kv_len, (split + 1) * pps * KVB);

  float qr[MAXG][VEC];
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    if (g < G) {
      const bf16* qp = q + ((size_t)t * n_q + kvh * G + g) * D + lane * VEC;
#pragma unroll
      for (int v = 0; v < VEC; ++v) qr[g][v] = __bfloat162float(qp[v]) * scale_log2e;
    } else {
#pragma unroll
      for (int v = 0; v < VEC; ++v) qr[g][v] = 0.f;
    }
  }
  float m[MAXG], l[MAXG], acc[MAXG][VEC];
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    m[g] = -INFINITY, l[g] = 0.f;
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[g][v] = 0.f;
  }
  for (int j = lo + warp; j < hi; j += 8) {
    const int blk = table[j / KVB];
    const size_t ridx = ((size_t)blk * n_kv + kvh) * KVB + (j % KVB);
    const size_t off = ridx * D + lane * VEC;
    float kf[VEC], vf[VEC];
    load_e4m3_row<VEC>(kcache + off, kf);
    load_e4m3_row<VEC>(vcache + off, vf);
    const float ks = kscale[ridx], vs = vscale[ridx];
#pragma unroll
    for (int g = 0; g < MAXG; ++g) {
      if (g < G) {
        float s = 0.f;
#pragma unroll
        for (int v = 0; v < VEC; ++v) s = fmaf(qr[g][v], kf[v], s);
        s = warp_sum(s) * ks;
        const float mn = fmaxf(m[g], s);
        const float corr = exp2f(m[g] - mn), p = exp2f(s - mn);
        l[g] = l[g] * corr + p;
        const float pv = p * vs;
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[g][v] = fmaf(acc[g][v], corr, pv * vf[v]);
        m[g] = mn;
      }
    }
  }
  // merge the 8 warps
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    if (g < G) {
      if (lane == 0) s_m[warp][g] = m[g], s_l[warp][g] = l[g];
#pragma unroll
      for (int v = 0; v < VEC; ++v) s_acc[((size_t)warp * MAXG + g) * D + lane * VEC + v] = acc[g][v];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
    const int g = idx / D, d = idx % D;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 8; ++w) mm = fmaxf(mm, s_m[w][g]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float c = (s_m[w][g] == -INFINITY) ? 0.f : exp2f(s_m[w][g] - mm);
      ll += s_l[w][g] * c;
      a += s_acc[((size_t)w * MAXG + g) * D + d] * c;
    }
    const int h = kvh * G + g;
    if (n_splits == 1) {
      float o = ll > 0.f ? a / ll : 0.f;
      if (gated) o *= sigmoid_f(__bfloat162float(gate_src[(size_t)t * gate_ld + (size_t)h * 2 * D + D + d]));
      out[((size_t)t * n_q + h) * D + d] = __float2bfloat16(o);
    } else {
      const size_t base = ((size_t)t * n_q + h) * n_splits + split;
      po[base * D + d] = a;
      if (d == 0) pm[base] = mm, pl[base] = ll;
    }
  }
}

// ---- head dim 256 on the tensor cores ------------------------------------------------------------------
// What bounds it is the pool's bytes, so a key's K and V are read once for the (up to 8) query heads of its kv head and go
// from global memory to MMA fragments in registers, without a pass through shared memory.  Everything is transposed, so that
// the few heads are the MMA's 8 columns and the accumulators stay small: S^T = K Q^T (16 keys of a page x heads), then
// O^T += V^T P^T (16 dims x heads, 16 such tiles).  One warp works on one page at a time, its pages dealt round the block.
// Lane (g, t) = (lane / 4, lane % 4):
//   K   16 dims (16 bytes) of keys g and g + 8 a load: four MMAs under a fixed permutation of the dims, the query
//       fragments (registers) permuted alike.
//   V   16 bytes of keys 2t, 2t + 1, 2t + 8, 2t + 9 a load; byte i of two keys side by side is, converted, the A operand of
//       dims g * 16 + i and 128 + g * 16 + i.  The next page's K is loaded when this one's scores are done, its V after the
//       last product.
//   P^T two f16 parts (value and rest), moved from accumulator to operand layout by movmatrix.  The weights that multiply V
//       carry V's row scale (one fp32 product) and a power of two that puts the largest of them between 2^14 and 2^15: what
//       is above 2^-16 of the largest keeps 23 bits, and what is lost of a smaller one is below 2^-39 of the largest -- a
//       flat tail of tens of thousands of keys under one large weight loses 2^-24 of that.  The softmax's denominator is
//       summed in fp32 from the unscaled weights.
// An MMA's sums are cut off, not rounded, and the cuts of a long chain add up (a running O through 250 pages was 1e-5 off), so
// a chain is two products long and what it gives is added in fp32.
// Query rows are scaled by a power of two into f16's range: exact for elements above 2^-27 of the row's largest, within
// 2^-35 of the largest for those below.  12 sequences of 3 000 to 6 000 keys, 4 kv heads x 6:
// 620 us a layer with the one-key-a-warp kernel (products on the FMA pipe, a shuffle reduction for each score), 56 here with the
// merge of the splits, 51 without (the bytes: 17).
constexpr int F8_WARPS = 4, F8_D = 256;

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ uint32_t f2_to_h2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float max_over_g(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
}

// 2^e, e from -126 to 127 (beyond: the nearest of these)
__device__ __forceinline__ float pow2i(int e) { return __uint_as_float((uint32_t)(max(-126, min(127, e)) + 127) << 23); }
// The shift that puts the largest weight between 2^14 and 2^15; none known yet: as it is.
__device__ __forceinline__ int weight_shift(float largest, int now) {
  const int e = (int)((__float_as_uint(largest) >> 23) & 255u) - 127;
  return largest > 0.f ? min(120, 14 - e) : now;
}
// Pages of a split and splits that have any: a split gets `least` pages, so that a context shorter than the launch's split
// count was chosen for (a captured one is fixed) is not cut to pieces.  The splits after them are empty.
__device__ __forceinline__ int split_pages(int pages, int n_splits, int least) {
  const int n = max(1, min(n_splits, (pages + least - 1) / least));
  return (pages + n - 1) / n;
}
constexpr int F8_LEAST = 8;

__global__ void __launch_bounds__(F8_WARPS * 32)
attn_decode_fp8_kernel(const bf16* q, const bf16* gate_src, int gate_ld, const unsigned char* kcache,
                       const unsigned char* vcache, const float* kscale, const float* vscale, const int* block_table,
                       int max_blocks, const int* seq_ids, const int* positions, float* po, float* pm, float* pl, bf16* out,
                       int n_q, int n_kv, int n_splits, float scale_log2e, int gated) {
  __shared__ float s_m[F8_WARPS][MAXG], s_l[F8_WARPS][MAXG];
  __shared__ __align__(16) float s_acc[F8_WARPS][MAXG][F8_D];
  pdl_launch_dependents();
  pdl_wait();
  const int split = blockIdx.x, kvh = blockIdx.y, tok = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int G = n_q / n_kv;
  const int kv_len = positions[tok] + 1;
  const int* table = block_table + (size_t)seq_ids[tok] * max_blocks;
  const int pages = (kv_len + KVB - 1) / KVB;
  const int pps = split_pages(pages, n_splits, F8_LEAST);
  const int p_hi = min(pages, (split + 1) * pps);
  if (split * pps >= pages) {                      // an empty split: a neutral partial (which the merge does not read)
    for (int idx = threadIdx.x; idx < G * (F8_D / 4); idx += blockDim.x) {
      const size_t base = ((size_t)tok * n_q + kvh * G + idx / (F8_D / 4)) * n_splits + split;
      reinterpret_cast<float4*>(po + base * F8_D)[idx % (F8_D / 4)] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (idx % (F8_D / 4) == 0) pm[base] = -INFINITY, pl[base] = 0.f;
    }
    return;
  }
  int pg = split * pps + warp;

  uint4 kr[2][4], vr[4][2];                        // keys g, g + 8 x 64-dim steps; keys 2t, 2t + 1, 2t + 8, 2t + 9 x halves
  float ks[2], vs[2];
  auto page_row = [&](int p) { return ((size_t)table[p] * n_kv + kvh) * KVB; };
  auto load_k = [&](size_t row) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const unsigned char* src = kcache + (row + g + r * 8) * F8_D + t * 16;
#pragma unroll
      for (int st = 0; st < 4; ++st) kr[r][st] = __ldcg(reinterpret_cast<const uint4*>(src + st * 64));
      ks[r] = __ldcg(kscale + row + g + r * 8);
    }
  };
  auto load_v = [&](size_t row) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const unsigned char* src = vcache + (row + 2 * t + (r & 1) + (r >> 1) * 8) * F8_D + g * 16;
      vr[r][0] = __ldcg(reinterpret_cast<const uint4*>(src)), vr[r][1] = __ldcg(reinterpret_cast<const uint4*>(src + 128));
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) vs[r] = __ldcg(vscale + row + g + r * 8);
  };
  size_t row = 0;
  if (pg < p_hi) row = page_row(pg), load_k(row), load_v(row);

  // query fragments: head g, dims 64 st + 16 t .. + 15; element pairs in the order of the K loads
  uint32_t qf[4][8];
  float qs0, qs1;                                  // score scale of heads 2t and 2t + 1
  {
    uint32_t raw[4][8];
    float am = 0.f;
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      uint4 u0 = make_uint4(0u, 0u, 0u, 0u), u1 = u0;
      if (g < G) {
        const uint4* src = reinterpret_cast<const uint4*>(q + ((size_t)tok * n_q + kvh * G + g) * F8_D + st * 64 + t * 16);
        u0 = __ldcg(src), u1 = __ldcg(src + 1);
      }
      const uint32_t w[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        raw[st][i] = w[i];
        const float2 f = bf162_bits_to_f2(w[i]);
        am = fmaxf(am, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    int e = (int)((__float_as_uint(am) >> 23) & 255u) - 127 - 10;      // the largest element to 2^10 .. 2^11
    e = am > 0.f ? max(-116, min(126, e)) : 0;
    const float down = __uint_as_float((uint32_t)(127 - e) << 23), up = __uint_as_float((uint32_t)(127 + e) << 23);
#pragma unroll
    for (int st = 0; st < 4; ++st)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 f = bf162_bits_to_f2(raw[st][i]);
        qf[st][i] = f2_to_h2_bits(f.x * down, f.y * down);
      }
    qs0 = __shfl_sync(0xffffffffu, up, t * 8) * scale_log2e;
    qs1 = __shfl_sync(0xffffffffu, up, t * 8 + 4) * scale_log2e;
  }

  float o[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  // of heads 2t and 2t + 1: largest score, largest weight (as of the last shift), shift, denominator
  float m0 = -INFINITY, m1 = -INFINITY, n0 = 0.f, n1 = 0.f, l0 = 0.f, l1 = 0.f;
  int s0 = 0, s1 = 0;
  while (pg < p_hi) {
    const int left = kv_len - pg * KVB;            // keys of this page that exist
    // ---- S^T = K Q^T
    float sc[4], part[4];
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      const uint32_t ka[4] = {kr[0][st].x, kr[0][st].y, kr[0][st].z, kr[0][st].w};
      const uint32_t kb[4] = {kr[1][st].x, kr[1][st].y, kr[1][st].z, kr[1][st].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t a[4] = {cvt_e4m3x2_to_h2((uint16_t)ka[i]), cvt_e4m3x2_to_h2((uint16_t)kb[i]),
                               cvt_e4m3x2_to_h2((uint16_t)(ka[i] >> 16)), cvt_e4m3x2_to_h2((uint16_t)(kb[i] >> 16))};
        if (i % 2 == 0) part[0] = part[1] = part[2] = part[3] = 0.f;
        mma_f16(part, a, qf[st][2 * i], qf[st][2 * i + 1]);
        if (i % 2 == 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[e] = st == 0 && i == 1 ? part[e] : sc[e] + part[e];
        }
      }
    }
    const float k0 = ks[0], k1 = ks[1];
    const int nxt = pg + F8_WARPS;
    size_t nrow = 0;
    if (nxt < p_hi) nrow = page_row(nxt), load_k(nrow);
    // ---- scores (base 2) and their running maximum
    const bool in0 = g < left, in1 = g + 8 < left;
    const float v0 = in0 ? vs[0] : 0.f, v1 = in1 ? vs[1] : 0.f;
    const float a0 = in0 ? sc[0] * (k0 * qs0) : -INFINITY, a1 = in0 ? sc[1] * (k0 * qs1) : -INFINITY;
    const float a2 = in1 ? sc[2] * (k1 * qs0) : -INFINITY, a3 = in1 ? sc[3] * (k1 * qs1) : -INFINITY;
    const float mm0 = fmaxf(m0, max_over_g(fmaxf(a0, a2))), mm1 = fmaxf(m1, max_over_g(fmaxf(a1, a3)));
    const float mb0 = mm0 == -INFINITY ? 0.f : mm0, mb1 = mm1 == -INFINITY ? 0.f : mm1;
    const float e0 = exp2f(a0 - mb0), e1 = exp2f(a1 - mb1), e2 = exp2f(a2 - mb0), e3 = exp2f(a3 - mb1);
    const float t0 = exp2f(m0 - mb0), t1 = exp2f(m1 - mb1);
    l0 = fmaf(l0, t0, e0 + e2), l1 = fmaf(l1, t1, e1 + e3);             // this lane's keys; summed over g at the end
    // ---- weights on V, and the power of two that they are held with
    const float w0 = e0 * v0, w1 = e1 * v0, w2 = e2 * v1, w3 = e3 * v1;
    const float x0 = fmaxf(fabsf(w0), fabsf(w2)), x1 = fmaxf(fabsf(w1), fabsf(w3));
    if (__any_sync(0xffffffffu, mm0 != m0 || mm1 != m1 || x0 * pow2i(s0) > 32768.f || x1 * pow2i(s1) > 32768.f)) {
      n0 = fmaxf(n0 * t0, max_over_g(x0)), n1 = fmaxf(n1 * t1, max_over_g(x1));
      const int r0 = weight_shift(n0, s0), r1 = weight_shift(n1, s1);
      const float c0 = t0 * pow2i(r0 - s0), c1 = t1 * pow2i(r1 - s1);
      s0 = r0, s1 = r1;
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i][0] *= c0, o[i][1] *= c1, o[i][2] *= c0, o[i][3] *= c1;
    }
    m0 = mm0, m1 = mm1;
    // ---- P^T: value and rest, transposed into the B operand
    const float f_0 = pow2i(s0), f_1 = pow2i(s1);
    const float p0 = w0 * f_0, p1 = w1 * f_1, p2 = w2 * f_0, p3 = w3 * f_1;
    const uint32_t h0 = f2_to_h2_bits(p0, p1), h1 = f2_to_h2_bits(p2, p3);
    const float2 f0 = h2_to_f2(h0), f1 = h2_to_f2(h1);
    const uint32_t bh0 = movmatrix_t(h0), bh1 = movmatrix_t(h1);
    const uint32_t bl0 = movmatrix_t(f2_to_h2_bits(p0 - f0.x, p1 - f0.y)), bl1 = movmatrix_t(f2_to_h2_bits(p2 - f1.x, p3 - f1.y));
    if (left < KVB) {
      // the last page's keys past the sequence hold whatever the pool holds: their weights are 0, and 0 x V must be 0
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (2 * t + (r & 1) + (r >> 1) * 8 >= left) vr[r][0] = vr[r][1] = make_uint4(0u, 0u, 0u, 0u);
    }
    // ---- O^T += V^T P^T
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
      uint32_t x[4][2];                            // [key][half] words wi: bytes 4 wi .. 4 wi + 3
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          x[r][h] = wi == 0 ? vr[r][h].x : wi == 1 ? vr[r][h].y : wi == 2 ? vr[r][h].z : vr[r][h].w;
#pragma unroll
      for (int b2 = 0; b2 < 2; ++b2) {             // two dims a byte permutation
        const uint32_t sel = b2 == 0 ? 0x5140u : 0x7362u;
        const uint32_t y0 = __byte_perm(x[0][0], x[1][0], sel), y1 = __byte_perm(x[0][1], x[1][1], sel);
        const uint32_t y2 = __byte_perm(x[2][0], x[3][0], sel), y3 = __byte_perm(x[2][1], x[3][1], sel);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const uint32_t a[4] = {cvt_e4m3x2_to_h2((uint16_t)(y0 >> (16 * b))), cvt_e4m3x2_to_h2((uint16_t)(y1 >> (16 * b))),
                                 cvt_e4m3x2_to_h2((uint16_t)(y2 >> (16 * b))), cvt_e4m3x2_to_h2((uint16_t)(y3 >> (16 * b)))};
          float part[4] = {0.f, 0.f, 0.f, 0.f};
          mma_f16(part, a, bh0, bh1);
          mma_f16(part, a, bl0, bl1);
#pragma unroll
          for (int i = 0; i < 4; ++i) o[wi * 4 + b2 * 2 + b][i] += part[i];
        }
      }
    }
    if (nxt < p_hi) load_v(nrow);
    pg = nxt;
  }
#pragma unroll
  for (int s = 4; s < 32; s <<= 1) l0 += __shfl_xor_sync(0xffffffffu, l0, s), l1 += __shfl_xor_sync(0xffffffffu, l1, s);

  // ---- merge the warps: every accumulator relative to the warp's score maximum, without its shift
  {
    const float c0 = pow2i(-s0), c1 = pow2i(-s1);
    if (g == 0) s_m[warp][2 * t] = m0, s_m[warp][2 * t + 1] = m1, s_l[warp][2 * t] = l0, s_l[warp][2 * t + 1] = l1;
#pragma unroll
    for (int i = 0; i < 16; i += 4)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<float4*>(&s_acc[warp][2 * t][h * 128 + g * 16 + i]) =
            make_float4(o[i][2 * h] * c0, o[i + 1][2 * h] * c0, o[i + 2][2 * h] * c0, o[i + 3][2 * h] * c0);
        *reinterpret_cast<float4*>(&s_acc[warp][2 * t + 1][h * 128 + g * 16 + i]) =
            make_float4(o[i][2 * h + 1] * c1, o[i + 1][2 * h + 1] * c1, o[i + 2][2 * h + 1] * c1, o[i + 3][2 * h + 1] * c1);
      }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * F8_D; idx += blockDim.x) {
    const int gg = idx / F8_D, d = idx % F8_D;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < F8_WARPS; ++w) mm = fmaxf(mm, s_m[w][gg]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < F8_WARPS; ++w) {
      const float c = (s_m[w][gg] == -INFINITY) ? 0.f : exp2f(s_m[w][gg] - mm);
      ll += s_l[w][gg] * c;
      a += s_acc[w][gg][d] * c;
    }
    const int h = kvh * G + gg;
    if (n_splits == 1) {
      float v = ll > 0.f ? a / ll : 0.f;
      if (gated) v *= sigmoid_f(__bfloat162float(gate_src[(size_t)tok * gate_ld + (size_t)h * 2 * F8_D + F8_D + d]));
      out[((size_t)tok * n_q + h) * F8_D + d] = __float2bfloat16(v);
    } else {
      const size_t base = ((size_t)tok * n_q + h) * n_splits + split;
      po[base * F8_D + d] = a;
      if (d == 0) pm[base] = mm, pl[base] = ll;
    }
  }
}

__global__ void __launch_bounds__(256)
attn_combine_fp8_kernel(const float* po, const float* pm,
                        const float* pl, const bf16* gate_src, int gate_ld, const int* positions,
                        bf16* out, int n_q, int D, int n_splits, int least, int gated) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  const size_t base = ((size_t)t * n_q + h) * n_splits;
  const int pages = (positions[t] + KVB) / KVB, pps = split_pages(pages, n_splits, least);
  const int used = (pages + pps - 1) / pps;        // the splits after these are empty
  float mm = -INFINITY;
  for (int s = 0; s < used; ++s) mm = fmaxf(mm, pm[base + s]);
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float ll = 0.f, a = 0.f;
    for (int s = 0; s < used; ++s) {
      const float ms = pm[base + s];
      const float c = (ms == -INFINITY) ? 0.f : exp2f(ms - mm);
      ll += pl[base + s] * c;
      a += po[(base + s) * D + d] * c;
    }
    float o = ll > 0.f ? a / ll : 0.f;
    if (gated) o *= sigmoid_f(__bfloat162float(gate_src[(size_t)t * gate_ld + (size_t)h * 2 * D + D + d]));
    out[((size_t)t * n_q + h) * D + d] = __float2bfloat16(o);
  }
}

}  // namespace

// kcache / vcache: e4m3 bytes of one layer; kscale / vscale: its fp32 row scales.
TRL_API int trl_attn_prep_fp8(const void* qkv, int ld, const void* q_norm, const void* k_norm,
                              const void* positions, const void* slot_mapping, void* q_out, void* kcache,
                              void* vcache, void* kscale, void* vscale, int T, int n_q, int n_kv, int D,
                              int rotary, float theta, float eps, int gated, void* stream) {
  const int threads = 256;
  if (rotary > D || (rotary & 1)) return (int)cudaErrorInvalidValue;
  const size_t smem = (size_t)(rotary + (threads / 32) * D) * sizeof(float);
  return (int)trl_launch(attn_prep_fp8_kernel, dim3(T), dim3(threads), smem, (cudaStream_t)stream,
                         (const bf16*)qkv, ld, (const float*)q_norm, (const float*)k_norm,
                         (const int*)positions, (const int*)slot_mapping, (bf16*)q_out,
                         (unsigned char*)kcache, (unsigned char*)vcache, (float*)kscale, (float*)vscale, n_q,
                         n_kv, D, rotary, log2f(theta), eps, gated);
}

// Scratch as for the bf16 split kernel: po [T*n_q*n_splits*D] fp32, pm/pl [T*n_q*n_splits] fp32.
TRL_API int trl_attn_paged_fp8(const void* q, const void* gate_src, int gate_ld, const void* kcache,
                               const void* vcache, const void* kscale, const void* vscale,
                               const void* block_table, int max_blocks, const void* seq_ids,
                               const void* positions, void* po, void* pm, void* pl, void* out, int T, int n_q,
                               int n_kv, int D, int n_splits, float scale, int gated, void* stream) {
  if (n_q % n_kv != 0 || n_q / n_kv > MAXG) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  const float sl2 = scale * 1.4426950408889634f;
  const dim3 grid(n_splits, n_kv, T);
  const size_t smem = (size_t)8 * MAXG * D * sizeof(float);
  cudaError_t e;
#define SPLIT_CASE(V)                                                                                 \
  {                                                                                                   \
    auto kern = attn_split_fp8_kernel<V>;                                                             \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
    e = trl_launch(kern, grid, dim3(256), smem, st, (const bf16*)q, (const bf16*)gate_src, gate_ld,   \
                   (const unsigned char*)kcache, (const unsigned char*)vcache, (const float*)kscale,  \
                   (const float*)vscale, (const int*)block_table, max_blocks, (const int*)seq_ids,    \
                   (const int*)positions, (float*)po, (float*)pm, (float*)pl, (bf16*)out, n_q, n_kv,  \
                   n_splits, sl2, gated);                                                             \
  }
  // the tensor-core kernel reads rows 16 bytes at a time, the other one 8 (K, V) and 2 (query)
  const bool tc = D == F8_D && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15) == 0;
  if (tc)
    e = trl_launch(attn_decode_fp8_kernel, grid, dim3(F8_WARPS * 32), 0, st, (const bf16*)q, (const bf16*)gate_src, gate_ld,
                   (const unsigned char*)kcache, (const unsigned char*)vcache, (const float*)kscale, (const float*)vscale,
                   (const int*)block_table, max_blocks, (const int*)seq_ids, (const int*)positions, (float*)po, (float*)pm,
                   (float*)pl, (bf16*)out, n_q, n_kv, n_splits, sl2, gated);
  else if (D == F8_D) SPLIT_CASE(8)
  else if (D == 128) SPLIT_CASE(4)
  else if (D == 64) SPLIT_CASE(2)
  else return (int)cudaErrorInvalidValue;
#undef SPLIT_CASE
  if (e != cudaSuccess) return (int)e;
  if (n_splits > 1)
    e = trl_launch(attn_combine_fp8_kernel, dim3(T, n_q), dim3(min(D, 256)), 0, st, (const float*)po,
                   (const float*)pm, (const float*)pl, (const bf16*)gate_src, gate_ld, (const int*)positions, (bf16*)out, n_q, D,
                   n_splits, tc ? F8_LEAST : 1, gated);
  return (int)e;
}
