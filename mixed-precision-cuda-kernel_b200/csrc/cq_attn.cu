// Single-query attention over the KV cache (decode) for 64- and 128-wide heads and up to 8 query heads per KV head, on
// mma.sync; in the reference a part of its vendored LLaMA (llama/modeling_llama_quant.py:371-419 of the reference project).
//
// The bound is the cache itself, read once.  With fp32 dot products a step of 8 query heads per KV head was bound by its
// arithmetic, one head per KV head by latencies and registers; here the arithmetic is small beside the loads in either
// case (32 MMAs per 8 KB of cache and warp), so one kernel serves both:
//   * scores S (heads x positions) = Q . K^T, m16n8k16: rows 0-7 of A are the query heads.  A lane's share of a
//     position's key is two or four 16-byte pieces, loaded straight from the cache: the order of the columns inside a
//     step is free as long as both operands agree;
//   * the sums land where P . V needs its A operand.  Rows 0-7 take the upper 11 bits of the weights, rows 8-15, which
//     the heads leave empty, the next 11;
//   * V is the B operand, two positions' 16-byte pieces interleaved in registers (which columns of the head an MMA
//     covers is free, too).
// A warp takes 16 positions a turn with all of their keys and values in flight, and keeps its own running maximum, sum
// and weighted values; the warps meet once in shared memory, the ranges of positions (blockIdx.z) in the workspace, where
// the CTA that arrives last merges them.
//
// Precision: a weight loses at most 2^-23 of itself in its two halves (a quarter of them their last bit), and what lies below
// 2^-38 of the largest.  An MMA cuts its sums off instead of rounding them, the more the larger its addend, so each one
// sums its 16 products alone and fp32 additions do the rest; sums are rescaled by whole powers of two, and added in pairs
// where warps and ranges meet.  Outputs that differ from the correctly rounded result, against 64 bits over 100 calls of
// 64- and 128-wide heads, 60 to 4096 positions: 1.1e-4 of them with scores of deviation 1 (the fp32 kernels of cq_model_ops.cu
// 1.1e-4), 1.1e-3 with deviation 4 (1.25e-3); with the sums left to the MMAs it was 1.8e-4 and 1.7e-3.  The chains of MMAs
// gone, a call is no slower: 64 query heads on 8 KV heads at 4000 positions, 16 sequences, 50 us and 53.
//
// ROPE: the step's rotary embedding and cache write ride along (one launch less a layer): queries are rotated on their way
// into shared memory, the new position's key and value go into the caches by the CTA whose range ends with it.
#include <algorithm>
#include <type_traits>

#include "cq_attn.cuh"

namespace {

constexpr int AM_SM_WARPS = 12;              // warps an SM holds (168 registers a thread)
constexpr int AM_HEADS = 8;                  // query heads of a CTA
constexpr int AM_POS = 16;                   // positions of a turn
constexpr int AM_MAX_SPLITS = 32;            // (a lane per range in the merge)

// sums of 16 products, without an addend: the unit cuts its sums off, fp32 additions outside round them
__device__ __forceinline__ void am_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// with results below the normal numbers
__device__ __forceinline__ float ex2_full(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^d of a whole number d <= 0; 0 below the normal numbers (and 1 for NaN, whose sums are NaN)
__device__ __forceinline__ float whole_pow2(float d) { return __int_as_float(max(0, 127 + __float2int_rn(d)) << 23); }
// the share of a warp's or range's sums (maximum m, sum of weights l) in those that reach up to `top`: 0 where it has no
// position, but 1 where its only scores are NaN
__device__ __forceinline__ float share_of(float m, float l, float top) {
  if (m == -INFINITY) return l == 0.f ? 0.f : 1.f;
  const int d = __float2int_rn(m - top);
  return d < -126 ? (d < -149 ? 0.f : __int_as_float(1 << (149 + d))) : whole_pow2(m - top);
}
// 16 bytes of a cache; not as read-only data where the launch itself writes a row of it
template <bool WRITTEN> __device__ __forceinline__ uint4 ld_cache(const __half* p) {
  if (!WRITTEN) return __ldg(reinterpret_cast<const uint4*>(p));
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// the upper 11 bits of two weights, and what is left of them
__device__ __forceinline__ uint2 split_weights(float a, float b) {
  const __half2 hi = __floats2half2_rn(a, b);
  const float2 f = __half22float2(hi);
  const __half2 lo = __floats2half2_rn(a - f.x, b - f.y);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&hi), *reinterpret_cast<const uint32_t*>(&lo));
}

struct RopeStep {
  const __half* k;            // [sequence][KV][D], not rotated
  const __half* v;
  const float* cos_t;         // [max_seq][D / 2]
  const float* sin_t;
};

// eight columns of the lower half of a head (x1) and the same of the upper half (x2), rotated as rope_cache_kernel does
__device__ __forceinline__ void rotate8(uint4& x1, uint4& x2, const float* __restrict__ cos_p, const float* __restrict__ sin_p) {
  __half* h1 = reinterpret_cast<__half*>(&x1);
  __half* h2 = reinterpret_cast<__half*>(&x2);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float a = __half2float(h1[e]), b = __half2float(h2[e]), c = cos_p[e], s = sin_p[e];
    h1[e] = __float2half(a * c - b * s);
    h2[e] = __float2half(b * c + a * s);
  }
}

template <int D, int WARPS, bool ROPE>
__global__ void __launch_bounds__(WARPS * 32, AM_SM_WARPS / WARPS) attn_decode_mma_kernel(
    const __half* __restrict__ q, __half* k_cache, __half* v_cache, const RopeStep rope,
    const long long* __restrict__ pos, __half* __restrict__ out, float* __restrict__ part,
    unsigned int* __restrict__ counters, int H, int KV, int max_seq, float scale) {
  constexpr int THREADS = WARPS * 32;
  constexpr int KP = D / 32;                 // 16-byte pieces of a position's key per lane (four lanes a position)
  constexpr int VS = D / 64;                 // of a position's value (eight lanes a position)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(16) float am_sum[];          // [warp][head][D]
  __shared__ __align__(16) __half s_q[AM_HEADS][D + 32];
  __shared__ float s_m[WARPS][AM_HEADS], s_l[WARPS][AM_HEADS];
  __shared__ float s_f[AM_HEADS][AM_MAX_SPLITS], s_r[AM_HEADS][AM_MAX_SPLITS], s_top[AM_HEADS], s_tot[AM_HEADS];
  __shared__ int s_last;
  const int kvh = blockIdx.x, seq = blockIdx.y, split = blockIdx.z, nsplit = gridDim.z;
  const int G = H / KV, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long pl = pos[seq];
  const int n_all = pl < 0 ? 1 : (pl >= max_seq ? max_seq : (int)pl + 1);
  const int chunk = (n_all + nsplit - 1) / nsplit;
  const int pbeg = split * chunk;
  const int n_pos = max(0, min(n_all - pbeg, chunk));
  const size_t row = (size_t)KV * D;         // elements between consecutive positions of a cache
  const size_t first = ((size_t)seq * max_seq + pbeg) * row + (size_t)kvh * D;
  const size_t head0 = (size_t)seq * H + (size_t)kvh * G;

  // queries in shared memory (in registers they would spill): a lane's pieces 8 t4 + 32 i of head g8
  const bool step = ROPE && pl >= 0 && pl < max_seq;       // (a position outside the tables and caches: as it is, nothing is written)
  if (ROPE) {
    const float* cos_p = rope.cos_t + (step ? pl : 0) * (D / 2);
    const float* sin_p = rope.sin_t + (step ? pl : 0) * (D / 2);
    constexpr int PIECES = D / 16;
    for (int i = tid; i < AM_HEADS * PIECES; i += THREADS) {
      const int g = i / PIECES, c = 8 * (i - g * PIECES);
      uint4 x1 = make_uint4(0, 0, 0, 0), x2 = x1;
      if (g < G) {
        x1 = *reinterpret_cast<const uint4*>(q + (head0 + g) * D + c);
        x2 = *reinterpret_cast<const uint4*>(q + (head0 + g) * D + c + D / 2);
        if (step) rotate8(x1, x2, cos_p + c, sin_p + c);
      }
      *reinterpret_cast<uint4*>(&s_q[g][c]) = x1;
      *reinterpret_cast<uint4*>(&s_q[g][c + D / 2]) = x2;
    }
    if (step && n_pos > 0 && pbeg + n_pos == n_all && tid < 2 * PIECES) {
      const size_t from = ((size_t)seq * KV + kvh) * D, to = first + (size_t)(n_pos - 1) * row;
      const int c = 8 * (tid % PIECES);
      const bool value = tid >= PIECES;
      const __half* src = (value ? rope.v : rope.k) + from + c;
      __half* dst = (value ? v_cache : k_cache) + to + c;
      uint4 x1 = *reinterpret_cast<const uint4*>(src), x2 = *reinterpret_cast<const uint4*>(src + D / 2);
      if (!value) rotate8(x1, x2, cos_p + c, sin_p + c);
      *reinterpret_cast<uint4*>(dst) = x1;
      *reinterpret_cast<uint4*>(dst + D / 2) = x2;
    }
  } else {
    for (int i = tid; i < AM_HEADS * D / 8; i += THREADS) {
      const int g = i / (D / 8), c = 8 * (i - g * (D / 8));
      *reinterpret_cast<uint4*>(&s_q[g][c]) = g < G ? *reinterpret_cast<const uint4*>(q + (head0 + g) * D + c) : make_uint4(0, 0, 0, 0);
    }
  }
  __syncthreads();
  const __half* mine_q = &s_q[g8][8 * t4];

  const float scale2 = scale * 1.4426950408889634f;        // scores in powers of two
  float m = -INFINITY, l = 0.f;
  float o[8 * VS][2];                        // MMA j + 8 s: its column n is column 64 s + 8 n + j of the head
#pragma unroll
  for (int i = 0; i < 8 * VS; ++i) o[i][0] = o[i][1] = 0.f;

#pragma unroll 1
  for (int base = warp * AM_POS; base < n_pos; base += WARPS * AM_POS) {
    uint4 kk[2][KP], vv[4][VS];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int p = base + 8 * h + g8;
#pragma unroll
      for (int i = 0; i < KP; ++i)
        kk[h][i] = p < n_pos ? ld_cache<ROPE>(k_cache + first + (size_t)p * row + 8 * t4 + 32 * i) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = base + 8 * (u >> 1) + 2 * t4 + (u & 1);
#pragma unroll
      for (int i = 0; i < VS; ++i)
        vv[u][i] = p < n_pos ? ld_cache<ROPE>(v_cache + first + (size_t)p * row + 8 * g8 + 64 * i) : make_uint4(0, 0, 0, 0);
    }
    float s[2][2] = {};
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const uint4 qa = *reinterpret_cast<const uint4*>(mine_q + 32 * i);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float d0[4], d1[4];
        am_mma(d0, qa.x, 0u, qa.y, 0u, kk[h][i].x, kk[h][i].y);
        am_mma(d1, qa.z, 0u, qa.w, 0u, kk[h][i].z, kk[h][i].w);
        s[h][0] += d0[0] + d1[0];
        s[h][1] += d0[1] + d1[1];
      }
    }
    // this lane: head g8, positions base + 8 h + 2 t4 + e
    float top = m;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) top = fmaxf(top, base + 8 * h + 2 * t4 + e < n_pos ? s[h][e] * scale2 : -INFINITY);
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    // A whole number at or above the maximum, so that rescaling sums is exact.  (No finite score so far: weights 0, or NaN
    // where a score is NaN, which no maximum shows.)
    top = ceilf(top);
    const float ref = top == -INFINITY ? 0.f : top;
    const float keep = whole_pow2(m - ref);
    m = top;
    // weights times 2^15: the halves of their split then reach down to 2^-38 of the largest.  (One rounding between the score
    // and the exponent, of the size of the exponent, not of the score.)
    float w[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        w[h][e] = base + 8 * h + 2 * t4 + e < n_pos ? 32768.f * ex2(__fmaf_rn(s[h][e], scale2, -ref)) : 0.f;
    l = l * keep + ((w[0][0] + w[0][1]) + (w[1][0] + w[1][1]));
    const uint2 w0 = split_weights(w[0][0], w[0][1]), w1 = split_weights(w[1][0], w[1][1]);
#pragma unroll
    for (int i = 0; i < VS; ++i) {
      const uint32_t* v0 = reinterpret_cast<const uint32_t*>(&vv[0][i]);
      const uint32_t* v1 = reinterpret_cast<const uint32_t*>(&vv[1][i]);
      const uint32_t* v2 = reinterpret_cast<const uint32_t*>(&vv[2][i]);
      const uint32_t* v3 = reinterpret_cast<const uint32_t*>(&vv[3][i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
        float d[4];
        am_mma(d, w0.x, w0.y, w1.x, w1.y, __byte_perm(v0[j >> 1], v1[j >> 1], sel), __byte_perm(v2[j >> 1], v3[j >> 1], sel));
        o[8 * i + j][0] = o[8 * i + j][0] * keep + (d[0] + d[2]);
        o[8 * i + j][1] = o[8 * i + j][1] * keep + (d[1] + d[3]);
      }
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t4 == 0) {
    s_m[warp][g8] = m;
    s_l[warp][g8] = l;
  }
  if (g8 < G) {
    float* to = am_sum + (warp * AM_HEADS + g8) * D;
#pragma unroll
    for (int i = 0; i < VS; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c)            // columns n = 2 t4 + c
#pragma unroll
        for (int j = 0; j < 8; j += 4)
          *reinterpret_cast<float4*>(to + 64 * i + 8 * (2 * t4 + c) + j) =
              make_float4(o[8 * i + j][c], o[8 * i + j + 1][c], o[8 * i + j + 2][c], o[8 * i + j + 3][c]);
  }
  __syncthreads();
  // The warps' shares in each head's sums.  (A share of 0 is multiplied all the same: what is NaN or infinite stays so or
  // becomes NaN, as a weight of 0 does.)
  for (int g = warp; g < G; g += WARPS) {
    const float mw = lane < WARPS ? s_m[lane][g] : -INFINITY, lw = lane < WARPS ? s_l[lane][g] : 0.f;
    float top = mw;
    for (int d = 8; d; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
    const float f = share_of(mw, lw, top);
    float tot = f * lw;
    for (int d = 8; d; d >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, d);
    if (lane < WARPS) s_f[g][lane] = f;
    if (lane == 0) {
      s_top[g] = top;
      s_tot[g] = tot;
    }
  }
  __syncthreads();
  for (int e = tid; e < G * D / 4; e += THREADS) {
    const int g = e / (D / 4), d = 4 * (e - g * (D / 4));
    float4 sums[WARPS];
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = s_f[g][w];
      const float4 x = *reinterpret_cast<const float4*>(am_sum + (w * AM_HEADS + g) * D + d);
      sums[w] = make_float4(f * x.x, f * x.y, f * x.z, f * x.w);
    }
#pragma unroll
    for (int n = WARPS; n > 1; n = (n + 1) / 2)             // (pairs of pairs: fewer roundings in a row)
#pragma unroll
      for (int w = 0; w < n / 2; ++w) {
        sums[w].x += sums[n - 1 - w].x;
        sums[w].y += sums[n - 1 - w].y;
        sums[w].z += sums[n - 1 - w].z;
        sums[w].w += sums[n - 1 - w].w;
      }
    float sum[4] = {sums[0].x, sums[0].y, sums[0].z, sums[0].w};
    const float top = s_top[g], tot = s_tot[g];
    if (!(fabsf(sum[0]) + fabsf(sum[1]) + fabsf(sum[2]) + fabsf(sum[3]) <= 3.0e38f) && tot == tot) {
      // An infinite or NaN value takes part.  The two halves of a weight turn infinity into NaN where the product does
      // not: these columns are added again, weight by weight.
      sum[0] = sum[1] = sum[2] = sum[3] = 0.f;
      for (int p = 0; p < n_pos; ++p) {
        const __half* kr = k_cache + first + (size_t)p * row;
        float dot = 0.f;
        for (int c = 0; c < D; ++c) dot += __half2float(s_q[g][c]) * __half2float(kr[c]);
        const float w = 32768.f * ex2_full(__fmaf_rn(dot, scale2, top == -INFINITY ? 0.f : -top));
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] += w * __half2float(v_cache[first + (size_t)p * row + d + c]);
      }
    }
    if (nsplit == 1) {
      __half2* to = reinterpret_cast<__half2*>(out + (head0 + g) * D + d);
      to[0] = __floats2half2_rn(sum[0] / tot, sum[1] / tot);
      to[1] = __floats2half2_rn(sum[2] / tot, sum[3] / tot);
    } else {
      float* mine = part + ((head0 + g) * nsplit + split) * (size_t)(D + 2);
      *reinterpret_cast<float2*>(mine + 2 + d) = make_float2(sum[0], sum[1]);
      *reinterpret_cast<float2*>(mine + 4 + d) = make_float2(sum[2], sum[3]);
      if (d == 0) *reinterpret_cast<float2*>(mine) = make_float2(top, tot);
    }
  }
  if (nsplit == 1) return;
  // several ranges: the last CTA of these heads merges
  __threadfence();
  __syncthreads();
  const size_t cidx = (size_t)seq * KV + kvh;
  if (tid == 0) s_last = atomicAdd(&counters[cidx], 1u) == (unsigned int)(nsplit - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the ranges' weights, then two columns a thread, whose first sums are on their way meanwhile
  const float* all = part + head0 * nsplit * (size_t)(D + 2);
  float2 x[8];
  auto fetch = [&](int e, int r0) {
    const float* src = all + (size_t)(e / (D / 2)) * nsplit * (D + 2) + 2 + 2 * (e % (D / 2));
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = __ldcg(reinterpret_cast<const float2*>(src + (size_t)min(r0 + u, nsplit - 1) * (D + 2)));
  };
  if (tid < G * D / 2) fetch(tid, 0);
  for (int e = tid; e < G * nsplit; e += THREADS) {
    const int g = e / nsplit, r = e - g * nsplit;
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(all + (size_t)e * (D + 2)));
    s_f[g][r] = ml.x;
    s_r[g][r] = ml.y;
  }
  __syncthreads();
  for (int g = warp; g < G; g += WARPS) {
    const float mr = lane < nsplit ? s_f[g][lane] : -INFINITY, lr = lane < nsplit ? s_r[g][lane] : 0.f;
    float top = mr;
    for (int d = 16; d; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
    const float f = share_of(mr, lr, top);
    float tot = f * lr;
    for (int d = 16; d; d >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, d);
    if (lane < nsplit) s_f[g][lane] = f;
    if (lane == 0) s_tot[g] = tot;
  }
  __syncthreads();
  for (int e = tid; e < G * D / 2; e += THREADS) {
    const int g = e / (D / 2), d = 2 * (e - g * (D / 2));
    float2 v[4] = {};
    for (int r0 = 0; r0 < nsplit; r0 += 8) {
      if (e != tid || r0) fetch(e, r0);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool in = r0 + u < nsplit;
        const float f = in ? s_f[g][r0 + u] : 0.f;
        v[u & 3].x = in ? __fmaf_rn(f, x[u].x, v[u & 3].x) : v[u & 3].x;
        v[u & 3].y = in ? __fmaf_rn(f, x[u].y, v[u & 3].y) : v[u & 3].y;
      }
    }
    *reinterpret_cast<__half2*>(out + (head0 + g) * D + d) =
        __floats2half2_rn(((v[0].x + v[1].x) + (v[2].x + v[3].x)) / s_tot[g], ((v[0].y + v[1].y) + (v[2].y + v[3].y)) / s_tot[g]);
  }
  if (tid == 0) counters[cidx] = 0u;                       // ready for the next launch
}

}  // namespace

bool cq_attn_mma_takes(int sequences, int n_heads, int n_kv_heads, int head_dim, int max_seq, bool step) {
  const int G = n_heads / n_kv_heads, sms = cq_sm_count();
  if ((head_dim != 64 && head_dim != 128) || G > AM_HEADS) return false;
  // Without grouped queries the two-sweep kernel has four CTAs of 256 threads on an SM against three of 128 here.  Up to one
  // wave of those, and for well-filled waves on short caches, this kernel is faster (128-wide heads on cold caches: 40 at
  // 2200 positions 15.0 us against 19.5; 256 at 192 9.0 and 11.1; 320 at 2200 70 and 81; 1280 at 512 60 and 68), beyond it is
  // not (512 at 512 37 and 29, 1024 at 4096 325 and 317).
  const long long tasks = (long long)sequences * n_kv_heads, slots = 3ll * sms;
  const long long waves = (tasks + slots - 1) / slots;
  if (!step) {
    // Where the rotation is not part of the call (its launch less, 1.9 us, makes up for it): one CTA for each of up to 148
    // heads at once, on caches just beyond one turn of twelve warps (256 positions, 32 heads 6.3 us against 4.9, 64 on 8 KV
    // heads 5.3 and 4.5); one-sweep CTAs of 256 positions that fill the chip once (32 heads at 1024 9.8 and 8.9); about two CTAs
    // an SM of 64-wide heads on long caches (256 heads at 1024 positions 20.9 and 19.1, 4096 59 and 53).
    const long long one_sweep = tasks * ((max_seq + 255) / 256);
    if (head_dim == 128 && max_seq > 12 * AM_POS && max_seq <= 256 && (long long)sequences * n_heads <= sms) return false;
    if (head_dim == 128 && G == 1 && max_seq >= 1024 && one_sweep <= sms && 10 * one_sweep >= 8 * sms) return false;
    if (head_dim == 64 && G == 1 && 2 * tasks > 3ll * sms && tasks <= 2ll * sms && max_seq > 768) return false;
  }
  return G > 1 || waves == 1 || (max_seq <= 512 && 10 * tasks >= 8 * waves * slots);
}

int cq_attn_mma_launch(const void* q, const void* k_cache, const void* v_cache, const long long* position, void* out, int sequences,
                       int n_heads, int n_kv_heads, int head_dim, int max_seq, float scale, int most, unsigned int* counters,
                       float* part, cudaStream_t stream, const void* k_new, const void* v_new, const float* cos_table,
                       const float* sin_table) {
  // CTAs of twelve warps, one on an SM, or of four, three on an SM, and ranges of positions: what takes the least time by a
  // model.  A turn brings 16 positions to each warp, in the latency of its loads where an SM has four warps, else in what its
  // warps need together; a CTA's start and its warps' meeting take 3 us, ranges their merge.  Over 615 calls (1 to 1280 heads,
  // 128 to 4096 positions) the plan is within 1 % of the best one measured, on average.  64 query heads on 8 KV heads at 4096
  // positions: 1 sequence 12.5 us, 4 20, 16 50, 32 93; the fp32 dot products took 47, 103, 271 and 429, flash_attn 20, 27, 64
  // and 194.  32 heads at 512 positions 7.4 us, against 8.1 of the two-sweep kernel; 160 at 4096 63 and 78.
  const int sms = cq_sm_count(), G = n_heads / n_kv_heads;
  const long long tasks = (long long)sequences * n_kv_heads;
  const double latency = head_dim == 64 ? 1.0 : 1.75, full = head_dim == 64 ? 1.3 : 2.1;      // us a turn: four warps on an SM, more
  if (most > AM_MAX_SPLITS) most = AM_MAX_SPLITS;
  int warps = 12, splits = 1;
  double best = 0;
  for (int w = 12; w >= 4; w -= 8)
    for (int n = 1; n <= most; ++n) {
      const int per_sm = AM_SM_WARPS / w;
      const long long waves = (tasks * n + per_sm * sms - 1) / (per_sm * sms), fullest = (tasks * n + sms - 1) / sms;
      const int turns = ((max_seq + n - 1) / n + w * AM_POS - 1) / (w * AM_POS);
      const double turn = per_sm > 1 && fullest == 1 ? latency : full;
      double t = (double)waves * (turns * turn + 3.0) + (n > 1 ? 1.7 + 0.3 * n + 0.3 * G : 0.0);
      // Ranges in several waves must pay for what they cost while the cache is nearly empty (320 64-wide heads, a tenth of 2048
      // positions: one range 8.0 us, four 14.2; all of them 43 both).
      if (n > 1 && waves > 1) t *= 1.2;
      if ((w == 12 && n == 1) || t < best) {
        best = t;
        warps = w;
        splits = n;
      }
    }
  auto pick = [&](auto rope) {
    constexpr bool R = decltype(rope)::value;
    return head_dim == 64 ? (warps == 4 ? attn_decode_mma_kernel<64, 4, R> : attn_decode_mma_kernel<64, 12, R>)
                          : (warps == 4 ? attn_decode_mma_kernel<128, 4, R> : attn_decode_mma_kernel<128, 12, R>);
  };
  auto fn = k_new ? pick(std::true_type()) : pick(std::false_type());
  const int smem = warps * AM_HEADS * head_dim * (int)sizeof(float);
  CQ_CUDA_TRY(cq_grant_smem((const void*)fn, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n_kv_heads, sequences, splits);
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, (const __half*)q, (__half*)k_cache, (__half*)v_cache,
                                 RopeStep{(const __half*)k_new, (const __half*)v_new, cos_table, sin_table}, position, (__half*)out, part,
                                 counters, n_heads, n_kv_heads, max_seq, scale));
  return CQ_OK;
}
