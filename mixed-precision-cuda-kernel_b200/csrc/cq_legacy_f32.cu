// fp32-I/O variant of the 3-bit operator, selected by `fp16 == false` in the
// reference (csrc/quant_cuda_kernel.cu:159-179 of the reference project:
// VecQuant3MatMulKernelCherryQBatched / ...G64, float x / scales / cherry / mul,
// int32 indices).  Only the reference's micro-benchmark uses it
// (benchmark_speed.py:32).  It reads the reference's uint8 layout directly and
// adds into `mul` with fp32 atomics like the reference.
//
// Products of 3-bit codes with fp32 activations on the integer tensor cores: per row of x and 128 compact columns (64
// where a scale group has 64) the activations become 31-bit fixed point (step 2^-29 of the power of two at the largest
// one, so everything down to 2^-6 of it keeps all its bits), four signed-byte planes of which are B operands of
// mma.sync.m16n8k32; the codes are the A operand.  Sums over a group are exact integers, (2 u - 7) x included, and meet
// the scale in fp32.  The columns that share a step share their scale too, and no |u - 3.5| is below 1/2: half a step is
// 2^-6 or less of what an fp32 addition rounds away beside the largest product (only activations that are smaller than
// 2^-24 of two large ones which cancel are lost where a chain of additions in a lucky order keeps them).  A loop of fp32
// multiply-adds needs 25 us of the FMA pipe for 16 rows of 4096 x 13824, before the decode of each code by the one
// thread that uses it.  That case: 52 us a call (93 with the loop), bound by the issue rate: staging of x by every
// column block, byte decode and the fp32 combination share it.
#include "cq_common.cuh"

namespace {

constexpr int F32_THREADS = 256;       // 8 warps, 32 output columns each
constexpr int F32_COLS = 256;
constexpr int F32_MAX_BLOCKS = 10;     // 128-column blocks a CTA stages

struct F32Params {
  const float* x;
  const uint8_t* q;
  const float* cw;
  const int32_t* idx;
  const float* sf;
  float* mul;
  int M, K, N, C, G, Kc, n_blk, blk_per_part, n_parts, aligned_q, aligned_f;
};

__device__ __forceinline__ int f32_source_col(const F32Params& p, int kc) {
  int low = 0, high = p.C;
  while (low < high) {
    const int mid = (low + high) >> 1;
    if (p.idx[mid] - mid <= kc) low = mid + 1; else high = mid;
  }
  return kc + low;
}

// 2^e as two factors (each a normal number) for -180 <= e <= 180
__device__ __forceinline__ float2 f32_pow2_pair(int e) {
  const int a = e >> 1, b = e - a;
  return make_float2(__int_as_float((a + 127) << 23), __int_as_float((b + 127) << 23));
}

__device__ __forceinline__ void imma(int (&d)[4], const uint32_t (&a)[4], uint2 b) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

// the byte rows of octet o for the four columns at n (zero past the matrix)
__device__ __forceinline__ void f32_load_codes(const F32Params& p, int o, int n, uint32_t (&r)[3]) {
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    r[b] = 0;
    if (8 * o < p.Kc) {
      const uint8_t* src = p.q + ((size_t)o * 3 + b) * p.N + n;
      if (p.aligned_q) {
        if (n < p.N) r[b] = __ldg(reinterpret_cast<const uint32_t*>(src));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) r[b] |= (uint32_t)src[j] << (8 * j);
      }
    }
  }
}

// TT = token tiles of 8 rows of x per sweep over the weights
template <int TT>
__global__ void __launch_bounds__(F32_THREADS, 2) matvec_f32_kernel(const F32Params p) {
  constexpr int TOK = 8 * TT, NTILE = 4 * TT;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_cta = blockIdx.y * F32_COLS;

  if ((int)blockIdx.x >= p.n_parts) {
    // cherry columns: one output column per thread
    float* xs = reinterpret_cast<float*>(smem);             // [64 cherry columns][TOK]
    const int n = n_cta + tid;
    for (int m0 = 0; m0 < p.M; m0 += TOK) {
      float acc[TOK];
#pragma unroll
      for (int t = 0; t < TOK; ++t) acc[t] = 0.f;
      for (int c0 = 0; c0 < p.C; c0 += 64) {
        const int len = min(64, p.C - c0);
        __syncthreads();
        for (int i = tid; i < len * TOK; i += F32_THREADS) {
          const int t = i / len, c = i - t * len;
          xs[c * TOK + t] = m0 + t < p.M ? p.x[(size_t)(m0 + t) * p.K + p.idx[c0 + c]] : 0.f;
        }
        __syncthreads();
        if (n < p.N)
          for (int c = 0; c < len; ++c) {
            const float wv = __ldg(p.cw + (size_t)(c0 + c) * p.N + n);
#pragma unroll
            for (int t = 0; t < TOK; ++t) acc[t] += wv * xs[c * TOK + t];
          }
      }
      if (n < p.N) {
#pragma unroll
        for (int t = 0; t < TOK; ++t)
          if (m0 + t < p.M) atomicAdd(p.mul + (size_t)(m0 + t) * p.N + n, acc[t]);
      }
    }
    return;
  }

  const int b0 = blockIdx.x * p.blk_per_part, nb = min(p.blk_per_part, p.n_blk - b0);
  // [block][chunk of 32 columns][plane][token tile][lane][8 B], then per block and token: step factors, sums, flags
  uint2* planes = reinterpret_cast<uint2*>(smem);
  float2* step = reinterpret_cast<float2*>(smem + (size_t)p.blk_per_part * 4 * NTILE * 256);    // [block][2 halves][TOK]
  int2* qsum = reinterpret_cast<int2*>(step + p.blk_per_part * 2 * TOK);                        // the same
  int* bad = reinterpret_cast<int*>(qsum + p.blk_per_part * 2 * TOK);                           // the same
  const int halves = p.G == 64 ? 2 : 1;
  const int g = lane >> 2, c = lane & 3;
  const int n = n_cta + warp * 32 + 4 * g;                  // this thread's four columns

  for (int m0 = 0; m0 < p.M; m0 += TOK) {
    __syncthreads();
    // ---- staging: a half-warp per (token, block), a lane per octet
    const int l16 = lane & 15;
    for (int it = warp * 2 + (lane >> 4); it < ((nb * TOK + 15) & ~15); it += F32_THREADS / 16) {
      const int j = it / TOK, t = it - j * TOK;
      const bool live = it < nb * TOK;
      const int kc = (b0 + j) * 128 + 8 * l16;
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.f;
      if (live && m0 + t < p.M && kc < p.Kc) {
        const float* xr = p.x + (size_t)(m0 + t) * p.K;
        int low = f32_source_col(p, kc) - kc;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          while (low < p.C && p.idx[low] - low <= kc + e) ++low;
          v[e] = __ldg(xr + kc + e + low);
        }
      }
      uint32_t mx = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) mx = max(mx, __float_as_uint(v[e]) & 0x7FFFFFFFu);
#pragma unroll
      for (int d = 4; d; d >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      const uint32_t mx2 = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      if (halves == 1) mx = mx2;                            // one step for the block, or one for each of its two groups
      const bool finite = mx < 0x7F800000u;
      // power of two at the largest value (subnormals count as 2^-126), less 29
      const int e2 = max((int)(mx >> 23), 1) - 127 - 29;
      const float2 up = f32_pow2_pair(-e2);
      int qv[8], hi = 0, lo = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) qv[e] = finite ? __float2int_rn(v[e] * up.x * up.y) : 0;
      uint32_t pl[4][2] = {};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        int r = qv[e];
        int d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          d[k] = k < 3 ? (int)(signed char)(r & 0xFF) : r;
          r = (r - d[k]) >> 8;
          pl[k][e >> 2] |= (uint32_t)(d[k] & 0xFF) << (8 * (e & 3));
        }
        hi += d[3] * 256 + d[2];
        lo += d[1] * 256 + d[0];
      }
#pragma unroll
      for (int d = 4; d; d >>= 1) {
        hi += __shfl_xor_sync(0xffffffffu, hi, d);
        lo += __shfl_xor_sync(0xffffffffu, lo, d);
      }
      if (live) {
        const int ch = l16 >> 2, dst = 4 * (t & 7) + (l16 & 3);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          planes[((size_t)(j * 4 + ch) * NTILE + k * TT + (t >> 3)) * 32 + dst] = make_uint2(pl[k][0], pl[k][1]);
        if ((l16 & 7) == 0) {
          const int at = (j * 2 + (l16 >> 3)) * TOK + t;
          qsum[at] = make_int2(hi, lo);
          step[at] = f32_pow2_pair(e2);
          bad[at] = finite ? 0 : 1;
        }
      }
    }
    __syncthreads();

    float y[4][TT][2];                                      // [column][token tile][token 2c, 2c + 1]
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int t = 0; t < TT; ++t) y[j][t][0] = y[j][t][1] = 0.f;
    uint32_t nxt[4][3];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) f32_load_codes(p, b0 * 16 + ch * 4 + c, n, nxt[ch]);
    for (int j = 0; j < nb; ++j) {
      int acc[2][NTILE][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < NTILE; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][k][e] = 0;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t r[3] = {nxt[ch][0], nxt[ch][1], nxt[ch][2]};
        if (j + 1 < nb) f32_load_codes(p, (b0 + j + 1) * 16 + ch * 4 + c, n, nxt[ch]);
        uint32_t a[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // the 24 bits of column i's octet, codes 0..3 and 4..7 spread to bytes
          const uint32_t two = __byte_perm(r[0], r[1], (uint32_t)i | ((uint32_t)(4 + i) << 4));
          const uint32_t w = __byte_perm(two, r[2], 0x0010u | ((uint32_t)(4 + i) << 8) | 0x3000u);
          a[i >> 1][i & 1] = (w & 0x7u) | ((w << 5) & 0x700u) | ((w << 10) & 0x70000u) | ((w << 15) & 0x7000000u);
          a[i >> 1][2 + (i & 1)] = ((w >> 12) & 0x7u) | ((w >> 7) & 0x700u) | ((w >> 2) & 0x70000u) | ((w << 3) & 0x7000000u);
        }
#pragma unroll
        for (int k = 0; k < NTILE; ++k) {
          const uint2 b = planes[((size_t)(j * 4 + ch) * NTILE + k) * 32 + lane];
          imma(acc[0][k], a[0], b);
          imma(acc[1][k], a[1], b);
        }
        if (ch == 3 || (ch == 1 && halves == 2)) {
          // end of a scale group (or of the block): exact integer sums -> fp32
          const int grp = ((b0 + j) * 128 + (halves == 2 ? 64 * (ch >> 1) : 0)) / p.G;
          float s[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) s[i] = 0.f;
          if ((size_t)grp * p.G < (size_t)p.Kc) {
            const float* sp = p.sf + (size_t)grp * p.N + n;
            if (p.aligned_f && n < p.N) {
              const float4 f = __ldg(reinterpret_cast<const float4*>(sp));
              s[0] = f.x; s[1] = f.y; s[2] = f.z; s[3] = f.w;
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (n + i < p.N) s[i] = __ldg(sp + i);
            }
          }
#pragma unroll
          for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int tok = 8 * t + 2 * c + e;
              const int at = (j * 2 + (halves == 2 ? ch >> 1 : 0)) * TOK + tok;
              int2 qs = qsum[at];
              if (halves == 1) {
                const int2 q2 = qsum[(j * 2 + 1) * TOK + tok];
                qs.x += q2.x;
                qs.y += q2.y;
              }
              const float2 st = step[at];
              const float f1 = 0.5f * st.x;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int ei = 2 * (i & 1) + e;
                const int hi = acc[i >> 1][3 * TT + t][ei] * 256 + acc[i >> 1][2 * TT + t][ei];
                const int lo = acc[i >> 1][TT + t][ei] * 256 + acc[i >> 1][t][ei];
                const float v = __fmaf_rn((float)(2 * hi - 7 * qs.x), 65536.f, (float)(2 * lo - 7 * qs.y));
                y[i][t][e] += v * f1 * s[i] * st.y;
              }
              if (bad[at]) {
                // an infinite or NaN activation among them: the plain sum over the group
                const int o0 = (b0 + j) * 16 + (halves == 2 ? 8 * (ch >> 1) : 0), o1 = o0 + (halves == 2 ? 8 : 16);
                for (int i = 0; i < 4; ++i) {
                  if (n + i >= p.N) break;
                  float part = 0.f;
                  for (int o = o0; o < o1 && 8 * o < p.Kc; ++o) {
                    const uint8_t* src = p.q + (size_t)o * 3 * p.N + n + i;
                    const uint32_t w = src[0] | ((uint32_t)src[p.N] << 8) | ((uint32_t)src[2 * (size_t)p.N] << 16);
                    for (int b = 0; b < 8; ++b)
                      part += ((float)((w >> (3 * b)) & 7u) - 3.5f) * p.x[(size_t)(m0 + tok) * p.K + f32_source_col(p, 8 * o + b)];
                  }
                  y[i][t][e] += s[i] * part;
                }
              }
            }
          if (halves == 2 && ch == 1) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int k = 0; k < NTILE; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][k][e] = 0;
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < TT; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tok = m0 + 8 * t + 2 * c + e;
        if (tok < p.M && n < p.N) {
          float* dst = p.mul + (size_t)tok * p.N + n;
          if (p.aligned_f) {
            atomicAdd(reinterpret_cast<float4*>(dst), make_float4(y[0][t][e], y[1][t][e], y[2][t][e], y[3][t][e]));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n + i < p.N) atomicAdd(dst + i, y[i][t][e]);
          }
        }
      }
  }
}

}  // namespace

// Host launcher used by cq_vecquant3matmul_cherryq (fp16 == 0).
int cq_launch_matvec_f32(const float* x, const uint8_t* q, const float* cw, const int32_t* idx, const float* sf, float* mul,
                         int M, int K, int N, int C, int G, cudaStream_t st) {
  F32Params p;
  p.x = x; p.q = q; p.cw = cw; p.idx = idx; p.sf = sf; p.mul = mul;
  p.M = M; p.K = K; p.N = N; p.C = C; p.G = G; p.Kc = K - C;
  p.n_blk = (p.Kc + 127) / 128;
  // Blocks per CTA: the split whose waves of two CTAs per SM take the fewest block times (a CTA's fixed part, x staging
  // set-up and the atomics, counts as one).  4096 x 13824, 16 rows: 8 blocks, one wave of 270.
  const int ny = (N + F32_COLS - 1) / F32_COLS;
  const int slots = 2 * cq_sm_count();
  int per = 1;
  long long best = 0;
  for (int b = 1; b <= F32_MAX_BLOCKS; ++b) {
    const long long ctas = (long long)ny * ((p.n_blk + b - 1) / b + (C > 0 ? 1 : 0));
    const long long t = (ctas + slots - 1) / slots * (b + 1);
    if (b == 1 || t < best) {
      best = t;
      per = b;
    }
  }
  p.blk_per_part = per;
  p.n_parts = (p.n_blk + per - 1) / per;
  p.aligned_q = N % 4 == 0 && ((uintptr_t)q & 3) == 0;
  p.aligned_f = N % 4 == 0 && ((uintptr_t)sf & 15) == 0 && ((uintptr_t)mul & 15) == 0;
  const int tt = M > 8 ? 2 : 1;
  const int smem_main = per * (4 * 4 * tt * 256 + 8 * tt * (16 + 16 + 8)), smem_cherry = 64 * 8 * tt * 4;
  const int smem = smem_main > smem_cherry ? smem_main : smem_cherry;
  const dim3 grid(p.n_parts + (C > 0 ? 1 : 0), ny);
  auto kernel = tt == 2 ? matvec_f32_kernel<2> : matvec_f32_kernel<1>;
  CQ_CUDA_TRY(cq_grant_smem((const void*)kernel, smem));
  kernel<<<grid, F32_THREADS, smem, st>>>(p);
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}
