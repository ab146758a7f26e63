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
// thread that uses it.  That case: 32 us a call (93 with the loop; 52 while every 256 columns staged x for themselves, with a
// search for each octet's columns and a digit at a time, and codes were spread to bytes column by column: 1640 instructions
// a warp and block of 128 columns).  Bound by its instructions still (54 % of the issue slots busy with 16 warps).  512 columns share the staging, the columns are searched
// once, the four digits of a value are one addition and one exclusive or, codes are taken out for four columns at once and
// turned; four cherry columns' loads are in flight (one after another a column took 0.5 us).  Other sizes, before and now: 1 row 33 and 21 us, 64 rows 190 and 103, 16384 x 28672 317 and 208, 1024 x 1024
// 8.8 and 8.7; groups of 64 16 rows 58 and 32, 64 rows 221 and 117 (more than 8 rows: 20 bytes of registers spilled).
#include <algorithm>

#include "cq_common.cuh"

namespace {

constexpr int F32_THREADS = 512;       // 16 warps, 32 output columns each
constexpr int F32_COLS = 512;
constexpr int F32_MAX_BLOCKS = 16;     // 128-column blocks a CTA stages
constexpr int F32_DIGITS = 0x808080;   // added to a value, then exclusive or: its bytes are signed digits

struct F32Params {
  const float* x;
  const uint8_t* q;
  const float* cw;
  const int32_t* idx;
  const float* sf;
  float* mul;
  int M, K, N, C, G, Kc, n_blk, blk_per_part, n_parts, cherry_parts, aligned_q, aligned_f;
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

template <bool FIRST> __device__ __forceinline__ void imma(int (&d)[4], const uint32_t (&a)[4], uint2 b) {
  if (FIRST) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "r"(0));
    return;
  }
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

// four words with a byte of each of four columns -> a word of each column
__device__ __forceinline__ void f32_turn(const uint32_t* r, uint32_t (&v)[4]) {
  const uint32_t p0 = __byte_perm(r[0], r[1], 0x5140), p1 = __byte_perm(r[0], r[1], 0x7362);
  const uint32_t p2 = __byte_perm(r[2], r[3], 0x5140), p3 = __byte_perm(r[2], r[3], 0x7362);
  v[0] = __byte_perm(p0, p2, 0x5410);
  v[1] = __byte_perm(p0, p2, 0x7632);
  v[2] = __byte_perm(p1, p3, 0x5410);
  v[3] = __byte_perm(p1, p3, 0x7632);
}

// The plain sum of column n over octets o0 .. o1 of row m, whose columns are at source[0 ..]: where an activation among
// them is infinite or NaN.
__device__ __noinline__ float f32_plain_sum(const F32Params& p, int n, int m, int o0, int o1, const int* source) {
  float part = 0.f;
  for (int o = o0; o < o1 && 8 * o < p.Kc; ++o, source += 8) {
    const uint8_t* src = p.q + (size_t)o * 3 * p.N + n;
    const uint32_t w = src[0] | ((uint32_t)src[p.N] << 8) | ((uint32_t)src[2 * (size_t)p.N] << 16);
#pragma unroll
    for (int b = 0; b < 8; ++b) part += ((float)((w >> (3 * b)) & 7u) - 3.5f) * p.x[(size_t)m * p.K + source[b]];
  }
  return part;
}

// TT = token tiles of 8 rows of x per sweep over the weights, HALVES = scale groups of a 128-column block (2: G = 64)
template <int TT, int HALVES>
__global__ void __launch_bounds__(F32_THREADS, 1) matvec_f32_kernel(const __grid_constant__ F32Params p) {
  constexpr int TOK = 8 * TT, NTILE = 4 * TT;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_cta = blockIdx.y * F32_COLS;
  const int b0 = blockIdx.x * p.blk_per_part, nb = min(p.blk_per_part, p.n_blk - b0);
  // [block][chunk of 32 columns][plane][token tile][lane][8 B]
  uint2* planes = reinterpret_cast<uint2*>(smem);
  // per block, half and token: -7 times the sums of the upper and lower two digits, half the first step factor, the second
  // (a first factor of 0: an activation is not finite)
  int4* meta = reinterpret_cast<int4*>(smem + (size_t)p.blk_per_part * 4 * NTILE * 256);
  int* source = reinterpret_cast<int*>(meta + p.blk_per_part * HALVES * TOK);                   // [block][128]
  int* bad = source + p.blk_per_part * 128;                                                     // [block]
  const int g = lane >> 2, c = lane & 3;
  const int n = n_cta + warp * 32 + 4 * g;                  // this thread's four columns

  for (int i = tid; i < nb * 128; i += F32_THREADS) source[i] = b0 * 128 + i < p.Kc ? f32_source_col(p, b0 * 128 + i) : 0;

  for (int m0 = 0; m0 < p.M; m0 += TOK) {
    if (tid < nb) bad[tid] = 0;
    __syncthreads();
    uint32_t nxt[4][3];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) f32_load_codes(p, b0 * 16 + ch * 4 + c, n, nxt[ch]);
    // ---- staging: a half-warp per (token, block), a lane per octet
    const int l16 = lane & 15;
    for (int it = warp * 2 + (lane >> 4); it < ((nb * TOK + 1) & ~1); it += F32_THREADS / 16) {
      const int j = it / TOK, t = it - j * TOK;
      const bool live = it < nb * TOK;
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.f;
      if (live && m0 + t < p.M && (b0 + j) * 128 + 8 * l16 < p.Kc) {
        const float* xr = p.x + (size_t)(m0 + t) * p.K;
        const int4* at = reinterpret_cast<const int4*>(source + j * 128 + 8 * l16);
        const int4 s0 = at[0], s1 = at[1];
        v[0] = __ldg(xr + s0.x); v[1] = __ldg(xr + s0.y); v[2] = __ldg(xr + s0.z); v[3] = __ldg(xr + s0.w);
        v[4] = __ldg(xr + s1.x); v[5] = __ldg(xr + s1.y); v[6] = __ldg(xr + s1.z); v[7] = __ldg(xr + s1.w);
      }
      uint32_t mx = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) mx = max(mx, __float_as_uint(v[e]) & 0x7FFFFFFFu);
#pragma unroll
      for (int d = 8 / HALVES; d; d >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      const bool finite = mx < 0x7F800000u;
      // power of two at the largest value (subnormals count as 2^-126), less 29
      const int e2 = max((int)(mx >> 23), 1) - 127 - 29;
      const float2 up = f32_pow2_pair(-e2);
      // |value| <= 2^30: four signed digits, the bytes of (value + F32_DIGITS) ^ F32_DIGITS
      uint32_t r[8];
      int hi = 0, lo = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        r[e] = (uint32_t)((finite ? __float2int_rn(v[e] * up.x * up.y) : 0) + F32_DIGITS);
        hi += (int)r[e] >> 16;
        lo += (int)(r[e] & 0xFFFFu);
        r[e] ^= (uint32_t)F32_DIGITS;
      }
      hi -= 8 * (F32_DIGITS >> 16);
      lo -= 8 * (F32_DIGITS & 0xFFFF);
#pragma unroll
      for (int d = 8 / HALVES; d; d >>= 1) {
        hi += __shfl_xor_sync(0xffffffffu, hi, d);
        lo += __shfl_xor_sync(0xffffffffu, lo, d);
      }
      if (live) {
        uint32_t pl[2][4];
        f32_turn(r, pl[0]);
        f32_turn(r + 4, pl[1]);
        const int ch = l16 >> 2, dst = 4 * (t & 7) + (l16 & 3);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          planes[((size_t)(j * 4 + ch) * NTILE + k * TT + (t >> 3)) * 32 + dst] = make_uint2(pl[0][k], pl[1][k]);
        if ((l16 & (16 / HALVES - 1)) == 0) {
          const float2 st = f32_pow2_pair(e2);
          meta[(j * HALVES + (HALVES == 2 ? l16 >> 3 : 0)) * TOK + t] =
              make_int4(-7 * hi, -7 * lo, finite ? __float_as_int(0.5f * st.x) : 0, __float_as_int(st.y));
          if (!finite) bad[j] = 1;
        }
      }
    }

    float y[4][TT][2];                                      // [column][token tile][token 2c, 2c + 1]
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int t = 0; t < TT; ++t) y[j][t][0] = y[j][t][1] = 0.f;
    auto load4 = [&](const float* row, float (&f)[4]) {     // row[n .. n + 3], zero past the matrix
      if (p.aligned_f) {
        const float4 v = n < p.N ? __ldg(reinterpret_cast<const float4*>(row + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = n + i < p.N ? __ldg(row + n + i) : 0.f;
      }
    };
    // ---- this part's share of the cherry columns
    const int share = (int)blockIdx.x - (int)gridDim.x + p.cherry_parts;
    const int c_end = share < 0 ? 0 : (int)((long long)p.C * (share + 1) / p.cherry_parts);
    constexpr int AHEAD = 4;                                // columns whose loads are in flight together
    for (int c0 = share < 0 ? 0 : (int)((long long)p.C * share / p.cherry_parts); c0 < c_end; c0 += AHEAD) {
      int col[AHEAD];
      float w[AHEAD][4], xv[AHEAD][TT][2];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) col[u] = c0 + u < c_end ? __ldg(p.idx + c0 + u) : -1;
      if (p.aligned_f) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const float4 v = n < p.N && col[u] >= 0 ? __ldg(reinterpret_cast<const float4*>(p.cw + (size_t)(c0 + u) * p.N + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
          w[u][0] = v.x; w[u][1] = v.y; w[u][2] = v.z; w[u][3] = v.w;
        }
      } else {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) w[u][i] = n + i < p.N && col[u] >= 0 ? __ldg(p.cw + (size_t)(c0 + u) * p.N + n + i) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
#pragma unroll
        for (int t = 0; t < TT; ++t)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int m = m0 + 8 * t + 2 * c + e;
            xv[u][t][e] = m < p.M && col[u] >= 0 ? __ldg(p.x + (size_t)m * p.K + col[u]) : 0.f;
          }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (col[u] >= 0) {
#pragma unroll
          for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
              for (int i = 0; i < 4; ++i) y[i][t][e] = __fmaf_rn(w[u][i], xv[u][t][e], y[i][t][e]);
        }
    }
    __syncthreads();

    for (int j = 0; j < nb; ++j) {
      int acc[2][NTILE][4];
      float s[HALVES][4];
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        const int k = (b0 + j) * 128 + 64 * h;
        if (k < p.Kc) load4(p.sf + (size_t)(k / p.G) * p.N, s[h]);
        else s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.f;
      }
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        // codes 0 .. 3 and 4 .. 7 of the octets of four columns
        const uint32_t r0 = nxt[ch][0], r1 = nxt[ch][1], r2 = nxt[ch][2];
        const uint32_t code[8] = {r0 & 0x07070707u, (r0 >> 3) & 0x07070707u, ((r0 >> 6) & 0x03030303u) | ((r1 << 2) & 0x04040404u),
                                  (r1 >> 1) & 0x07070707u, (r1 >> 4) & 0x07070707u,
                                  ((r1 >> 7) & 0x01010101u) | ((r2 << 1) & 0x06060606u), (r2 >> 2) & 0x07070707u, (r2 >> 5) & 0x07070707u};
        uint32_t front[4], back[4];
        f32_turn(code, front);
        f32_turn(code + 4, back);
        if (j + 1 < nb) f32_load_codes(p, (b0 + j + 1) * 16 + ch * 4 + c, n, nxt[ch]);
        const uint32_t a[2][4] = {{front[0], front[1], back[0], back[1]}, {front[2], front[3], back[2], back[3]}};
#pragma unroll
        for (int k = 0; k < NTILE; ++k) {
          const uint2 b = planes[((size_t)(j * 4 + ch) * NTILE + k) * 32 + lane];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (ch % (4 / HALVES) == 0) imma<true>(acc[i][k], a[i], b);
            else imma<false>(acc[i][k], a[i], b);
          }
        }
        if (ch % (4 / HALVES) == 4 / HALVES - 1) {
          // end of a scale group (or of the block): exact integer sums -> fp32
          constexpr int LAST = HALVES - 1;
          const int h = ch == 3 ? LAST : 0;
#pragma unroll
          for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int4 mt = meta[(j * HALVES + h) * TOK + 8 * t + 2 * c + e];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int ei = 2 * (i & 1) + e;
                const int hi = acc[i >> 1][3 * TT + t][ei] * 512 + (acc[i >> 1][2 * TT + t][ei] * 2 + mt.x);
                const int lo = acc[i >> 1][TT + t][ei] * 512 + (acc[i >> 1][t][ei] * 2 + mt.y);
                const float v = __fmaf_rn((float)hi, 65536.f, (float)lo);
                y[i][t][e] += v * __int_as_float(mt.z) * s[h][i] * __int_as_float(mt.w);
              }
            }
        }
      }
      if (bad[j]) {
#pragma unroll
        for (int h = 0; h < HALVES; ++h)
#pragma unroll
          for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int tok = 8 * t + 2 * c + e, o = (b0 + j) * 16 + 8 * h;
              if (meta[(j * HALVES + h) * TOK + tok].z != 0) continue;
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (n + i < p.N) y[i][t][e] += s[h][i] * f32_plain_sum(p, n + i, m0 + tok, o, o + 16 / HALVES, source + j * 128 + 64 * h);
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
    __syncthreads();
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
  // Blocks per CTA: the split whose waves of a CTA per SM take the fewest block times (a CTA's fixed part, x staging
  // set-up and the atomics, counts as one).  4096 x 13824, 16 rows: 7 blocks, one wave of 135.
  const int ny = (N + F32_COLS - 1) / F32_COLS;
  const int slots = cq_sm_count();
  int per = 1;
  long long best = 0;
  for (int b = 1; b <= F32_MAX_BLOCKS; ++b) {
    const long long ctas = (long long)ny * ((p.n_blk + b - 1) / b);
    const long long t = (ctas + slots - 1) / slots * (b + 1);
    if (b == 1 || t < best) {
      best = t;
      per = b;
    }
  }
  p.blk_per_part = per;
  p.n_parts = (p.n_blk + per - 1) / per;
  // Cherry columns (18 take a warp as long as a block): parts of their own where SMs are left, four columns each, unless they
  // are so many that they take longer there than shared by the main parts; else the last part, which may be shorter, or more
  // of the last ones where they are many.  (In every part they cost each one more rounding: 3 % more error at 1024 x 1024.  All
  // in the last part there: 10.9 us and 8.8.  11008 x 4096, 16 rows, 344 cherry columns: one part of their own 112 us, all parts
  // 28; 2048 x 2048, 512: 25 parts of their own 10.9, all parts 19.)
  const int spare = C > 0 ? std::min(slots / ny - p.n_parts, (C + 3) / 4) : 0;
  const double own = spare > 0 ? std::max((double)per, C / (18.0 * spare)) : 0.0, shared = per + 0.3 + C / (18.0 * p.n_parts);
  const int extra = spare > 0 && own <= shared ? spare : 0;
  p.cherry_parts = extra > 0 ? extra : (spare > 0 ? p.n_parts : (C <= 16 ? 1 : std::min(p.n_parts, C / per + 1)));
  p.aligned_q = N % 4 == 0 && ((uintptr_t)q & 3) == 0;
  p.aligned_f = N % 4 == 0 && ((uintptr_t)sf & 15) == 0 && ((uintptr_t)cw & 15) == 0 && ((uintptr_t)mul & 15) == 0;
  const int tt = M > 8 ? 2 : 1, halves = G == 64 ? 2 : 1;
  const int smem = per * (4 * 4 * tt * 256 + halves * 8 * tt * 16 + 128 * 4 + 4);
  const dim3 grid(p.n_parts + extra, ny);
  auto kernel = tt == 2 ? (halves == 2 ? matvec_f32_kernel<2, 2> : matvec_f32_kernel<2, 1>)
                        : (halves == 2 ? matvec_f32_kernel<1, 2> : matvec_f32_kernel<1, 1>);
  CQ_CUDA_TRY(cq_grant_smem((const void*)kernel, smem));
  kernel<<<grid, F32_THREADS, smem, st>>>(p);
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}
