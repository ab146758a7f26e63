// Fake quantisation of a training-side weight (llama/cherry_linear.py:69-99 and llama/quantizer.py:148-170 of the
// reference project): cherry columns keep their value, the other columns - compacted, in groups of G - become
// (round(clamp(w / s) - 0.5) + 0.5) * s with s = (max|w| + 1e-6) / 2^(bits-1) of their group, every step rounded to
// the weight's type as the element-wise torch expressions round it.  With `ste` the result is (real - w) + w, the
// value of the straight-through expression.
//
// Bound: HBM, one read and one write of the matrix; the chain of torch operations moves it about twenty times.  The order of
// the columns never changes, so there is no gather: a table made once per call gives every octet of columns its group, the
// columns of it that are quantised, and those of them that belong to the next group.
//   16-bit weights: a block goes down the rows.  One sweep takes the group maxima, the second re-reads the row from L1 and
//   writes.  Both run on packed pairs, rounded as the expressions round, and treat every octet as one whole group's; the
//   few others (a cherry column or a group's end inside) are on a list and are done apart, so that they do not hold up
//   the warps.  4096 x 11008 bf16: 111 us element by element (73 instructions a weight, bound by the issue rate).
//   fp32 weights: element by element, a block a row.
#include <cuda_bf16.h>

#include <type_traits>

#include "cq_common.cuh"

namespace {

constexpr int FQ_THREADS = 256;

// table[o] = group of octet o's first quantised column << 16 | mask of the columns of the next group << 8 | mask of all
// quantised columns (G >= 8: an octet has two groups at most)
__global__ void __launch_bounds__(1024) fq_table_kernel(const uint8_t* __restrict__ quantised, int n_oct, int G, int ng,
                                                        uint32_t* __restrict__ table) {
  __shared__ uint32_t warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n_oct + 1023) / 1024, o0 = min(n_oct, tid * per), o1 = min(n_oct, o0 + per);
  auto mask_of = [&](int o) {
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) m |= (quantised[8 * (size_t)o + e] ? 1u : 0u) << e;
    return m;
  };
  uint32_t sum = 0;
  for (int o = o0; o < o1; ++o) sum += __popc(mask_of(o));
  uint32_t inc = sum;
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += v;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  uint32_t rank = inc - sum;
  for (int w = 0; w < warp; ++w) rank += warp_sum[w];
  for (int o = o0; o < o1; ++o) {
    const uint32_t m = mask_of(o);
    const uint32_t g = min(rank / (uint32_t)G, (uint32_t)(ng - 1)), rest = (g + 1) * G - rank;
    uint32_t next = rest < 8 ? m : 0u;
    for (uint32_t i = 0; i < rest && next; ++i) next &= next - 1;
    table[o] = (g << 16) | (next << 8) | m;
    rank += __popc(m);
  }
}

// ------------------------------------------------------------------ 16-bit weights, in packed pairs
// (explicit roundings: nothing is contracted into a fused multiply-add)
#define FQ_OP2(name, instr)                                                       \
  static __device__ __forceinline__ uint32_t name(uint32_t a, uint32_t b) {      \
    uint32_t d;                                                                   \
    asm(instr " %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));                         \
    return d;                                                                     \
  }
template <typename T> struct FqPair;
template <> struct FqPair<__half> {
  static constexpr uint32_t HALF = 0x38003800u, MAGIC = 0x66006600u;     // 0.5; 1536: a sum up to 8.5 away is an integer
  FQ_OP2(add, "add.rn.f16x2")
  FQ_OP2(sub, "sub.rn.f16x2")
  FQ_OP2(mul, "mul.rn.f16x2")
  FQ_OP2(max, "max.NaN.f16x2")
  FQ_OP2(min, "min.NaN.f16x2")
  static __device__ __forceinline__ float2 widen(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
  static __device__ __forceinline__ uint32_t narrow(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};
template <> struct FqPair<__nv_bfloat16> {
  static constexpr uint32_t HALF = 0x3F003F00u, MAGIC = 0x43404340u;     // 0.5; 192
  FQ_OP2(add, "add.rn.bf16x2")
  FQ_OP2(sub, "sub.rn.bf16x2")
  FQ_OP2(mul, "mul.rn.bf16x2")
  FQ_OP2(max, "max.NaN.bf16x2")
  FQ_OP2(min, "min.NaN.bf16x2")
  static __device__ __forceinline__ float2 widen(uint32_t u) {
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
  }
  static __device__ __forceinline__ uint32_t narrow(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};
#undef FQ_OP2

// A pair of weights quantised with a scale (twice in s2; r = RN(1 / s)), before the straight-through expression.  The
// quotients: an fp32 product with r is within 2^-23 of the quotient, and no quotient of two 11-bit (8-bit) significands
// is that close to a midpoint of two normal numbers of the type; quotients below the normal numbers leave -0.5 or what is
// next to it after the subtraction, either way.  Every other step is one rounding of an exact sum or product, as in the
// expressions (fp32 holds the exact result of each; differences so wide apart that it does not are no midpoints).
template <typename T> __device__ __forceinline__ uint32_t fq_pair(uint32_t w, float r, uint32_t s2, uint32_t lim2) {
  using F = FqPair<T>;
  const float2 v = F::widen(w);
  uint32_t q = F::narrow(__fmul_rn(v.x, r), __fmul_rn(v.y, r));
  q = F::min(F::max(q, lim2 ^ 0x80008000u), lim2);
  q = F::sub(q, F::HALF);
  q = F::sub(F::add(q, F::MAGIC), F::MAGIC);
  return F::mul(F::add(q, F::HALF), s2);
}
template <typename T> __device__ __forceinline__ uint32_t fq_through(uint32_t q, uint32_t w, int ste) {
  return ste ? FqPair<T>::add(FqPair<T>::sub(q, w), w) : q;
}
// bits e and e + 1 of m as halves of ones
__device__ __forceinline__ uint32_t fq_halves(uint32_t m, int e) {
  return ((m >> e) & 1u ? 0xFFFFu : 0u) | ((m >> e) & 2u ? 0xFFFF0000u : 0u);
}
// the larger half as the bits of an fp32 number (NaN above all)
template <typename T> __device__ __forceinline__ uint32_t fq_larger(uint32_t u) {
  const float2 f = FqPair<T>::widen(u);
  return max(__float_as_uint(f.x), __float_as_uint(f.y));
}

constexpr int FQ_LIST = 1024;                // octets on the list; more are done among the others

// FQ_ROWS rows a turn: one look at the table for all, their loads in flight together.
template <typename T, int FQ_ROWS>
__global__ void __launch_bounds__(FQ_THREADS, 4) fake_quant_pairs_kernel(const T* __restrict__ w, const uint32_t* __restrict__ table,
                                                                         int bits, int K, int N, int ng, int ste, T* __restrict__ out) {
  using F = FqPair<T>;
  extern __shared__ __align__(8) uint32_t fq_smem[];
  uint2* scale = reinterpret_cast<uint2*>(fq_smem);           // [FQ_ROWS][ng] scale as a pair, 1 / scale
  uint32_t* gmax = fq_smem + 2 * FQ_ROWS * ng;                // [FQ_ROWS][ng] bits of the group maxima; zero between turns
  __shared__ int list[FQ_LIST], s_n;
  const int tid = threadIdx.x, lane = tid & 31, n_oct = K >> 3;
  auto whole = [](uint32_t t) { return (t & 0xFFFFu) == 0xFFu; };
  if (tid == 0) s_n = 0;
  for (int g = tid; g < FQ_ROWS * ng; g += FQ_THREADS) gmax[g] = 0u;
  __syncthreads();
  // (an octet a thread and one row: a list costs more than it saves)
  bool listed = FQ_ROWS > 1 || n_oct > FQ_THREADS;
  if (listed) {
    for (int o = tid; o < n_oct; o += FQ_THREADS)
      if (!whole(table[o])) {
        const int at = atomicAdd(&s_n, 1);
        if (at < FQ_LIST) list[at] = o;
      }
    __syncthreads();
    listed = s_n <= FQ_LIST;
  }
  const int n_list = listed ? s_n : 0;
  const float inv = 1.f / (float)(1 << (bits - 1));           // a power of two: the product is the quotient
  const uint32_t lim2 = F::narrow((float)((double)(1 << (bits - 1)) - 1e-2), (float)((double)(1 << (bits - 1)) - 1e-2));
  constexpr uint32_t ABS = 0x7FFF7FFFu;

  for (int n = blockIdx.x * FQ_ROWS; n < N; n += gridDim.x * FQ_ROWS) {
    const int rows = min(FQ_ROWS, N - n);
    const uint4* row[FQ_ROWS];                                // (rows past the matrix repeat its last one)
#pragma unroll
    for (int r = 0; r < FQ_ROWS; ++r) row[r] = reinterpret_cast<const uint4*>(w + (size_t)(n + min(r, rows - 1)) * K);
    // f(row, octet, table entry) for the listed octets, and of one that is not on a list
    auto others = [&](auto f) {
      for (int i = tid; i < n_list * FQ_ROWS; i += FQ_THREADS) {
        const int o = list[i / FQ_ROWS], r = i % FQ_ROWS;
        if (r < rows) f(r, o, table[o]);
      }
    };
    auto in_place = [&](int o, uint32_t t, auto f) {
      if (listed) return;
#pragma unroll 1
      for (int r = 0; r < rows; ++r) f(r, o, t);
    };
    auto take_max = [&](int r, int o, uint32_t t) {
      const uint4 v = reinterpret_cast<const uint4*>(w + (size_t)(n + r) * K)[o];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w}, next = (t >> 8) & 0xFFu, own = t & 0xFFu & ~next;
      uint32_t a = 0, b = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a = F::max(a, u[i] & ABS & fq_halves(own, 2 * i));
        b = F::max(b, u[i] & ABS & fq_halves(next, 2 * i));
      }
      if (own) atomicMax(&gmax[r * ng + (t >> 16)], fq_larger<T>(a));
      if (next) atomicMax(&gmax[r * ng + (t >> 16) + 1], fq_larger<T>(b));
    };
    auto write = [&](int r, int o, uint32_t t) {
      const uint4 v = reinterpret_cast<const uint4*>(w + (size_t)(n + r) * K)[o];
      const uint32_t next = (t >> 8) & 0xFFu, own = t & 0xFFu & ~next;
      const uint2 s0 = scale[r * ng + (t >> 16)], s1 = next ? scale[r * ng + (t >> 16) + 1] : s0;
      uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t a = fq_halves(own, 2 * i), b = fq_halves(next, 2 * i);
        uint32_t q = u[i] & ~(a | b);                             // cherry columns keep their value
        q |= fq_pair<T>(u[i], __uint_as_float(s0.y), s0.x, lim2) & a;
        q |= fq_pair<T>(u[i], __uint_as_float(s1.y), s1.x, lim2) & b;
        u[i] = fq_through<T>(q, u[i], ste);
      }
      reinterpret_cast<uint4*>(out + (size_t)(n + r) * K)[o] = make_uint4(u[0], u[1], u[2], u[3]);
    };
    // ---- group maxima
    for (int o0 = tid & ~31; o0 < n_oct; o0 += FQ_THREADS) {
      const int o = o0 + lane;
      uint32_t m[FQ_ROWS] = {};
      int g = 0x7fffffff;
      if (o < n_oct) {
        const uint32_t t = table[o];
        uint4 v[FQ_ROWS];
#pragma unroll
        for (int r = 0; r < FQ_ROWS; ++r) v[r] = row[r][o];
        if (whole(t)) {
          g = (int)(t >> 16);
#pragma unroll
          for (int r = 0; r < FQ_ROWS; ++r)
            m[r] = fq_larger<T>(F::max(F::max(v[r].x & ABS, v[r].y & ABS), F::max(v[r].z & ABS, v[r].w & ABS)));
        } else {
          in_place(o, t, take_max);
        }
      }
      // one maximum per group and warp
      const int g_lo = __reduce_min_sync(0xffffffffu, g), g_hi = __reduce_max_sync(0xffffffffu, g == 0x7fffffff ? -1 : g);
      for (int q = g_lo; q <= g_hi; ++q) {
        uint32_t top = 0;                                     // lane r: row r's
#pragma unroll
        for (int r = 0; r < FQ_ROWS; ++r) {
          const uint32_t x = __reduce_max_sync(0xffffffffu, g == q ? m[r] : 0u);
          if (lane == r) top = x;
        }
        if (lane < FQ_ROWS && top) atomicMax(&gmax[lane * ng + q], top);
      }
    }
    others(take_max);
    __syncthreads();
    // ---- scales
    for (int g = tid; g < FQ_ROWS * ng; g += FQ_THREADS) {
      const float a = F::widen(F::narrow(__fadd_rn(__uint_as_float(gmax[g]), 1e-6f), 0.f)).x;
      const uint32_t s2 = F::narrow(__fmul_rn(a, inv), __fmul_rn(a, inv));
      scale[g] = make_uint2(s2, __float_as_uint(__frcp_rn(F::widen(s2).x)));
      gmax[g] = 0u;
    }
    __syncthreads();
    // ---- weights
    for (int o = tid; o < n_oct; o += FQ_THREADS) {
      const uint32_t t = table[o];
      if (!whole(t)) {
        in_place(o, t, write);
        continue;
      }
      uint4 v[FQ_ROWS];
#pragma unroll
      for (int r = 0; r < FQ_ROWS; ++r) v[r] = row[r][o];
      uint4* dst = reinterpret_cast<uint4*>(out + (size_t)n * K) + o;
#pragma unroll
      for (int r = 0; r < FQ_ROWS; ++r) {
        const uint2 sc = scale[r * ng + (t >> 16)];
        const float x = __uint_as_float(sc.y);
        v[r].x = fq_through<T>(fq_pair<T>(v[r].x, x, sc.x, lim2), v[r].x, ste);
        v[r].y = fq_through<T>(fq_pair<T>(v[r].y, x, sc.x, lim2), v[r].y, ste);
        v[r].z = fq_through<T>(fq_pair<T>(v[r].z, x, sc.x, lim2), v[r].z, ste);
        v[r].w = fq_through<T>(fq_pair<T>(v[r].w, x, sc.x, lim2), v[r].w, ste);
        if (r < rows) *dst = v[r];
        dst += n_oct;
      }
    }
    others(write);
  }
}

// ------------------------------------------------------------------ fp32 weights
// minimum and maximum that keep NaN, as torch.clamp does
__device__ __forceinline__ float clamp_nan(float v, float lim) {
  float r;
  asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, %2;\n\tmin.NaN.f32 %0, t, %3;\n\t}" : "=f"(r) : "f"(v), "f"(-lim), "f"(lim));
  return r;
}
// nearest integer, ties to even, of |v| <= 2^21 (NaN stays NaN)
__device__ __forceinline__ float nearest(float v) { return __fsub_rn(__fadd_rn(v, 12582912.f), 12582912.f); }

__global__ void __launch_bounds__(FQ_THREADS) fake_quant_kernel(const float* __restrict__ w, const uint32_t* __restrict__ table,
                                                                int bits, int K, int ng, int ste, float* __restrict__ out) {
  extern __shared__ uint32_t gmax[];          // bits of the group maxima, then of the scales
  const int tid = threadIdx.x, lane = tid & 31, n_oct = K >> 3;
  const float* row = w + (size_t)blockIdx.x * K;
  float* dst = out + (size_t)blockIdx.x * K;
  for (int g = tid; g < ng; g += FQ_THREADS) gmax[g] = 0u;
  __syncthreads();
  auto load = [&](int o, float* v) {
    const float4 a = *reinterpret_cast<const float4*>(row + 8 * o), b = *reinterpret_cast<const float4*>(row + 8 * o + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  };
  for (int o0 = (tid >> 5) * 32; o0 < n_oct; o0 += FQ_THREADS) {
    const int o = o0 + lane;
    uint32_t m0 = 0, m1 = 0;                  // maxima as bits: integer order is that of |w|, NaN above all
    int g = 0x7fffffff;
    if (o < n_oct) {
      float v[8];
      load(o, v);
      const uint32_t t = table[o];
      g = (int)(t >> 16);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t a = __float_as_uint(v[e]) & 0x7FFFFFFFu;
        if ((t >> (8 + e)) & 1u) m1 = max(m1, a);
        else if ((t >> e) & 1u) m0 = max(m0, a);
      }
    }
    // one maximum per group and warp
    const int g_lo = __reduce_min_sync(0xffffffffu, g);
    const int g_hi = __reduce_max_sync(0xffffffffu, g == 0x7fffffff ? -1 : (m1 ? g + 1 : g));
    for (int q = g_lo; q <= g_hi; ++q) {
      const uint32_t r = __reduce_max_sync(0xffffffffu, g == q ? m0 : (g + 1 == q ? m1 : 0u));
      if (lane == 0 && q < ng && r) atomicMax(&gmax[q], r);
    }
  }
  __syncthreads();
  const float inv = 1.f / (float)(1 << (bits - 1));           // a power of two: the product is the quotient
  for (int g = tid; g < ng; g += FQ_THREADS) gmax[g] = __float_as_uint(__fmul_rn(__fadd_rn(__uint_as_float(gmax[g]), 1e-6f), inv));
  __syncthreads();
  const float lim = (float)((double)(1 << (bits - 1)) - 1e-2);
  for (int o = tid; o < n_oct; o += FQ_THREADS) {
    float v[8];
    load(o, v);
    const uint32_t t = table[o], sec = (t >> 8) & 0xFFu;
    const float s0 = __uint_as_float(gmax[t >> 16]), s1 = sec ? __uint_as_float(gmax[(t >> 16) + 1]) : s0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s = (sec >> e) & 1u ? s1 : s0;
      float q = __fsub_rn(clamp_nan(__fdiv_rn(v[e], s), lim), 0.5f);
      q = __fmul_rn(__fadd_rn(nearest(q), 0.5f), s);
      if (!((t >> e) & 1u)) q = v[e];
      v[e] = ste ? __fadd_rn(__fsub_rn(q, v[e]), v[e]) : q;
    }
    *reinterpret_cast<float4*>(dst + 8 * o) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + 8 * o + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
}

}  // namespace

extern "C" int cq_fake_quant(const void* weight, int dtype, const uint8_t* quantised, int bits, int K, int N, int G, int ste,
                             void* out, uint32_t* table, cq_stream_t stream) {
  if (!weight || !quantised || !out || !table) return CQ_ERR_BAD_ARG;
  if (((uintptr_t)weight & 15) || ((uintptr_t)out & 15)) return CQ_ERR_BAD_ARG;
  if (bits < 2 || bits > 4) return CQ_ERR_BAD_BITS;
  if (K <= 0 || N <= 0 || K % 8 || K >= (1 << 24)) return CQ_ERR_BAD_SHAPE;
  if (G < 8) return CQ_ERR_BAD_GROUP;
  if (G > K) G = K;
  const int ng = (K + G - 1) / G;
  if ((size_t)ng * 4 > 48 * 1024) return CQ_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype < 0 || dtype > 2) return CQ_ERR_BAD_ARG;
  fq_table_kernel<<<1, 1024, 0, st>>>(quantised, K / 8, G, ng, table);
  if (dtype == 1) {
    fake_quant_kernel<<<N, FQ_THREADS, (size_t)ng * 4, st>>>((const float*)weight, table, bits, K, ng, ste, (float*)out);
  } else {
    // Rows a turn: as many as leave the chip blocks enough, and whose groups fit shared memory comfortably.  4096 x 4096 bf16, one,
    // two and four rows a turn: 33.4, 25.1 and 22.4 us (element by element 45.2); 1024 x 2048 13.0, 9.6 and 7.8 (10.5); 2048 x
    // 1024 9.9, 7.9 and 8.0 (9.7); 4096 x 256 8.2, 8.3 and 9.2 (8.3).  Two waves of blocks at most, each of which makes its list
    // once and goes down the rows.
    const int blocks = 8 * cq_sm_count(), rows = ng > 1000 ? 1 : (N >= blocks ? 4 : (2 * N >= blocks ? 2 : 1));
    const int smem = rows * ng * 12, turns = (N + rows - 1) / rows;
    auto launch = [&](auto kernel, auto* wp, auto* op) -> int {
      CQ_CUDA_TRY(cq_grant_smem((const void*)kernel, smem));
      kernel<<<turns < blocks ? turns : blocks, FQ_THREADS, smem, st>>>(wp, table, bits, K, N, ng, ste, op);
      return CQ_OK;
    };
    auto pick = [&](auto* wp, auto* op) {
      using T = std::remove_pointer_t<decltype(op)>;
      return rows == 4   ? launch(fake_quant_pairs_kernel<T, 4>, wp, op)
             : rows == 2 ? launch(fake_quant_pairs_kernel<T, 2>, wp, op)
                         : launch(fake_quant_pairs_kernel<T, 1>, wp, op);
    };
    const int rc = dtype == 0 ? pick((const __half*)weight, (__half*)out) : pick((const __nv_bfloat16*)weight, (__nv_bfloat16*)out);
    if (rc != CQ_OK) return rc;
  }
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}
