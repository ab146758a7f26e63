// GPU versions of the reference's host-side layer conversion code
// (paths inside the reference project):
//   llama/qlinear.py:67-118   QuantLinear.pack    -> cq_pack
//   llama/qlinear.py:120-162  QuantLinear.unpack  -> cq_unpack_dense
//   csrc/quant_cuda_kernel.cu:838-1010 Dequantize{3,4}Normal -> cq_dequantize{3,4}_normal
// All three are bit-exact with the reference's torch arithmetic: fp16 element-wise
// operations are evaluated in fp32 and rounded once to fp16, exactly as torch does.
#include "cq_common.cuh"

namespace {

// The cherry columns are kept as 16-bit words and read as unsigned numbers (a layer may have up to 65534 columns).
// number of sorted cherry columns with idx[m] - m <= kc (compact -> original shift)
__device__ __forceinline__ int cherry_shift(const uint16_t* __restrict__ idx, int C, int kc) {
  int low = 0, high = C;
  while (low < high) {
    const int mid = (low + high) >> 1;
    if ((int)idx[mid] - mid <= kc) low = mid + 1; else high = mid;
  }
  return low;
}

__device__ __forceinline__ float load_w(const void* w, int is_f32, size_t i) {
  return is_f32 ? reinterpret_cast<const float*>(w)[i]
                : __half2float(reinterpret_cast<const __half*>(w)[i]);
}

// ------------------------------------------------------------------ pack
// llama/qlinear.py:72 — sort the cherry columns (rank sort; they are distinct).
__global__ void pack_sort_kernel(const int32_t* __restrict__ in, int C, int16_t* __restrict__ out) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
    const int v = in[c];
    int rank = 0;
    for (int m = 0; m < C; ++m) rank += (in[m] < v) || (in[m] == v && m < c);
    out[rank] = (int16_t)v;
  }
}

// llama/qlinear.py:74 — cherry_weight[c, n] = fp16(W[n, idx[c]]).
__global__ void pack_cherry_kernel(const void* __restrict__ w, int is_f32, const uint16_t* __restrict__ idx,
                                   int K, int N, int C, __half* __restrict__ cw) {
  const long long total = (long long)C * N;
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total;
       id += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(id % N), c = (int)(id / N);
    cw[id] = __float2half_rn(load_w(w, is_f32, (size_t)n * K + idx[c]));
  }
}

// llama/cherry_linear.py:69-75 + llama/quantizer.py:148-152 + llama/qlinear.py:78:
// s = fp16((max|w| + 1e-6) / 2^(bits-1)) per (row, group of the compact axis), evaluated in
// the weight dtype.  One warp per (n, group).
__global__ void pack_scales_kernel(const void* __restrict__ w, int is_f32, const uint16_t* __restrict__ idx,
                                   int bits, int K, int N, int C, int G, __half* __restrict__ scales) {
  const int Kc = K - C, ng = (Kc + G - 1) / G;
  const int lane = threadIdx.x & 31;
  const long long warp0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long id = warp0; id < (long long)ng * N; id += nwarps) {
    const int grp = (int)(id % ng), n = (int)(id / ng);
    const int k0 = grp * G, k1 = min(Kc, k0 + G);
    float mx = 0.f;
    for (int kc = k0 + lane; kc < k1; kc += 32)
      mx = fmaxf(mx, fabsf(load_w(w, is_f32, (size_t)n * K + kc + cherry_shift(idx, C, kc))));
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) {
      const float div = (float)(1 << (bits - 1));
      __half s;
      if (is_f32) {
        s = __float2half_rn(__fdiv_rn(__fadd_rn(mx, 1e-6f), div));
      } else {
        const __half a = __float2half_rn(__fadd_rn(mx, 1e-6f));   // fp16 add, rounded once
        s = __float2half_rn(__fdiv_rn(__half2float(a), div));     // fp16 divide, rounded once
      }
      scales[(size_t)grp * N + n] = s;
    }
  }
}

// llama/quantizer.py:154-158 + llama/qlinear.py:81-116: quantize 8 compact columns of one
// row and write their 3 or 4 bytes.
__global__ void pack_codes_kernel(const void* __restrict__ w, int is_f32, const uint16_t* __restrict__ idx,
                                  const __half* __restrict__ scales, int bits, int K, int N, int C,
                                  int G, uint8_t* __restrict__ q) {
  const int Kc = K - C;
  const long long total = (long long)(Kc / 8) * N;
  const float qmax = (float)((double)(1 << (bits - 1)) - 1e-2);
  const int qoff = 1 << (bits - 1);
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total;
       id += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(id % N), o = (int)(id / N);
    uint32_t word = 0;
    for (int i = 0; i < 8; ++i) {
      const int kc = 8 * o + i;
      const float wv = load_w(w, is_f32, (size_t)n * K + kc + cherry_shift(idx, C, kc));
      const float s = __half2float(scales[(size_t)(kc / G) * N + n]);
      float r = __fdiv_rn(wv, s);
      if (!is_f32) r = __half2float(__float2half_rn(r));  // fp16 / fp16 is rounded to fp16
      r = fminf(fmaxf(r, -qmax), qmax);
      const int code = (int)rintf(__fsub_rn(r, 0.5f)) + qoff;
      word |= (uint32_t)(code & ((1 << bits) - 1)) << (bits * i);
    }
    for (int b = 0; b < bits; ++b) q[((size_t)o * bits + b) * N + n] = (uint8_t)(word >> (8 * b));
  }
}

// One pass over the weights for groups of several chunks of 128 compact columns (multiples of 128, one group per row), for
// fp32 weights and for what the rule at cq_pack leaves of fp16 weights in groups of one chunk: a block owns PK_ROWS output rows of one group (two 64-wide ones), reads them once in chunks, reduces
// the maxima and writes scales and codes.  The general pair of kernels above reads the matrix twice, lanes a row
// apart, and divides per weight.  The loads are 2 bytes a lane, 64 contiguous bytes a warp, because the removed
// cherry columns leave the compact columns at any alignment; the tile turns them so that a thread quantises 32
// columns of one row and the byte stores have 32 consecutive rows a warp.  Groups of more than one chunk are read
// a second time for the codes (mostly from L2); cq_pack leaves those of few rows to the general pair.
constexpr int PK_ROWS = 64, PK_COLS = 128, PK_THREADS = 256;

template <typename T> struct PackTile;
template <> struct PackTile<__half> {
  static constexpr int STRIDE = PK_COLS + 8;        // 272 B: the 16-byte reads of 8 rows hit 8 different bank groups
  static __device__ __forceinline__ float f(__half v) { return __half2float(v); }
};
template <> struct PackTile<float> {
  static constexpr int STRIDE = PK_COLS + 4;
  static __device__ __forceinline__ float f(float v) { return v; }
};

// fp16(w / s) for fp16 w and s (held as floats), r = RN(1 / s).  One residual step after w * r (Markstein's division
// with fused multiply-add) leaves a relative error of at most 2^-24 (1 + 2^-20); a quotient of two 11-bit significands
// is never closer than 2^-23 to a midpoint of two fp16 numbers without being one exactly representable, so the fp16
// rounding is that of the exact quotient.  For an infinite s the caller passes 0 in the residual's place: the result is
// then w * 0, as w / infinity is.  An exact division per weight took half of the kernel's instructions.
__device__ __forceinline__ float div_fp16(float w, float s_residual, float r) {
  const float q = __fmul_rn(w, r);
  return __fmaf_rn(__fmaf_rn(-q, s_residual, w), r, q);
}

template <typename T, int BITS>
__global__ void __launch_bounds__(PK_THREADS, sizeof(T) == 2 ? 5 : 3) pack_fused_kernel(
    const T* __restrict__ w, const uint16_t* __restrict__ idx, int K, int N, int C, int G, int span, int n_tiles,
    int n_spans, __half* __restrict__ scales, uint8_t* __restrict__ q, __half* __restrict__ cw) {
  constexpr int ST = PackTile<T>::STRIDE, VEC = 16 / sizeof(T);
  __shared__ __align__(16) T tile[PK_ROWS * ST];
  __shared__ float red[4][PK_ROWS];
  __shared__ int source[PK_COLS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = (int)(blockIdx.x % n_tiles) * PK_ROWS, sp = (int)(blockIdx.x / n_tiles);
  const int rows = min(PK_ROWS, N - n0);
  if (sp >= n_spans) {
    // the last block of a row tile copies its cherry columns: cherry_weight[c, n] = fp16(W[n, idx[c]])
    for (int id = tid; id < C * PK_ROWS; id += PK_THREADS) {
      const int r = id % PK_ROWS, c = id / PK_ROWS;
      if (r < rows) cw[(size_t)c * N + n0 + r] = __float2half_rn(PackTile<T>::f(w[(size_t)(n0 + r) * K + idx[c]]));
    }
    return;
  }
  const int Kc = K - C;
  const int k_begin = sp * span, k_end = min(Kc, k_begin + span);
  const int n_chunks = (k_end - k_begin + PK_COLS - 1) / PK_COLS;
  const int row = tid & (PK_ROWS - 1), part = tid / PK_ROWS;      // this thread's 32 columns of the tile
  const bool two = G == 64;                                       // two groups in the block's 128 columns

  auto load_chunk = [&](int k0) {
    // lane l of every warp loads compact columns k0 + 32 j + l; rows go round over the warps
    __syncthreads();
    if (tid < PK_COLS) {
      const int kc = k0 + tid;
      source[tid] = kc < k_end ? kc + cherry_shift(idx, C, kc) : -1;
    }
    __syncthreads();
    int col[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) col[j] = source[32 * j + lane];
    const T* src = w + (size_t)(n0 + min(warp, rows - 1)) * K;
    const size_t step = (size_t)(PK_THREADS / 32) * K;
#pragma unroll 4
    for (int r = warp; r < PK_ROWS; r += PK_THREADS / 32) {
#pragma unroll
      for (int j = 0; j < 4; ++j) tile[r * ST + 32 * j + lane] = col[j] >= 0 ? src[col[j]] : (T)0.f;
      if (r + PK_THREADS / 32 < rows) src += step;               // (rows past the matrix repeat one of its rows)
    }
    __syncthreads();
  };
  uint4 raw[32 / VEC];
  auto read_part = [&]() {
#pragma unroll
    for (int i = 0; i < 32 / VEC; ++i) raw[i] = reinterpret_cast<const uint4*>(tile + row * ST + 32 * part)[i];
  };
  // two consecutive values
  auto pair = [&](int i) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(raw);
    if constexpr (sizeof(T) == 2)
      return __half22float2(*reinterpret_cast<const __half2*>(&u[i >> 1]));
    else
      return make_float2(__uint_as_float(u[i]), __uint_as_float(u[i + 1]));
  };

  float mx = 0.f;
  for (int c = 0; c < n_chunks; ++c) {
    load_chunk(k_begin + c * PK_COLS);
    read_part();
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float2 f = pair(i);
      mx = fmaxf(mx, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  red[part][row] = mx;
  __syncthreads();
  if (two)
    mx = fmaxf(red[part & 2][row], red[(part & 2) + 1][row]);
  else
    mx = fmaxf(fmaxf(red[0][row], red[1][row]), fmaxf(red[2][row], red[3][row]));
  const float div = (float)(1 << (BITS - 1));
  __half sh;
  if constexpr (sizeof(T) == 4) {
    sh = __float2half_rn(__fdiv_rn(__fadd_rn(mx, 1e-6f), div));
  } else {
    const __half a = __float2half_rn(__fadd_rn(mx, 1e-6f));       // fp16 add, rounded once
    sh = __float2half_rn(__fdiv_rn(__half2float(a), div));        // fp16 divide, rounded once
  }
  const int grp = k_begin / G + (two ? (part >> 1) : 0);
  if (row < rows && (part == 0 || (two && part == 2)) && grp < (Kc + G - 1) / G) scales[(size_t)grp * N + n0 + row] = sh;

  const float s = __half2float(sh), rs = __frcp_rn(s), s_residual = s < 65536.f ? s : 0.f;
  const float qmax = (float)((double)(1 << (BITS - 1)) - 1e-2);
  for (int c = 0; c < n_chunks; ++c) {
    const int k0 = k_begin + c * PK_COLS;
    if (n_chunks > 1) {
      load_chunk(k0);
      read_part();
    }
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      uint32_t word = 0;
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        float2 r = pair(8 * o + i);
        if constexpr (sizeof(T) == 2)                             // fp16 / fp16 is rounded to fp16
          r = __half22float2(__floats2half2_rn(div_fp16(r.x, s_residual, rs), div_fp16(r.y, s_residual, rs)));
        else
          r = make_float2(__fdiv_rn(r.x, s), __fdiv_rn(r.y, s));
        r.x = fminf(fmaxf(r.x, -qmax), qmax);
        r.y = fminf(fmaxf(r.y, -qmax), qmax);
        // adding 1.5 * 2^23 (+ the code offset) rounds to the nearest integer, ties to even, like rint
        const float magic = 12582912.f + (float)(1 << (BITS - 1));
        word |= (__float_as_uint(__fadd_rn(__fsub_rn(r.x, 0.5f), magic)) & ((1u << BITS) - 1)) << (BITS * i);
        word |= (__float_as_uint(__fadd_rn(__fsub_rn(r.y, 0.5f), magic)) & ((1u << BITS) - 1)) << (BITS * (i + 1));
      }
      const int oct = (k0 >> 3) + 4 * part + o;
      if (row < rows && 8 * oct < k_end) {
        uint8_t* dst = q + (size_t)oct * BITS * N + n0 + row;
#pragma unroll
        for (int b = 0; b < BITS; ++b) dst[(size_t)b * N] = (uint8_t)(word >> (8 * b));
      }
    }
  }
}

// fp16 weights of large matrices in groups of one chunk: a block keeps 128 compact columns, one group (two 64-wide ones); each
// of its warps goes down the rows, 32 at a time, a lane a row, without a barrier.
//   * Bound by its instructions (62 % of the issue slots busy): the kernel above executes 31 a weight, much of it set-up per 32
//     weights, this one 19.  Here the rows come in with 16-byte copies, in their original order; the removed cherry columns
//     only show when a lane takes 32 compact columns of its row from shared memory, at some position (the same for the whole
//     warp: each position has its own straight code): those after a cherry column move up.  (Picked one by one where a cherry column lay among
//     them, such blocks were the last to end: 57 us for 11008 x 4096 3-bit with 40, 36 without.)  Maxima, clamps and
//     roundings run on packed pairs.  Four rows' bytes are turned into words for the stores.
//   * The 128 columns go in four turns of one loop, twice, instead of 64 registers a lane: unrolled, a fourth of the issue
//     slots waited for instructions.  What depends on the columns alone is done once per block.
// 4096 x 11008 4-bit: 46 us (58 with the kernel above), 16384 x 28672: 342 (542).
constexpr int PG_WARPS = 4, PG_ROWS = 32, PG_BLOCKS = 4;        // warps of a block, rows of a warp's turn, blocks of an SM
constexpr int PG_SPAN = 160;                          // original columns that fit the tile
constexpr int PG_STRIDE = PG_SPAN + 8;                // an odd number of 16-byte pieces: those of 8 rows hit 8 different bank groups

// The 32 values from position OFF on of the 16-byte pieces at `u`, as pairs.
template <int OFF> __device__ __forceinline__ void take32(const uint4* u, uint32_t (&raw)[16]) {
  constexpr int N = OFF ? 5 : 4;
  uint32_t w[4 * N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint4 v = u[i];
    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) raw[i] = (OFF & 1) ? __funnelshift_r(w[OFF / 2 + i], w[OFF / 2 + i + (OFF & 1)], 16) : w[OFF / 2 + i];
}
// rint(r - 0.5) + 2^(BITS-1) of both halves, in the low bytes.  The difference of an fp16 number and 0.5 is exact in fp32;
// adding 1.5 * 2^23 (+ the code offset) rounds it to the nearest integer, ties to even.
template <int BITS> __device__ __forceinline__ void codes_of(uint32_t h, uint32_t& c0, uint32_t& c1) {
  const float magic = 12582912.f + (float)(1 << (BITS - 1));
  float a, b;
  asm("{\n\t.reg .f16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.f16 %0, l, %3;\n\tadd.rn.f32.f16 %1, h, %3;\n\t}"
      : "=f"(a), "=f"(b) : "r"(h), "f"(-0.5f));
  c0 = __float_as_uint(__fadd_rn(a, magic));
  c1 = __float_as_uint(__fadd_rn(b, magic));
}

template <int BITS>
__global__ void __launch_bounds__(PG_WARPS * 32, PG_BLOCKS) pack_group_kernel(
    const __half* __restrict__ w, const uint16_t* __restrict__ idx, int K, int N, int C, int G,
    __half* __restrict__ scales, uint8_t* __restrict__ q, __half* __restrict__ cw) {
  __shared__ __align__(16) __half tiles[PG_WARPS][PG_ROWS * PG_STRIDE + 32];      // (+ 32: reads of 32 columns where fewer are left)
  __shared__ int source[PK_COLS], s_at[4], s_gaps[4], s_gap[4], s_end;
  __shared__ __align__(16) uint32_t turned[PG_WARPS][4][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Kc = K - C, k0 = blockIdx.x * PK_COLS, cols = min(PK_COLS, Kc - k0);
  const bool two = G == 64;                                       // two groups in the block's 128 columns

  // ---- where the columns are
  static_assert(PG_WARPS * 32 == PK_COLS, "a thread a column");
  source[tid] = tid < cols ? k0 + tid + cherry_shift(idx, C, k0 + tid) : -1;
  if (tid == 0) s_end = k0 + PK_COLS >= Kc ? C : cherry_shift(idx, C, k0 + PK_COLS);
  __syncthreads();
  // the cherry columns before the next block's first column are this block's to copy
  const int c_begin = blockIdx.x == 0 ? 0 : source[0] - k0, c_end = s_end;
  const int first = c_begin < c_end ? min(idx[c_begin], source[0]) : source[0];
  const int last = c_begin < c_end ? max(idx[c_end - 1], source[cols - 1]) : source[cols - 1];
  const int base = first & ~7, pieces = (last - base) / 8 + 1;
  const bool wide = pieces * 8 <= PG_SPAN;                        // (K is a multiple of 8, w aligned to 16 bytes)
  // of each 32 columns: where the first is in the tile, how many cherry columns lie among them, the first of these
  const int parts = (cols + 31) / 32;
  if (tid < parts) {
    const int j = 32 * tid, from = source[j], to = source[min(j + 31, cols - 1)];
    s_at[tid] = wide ? from - base : j;
    s_gaps[tid] = wide ? to - from - min(31, cols - 1 - j) : 0;
    s_gap[tid] = from - (k0 + j);
  }
  __syncthreads();
  // this lane's first piece, and how far its next one is: rows, pieces
  const int piece_r = lane / pieces, piece_c = lane - piece_r * pieces, step_r = 32 / pieces, step_c = 32 - step_r * pieces;
  __half* tile = tiles[warp];
  const uint32_t tile_s = (uint32_t)__cvta_generic_to_shared(tile);
  auto copy = [&](int n0) {
    const int rows = min(PG_ROWS, N - n0);
    if (wide) {
      const __half* src = w + (size_t)(n0 + piece_r) * K + base + 8 * piece_c;
      uint32_t dst = tile_s + (piece_r * PG_STRIDE + 8 * piece_c) * 2;
      int c = piece_c;
      for (int r = piece_r; r < rows;) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        const bool wrap = c + step_c >= pieces;
        const int dr = step_r + wrap, dc = step_c - (wrap ? pieces : 0);
        r += dr;
        c += dc;
        src += dr * K + 8 * dc;
        dst += (dr * PG_STRIDE + 8 * dc) * 2;
      }
    } else {
      // so many cherry columns inside the chunk that it does not fit: compact columns one by one
      for (int j = lane; j < cols; j += 32) {
        const __half* src = w + (size_t)n0 * K + source[j];
#pragma unroll 16
        for (int r = 0; r < rows; ++r) tile[r * PG_STRIDE + j] = src[(size_t)r * K];
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  const int step = gridDim.y * PG_WARPS * PG_ROWS;
  int n0 = (blockIdx.y * PG_WARPS + warp) * PG_ROWS;
  if (n0 < N) copy(n0);
  for (; n0 < N; n0 += step) {
    const bool live = n0 + lane < N;
    const int n = live ? n0 + lane : N - 1;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    uint32_t raw[16];
    const __half* t = tile + lane * PG_STRIDE;
    // cherry_weight[c, n] = W[n, idx[c]]
    if (wide) {
      for (int c = c_begin; c < c_end; ++c) {
        const __half v = t[idx[c] - base];
        if (live) cw[(size_t)c * N + n] = v;
      }
    } else {
      // not in the tile, but the 32 columns after the 128 are free
      const int rows = min(PG_ROWS, N - n0);
      for (int c0 = c_begin; c0 < c_end; c0 += 32) {
        if (c0 + lane < c_end) {
          const __half* src = w + (size_t)n0 * K + idx[c0 + lane];
#pragma unroll 16
          for (int r = 0; r < rows; ++r) tile[r * PG_STRIDE + PK_COLS + lane] = src[(size_t)r * K];
        }
        __syncwarp();
        for (int c = c0; c < min(c_end, c0 + 32); ++c)
          if (live) cw[(size_t)c * N + n] = t[PK_COLS + c - c0];
        __syncwarp();
      }
    }
    auto take = [&](int p) {                                      // this lane's columns 32 p .. 32 p + 31
      const int at = s_at[p], gaps = s_gaps[p], left = cols - 32 * p;
      const uint4* u = reinterpret_cast<const uint4*>(t + (at & ~7));
      switch (at & 7) {                                           // the same for the whole warp
        case 0: take32<0>(u, raw); break;
        case 1: take32<1>(u, raw); break;
        case 2: take32<2>(u, raw); break;
        case 3: take32<3>(u, raw); break;
        case 4: take32<4>(u, raw); break;
        case 5: take32<5>(u, raw); break;
        case 6: take32<6>(u, raw); break;
        default: take32<7>(u, raw); break;
      }
#pragma unroll 1
      for (int g = 0; g < gaps; ++g) {                            // a cherry column goes, those after it move up
        const int pos = idx[s_gap[p] + g] - base - at - g;
        const uint32_t next = reinterpret_cast<const unsigned short*>(t)[min(at + 32 + g, PG_SPAN)];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t follow = i < 15 ? raw[i + 1 < 16 ? i + 1 : 15] : next;
          if (2 * i + 1 >= pos) raw[i] = __byte_perm(raw[i], follow, 2 * i + 1 == pos ? 0x5410 : 0x5432);
        }
      }
      if (left < 32) {
#pragma unroll
        for (int i = 0; i < 16; ++i) raw[i] = 2 * i + 1 < left ? raw[i] : (2 * i < left ? raw[i] & 0xffffu : 0u);
      }
    };
    // ---- scales of the two 64-column halves (of one group: the same)
    float s[2];
    __half2 m2[2] = {__float2half2_rn(0.f), __float2half2_rn(0.f)};       // (the maximum leaves NaN out, as fmaxf does)
#pragma unroll 1
    for (int p = 0; p < parts; ++p) {
      take(p);
      __half2 m = __float2half2_rn(0.f);
#pragma unroll
      for (int i = 0; i < 16; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __half2*>(&raw[i])));
      if (p < 2) m2[0] = __hmax2(m2[0], m);
      else m2[1] = __hmax2(m2[1], m);
    }
    if (!two) m2[0] = m2[1] = __hmax2(m2[0], m2[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && !two) { s[1] = s[0]; break; }
      const float mx = fmaxf(__low2float(m2[h]), __high2float(m2[h]));
      // fp16 add and fp16 divide (by a power of two: the product is the quotient), each rounded once
      const __half sh = __float2half_rn(__fmul_rn(__half2float(__float2half_rn(__fadd_rn(mx, 1e-6f))), 1.f / (1 << (BITS - 1))));
      const int grp = k0 / G + h;
      if (live && grp < (Kc + G - 1) / G) scales[(size_t)grp * N + n] = sh;
      s[h] = __half2float(sh);
    }
    // ---- quotients fp16(w / s) from the product with r = RN(1 / s): the product's relative error is below 2^-23; a quotient
    // of two 11-bit significands is farther than 2^-23 (1 + 2^-12) from a midpoint of two normal fp16 numbers, so the fp16
    // rounding is that of the quotient.  Quotients below 2^-14 may lie on a midpoint; of those only -2^-25, between -0 and
    // the first number that gets another code, matters, and w = -2^-25 s needs s >= 2.  Such scales (and infinite ones)
    // take the residual step of div_fp16.
    const bool large = __any_sync(0xffffffffu, !(s[0] < 2.f && s[1] < 2.f));
    const __half2 top = __float2half2_rn(BITS == 4 ? 7.98828125f : 3.98828125f), bottom = __hneg2(top);
#pragma unroll 1
    for (int p = 0; p < parts; ++p) {
      take(p);
      const float sp = p < 2 ? s[0] : s[1], rs = __frcp_rn(sp);
      if (large) {
        const float s_residual = sp < 65536.f ? sp : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&raw[i]));
          const __half2 h = __floats2half2_rn(div_fp16(f.x, s_residual, rs), div_fp16(f.y, s_residual, rs));
          raw[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&raw[i]));
          const __half2 h = __floats2half2_rn(__fmul_rn(f.x, rs), __fmul_rn(f.y, rs));
          raw[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
      }
      // ---- codes, clamped at an fp16 number just below 2^(BITS-1) - 0.01: the same code, whose middle is half a code away
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        uint32_t code[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __half2 h = __hmin2(__hmax2(*reinterpret_cast<const __half2*>(&raw[4 * o + i]), bottom), top);
          codes_of<BITS>(*reinterpret_cast<const uint32_t*>(&h), code[2 * i], code[2 * i + 1]);
        }
        // bytes 0, 2, 4, 6 and 1, 3, 5, 7
        const uint32_t even = __byte_perm(__byte_perm(code[0], code[2], 0x0040), __byte_perm(code[4], code[6], 0x0040), 0x5410);
        const uint32_t odd = __byte_perm(__byte_perm(code[1], code[3], 0x0040), __byte_perm(code[5], code[7], 0x0040), 0x5410);
        uint32_t word = even | (odd << BITS);
        if (BITS == 3) word = (word & 0x3Fu) | ((word >> 2) & 0xFC0u) | ((word >> 4) & 0x3F000u) | ((word >> 6) & 0xFC0000u);
        turned[warp][o][lane] = word;
      }
      __syncwarp();
      {
        // this lane: octet lane / 8 of the four, rows 4 (lane & 7) .. + 3 of the 32: four words to BITS rows of four bytes
        const int o = lane >> 3, m = n0 + 4 * (lane & 7);
        const uint4 v = *reinterpret_cast<const uint4*>(&turned[warp][o][4 * (lane & 7)]);
        if (m < N && 32 * p + 8 * o < cols) {                     // (N is a multiple of 8)
          const uint32_t p0 = __byte_perm(v.x, v.y, 0x5140), p1 = __byte_perm(v.x, v.y, 0x7362);
          const uint32_t p2 = __byte_perm(v.z, v.w, 0x5140), p3 = __byte_perm(v.z, v.w, 0x7362);
          const uint32_t b[4] = {__byte_perm(p0, p2, 0x5410), __byte_perm(p0, p2, 0x7632), __byte_perm(p1, p3, 0x5410), __byte_perm(p1, p3, 0x7632)};
          uint8_t* dst = q + (size_t)((k0 >> 3) + 4 * p + o) * BITS * N + m;
          if ((reinterpret_cast<uintptr_t>(q) & 3) == 0) {
#pragma unroll
            for (int i = 0; i < BITS; ++i) *reinterpret_cast<uint32_t*>(dst + (size_t)i * N) = b[i];
          } else {
            for (int i = 0; i < BITS; ++i)
              for (int e = 0; e < 4; ++e) dst[(size_t)i * N + e] = (uint8_t)(b[i] >> (8 * e));
          }
        }
      }
      __syncwarp();
    }
    if (n0 + step < N) copy(n0 + step);                           // (every lane is done with the tile)
  }
}

// ------------------------------------------------------------------ dense unpack
// llama/qlinear.py:120-162: dense[n, k] = cherry ? cherry_weight : fp16((q + 0.5) * s).
// Two kernels, both with blocks of 64 rows x 128 columns.  A thread makes one octet of 8 original columns of four consecutive
// rows.  The octet's codes are consecutive compact columns: the bytes of two compact octets (one 32-bit load per byte row
// covers the four rows), shifted by the position inside the first; a cherry column inside leaves a gap in the word, and its
// values go over the finished octet.  The tile in shared memory (16-byte slots, slot number XOR row quad against bank
// conflicts) turns the octets into rows of 256 contiguous bytes.
constexpr int UP_ROWS = 64, UP_COLS = 128, UP_BLOCKS = 4;       // blocks of an SM

__device__ __forceinline__ uint32_t load_quad(const uint8_t* p, bool aligned) {
  if (aligned) return __ldg(reinterpret_cast<const uint32_t*>(p));
  return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}
// four consecutive scales
__device__ __forceinline__ uint2 load_scales(const __half* p, bool aligned) {
  if (aligned) return __ldg(reinterpret_cast<const uint2*>(p));
  const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
  return make_uint2((uint32_t)u[0] | ((uint32_t)u[1] << 16), (uint32_t)u[2] | ((uint32_t)u[3] << 16));
}

// the codes of a word, 2 i and 2 i + 1 in field bits P_i of the halves of t[i], into (u - off) * s with the pair's scales
template <int BITS, int P> __device__ __forceinline__ uint32_t scaled_pair(uint32_t t, uint32_t s2) {
  constexpr uint32_t FIELD = (uint32_t)(((1 << BITS) - 1) << P), ONE = (uint32_t)(15 - P) << 10;      // 2^-P
  // -(1024 * 2^-P + off)
  constexpr uint32_t CENTER = BITS == 4 ? 0xD478u : (P == 1 ? 0xE007u : 0xC9C0u);       // -71.5; -515.5, -11.5
  static_assert(BITS == 4 ? P == 4 : (P == 1 || P == 7), "no other fields are used");
  uint32_t d;
  asm("{\n\t.reg .b32 v;\n\tfma.rn.f16x2 v, %1, %2, %3;\n\tmul.rn.f16x2 %0, v, %4;\n\t}"
      : "=r"(d) : "r"((t & (FIELD | (FIELD << 16))) | 0x64006400u), "r"(ONE | (ONE << 16)), "r"(CENTER | (CENTER << 16)), "r"(s2));
  return d;
}
// eight codes (consecutive fields of `word`) times the scales of each pair
template <int BITS> __device__ __forceinline__ uint4 scaled_octet(uint32_t word, const uint32_t (&s2)[4]) {
  uint4 v;
  if constexpr (BITS == 4) {
    const uint32_t up = word << 4;            // byte i of `up` has code 2 i above, byte i of `word` code 2 i + 1
    v.x = scaled_pair<4, 4>(__byte_perm(up, word, 0x4400), s2[0]);
    v.y = scaled_pair<4, 4>(__byte_perm(up, word, 0x5511), s2[1]);
    v.z = scaled_pair<4, 4>(__byte_perm(up, word, 0x6622), s2[2]);
    v.w = scaled_pair<4, 4>(__byte_perm(up, word, 0x7733), s2[3]);
  } else {
    // low half: codes 0 .. 4 from bit 1 on, high half: codes 1 .. 5
    const uint32_t a = ((word << 1) & 0xFFFFu) | ((word << 14) & 0xFFFF0000u);
    const uint32_t b = ((word >> 11) & 0xFFFFu) | ((word << 2) & 0xFFFF0000u);      // the same from code 4 on
    v.x = scaled_pair<3, 1>(a, s2[0]);
    v.y = scaled_pair<3, 7>(a, s2[1]);
    v.z = scaled_pair<3, 1>(b, s2[2]);
    v.w = scaled_pair<3, 7>(b, s2[3]);
  }
  return v;
}

// A block makes one tile, with gaps and group boundaries in every octet: for layers with many cherry columns, narrow groups, and
// matrices that are small or narrow (the rule and both sides' times stand at cq_unpack_dense).  Pairs of codes become the low
// mantissa bits of 1024 + u, minus (1024 + off), times the scale: each step but the last exact, so the product is rounded once
// as in the reference.
// codes 2 i, 2 i + 1 of a word as fp16 (u - off)
template <int BITS> __device__ __forceinline__ __half2 code_pair(uint32_t word, int i) {
  const uint32_t x = word >> (2 * BITS * i);
  constexpr uint32_t M = (1u << BITS) - 1;
  const uint32_t v = (x & M) | ((x << (16 - BITS)) & (M << 16)) | 0x64006400u;
  constexpr uint32_t CENTER = BITS == 4 ? 0x64076407u : 0x64036403u;       // 1024 + floor(off)
  const uint32_t half = 0x38003800u;
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&CENTER));
  return __hsub2(d, *reinterpret_cast<const __half2*>(&half));
}

template <int BITS, bool CHERRY>
__global__ void __launch_bounds__(256, 5) unpack_dense_kernel(
    const uint8_t* __restrict__ q, const __half* __restrict__ scales, const __half* __restrict__ cw,
    const uint16_t* __restrict__ idx, int K, int N, int C, int G, int g_shift, __half* __restrict__ dense, int aligned) {
  __shared__ __align__(16) uint4 tile[UP_ROWS * (UP_COLS / 8)];
  __shared__ int before[UP_COLS / 8 + 1];           // cherry columns before each octet
  const int tid = threadIdx.x, nq = tid & 15, oct = tid >> 4;
  const int k0 = blockIdx.x * UP_COLS, n0 = blockIdx.y * UP_ROWS;
  const int k = k0 + 8 * oct, n = n0 + 4 * nq;
  const int Kc = K - C, n_oct = Kc / 8;
  if (CHERRY && tid <= UP_COLS / 8) {
    const int kk = k0 + 8 * tid;
    int low = 0, high = C;
    while (low < high) {
      const int mid = (low + high) >> 1;
      if ((int)idx[mid] < kk) low = mid + 1; else high = mid;
    }
    before[tid] = low;
  }
  __syncthreads();
  if (k < K && n < N) {
    const int low = CHERRY ? before[oct] : 0;
    const int cnt = CHERRY ? max(0, min(8, before[oct + 1] - low)) : 0, n_codes = 8 - cnt;      // cherry columns and codes
    const int kc = max(k - low, 0), o = kc >> 3, r = kc & 7;
    // the bytes of compact octets o and o + 1, four rows in each word
    uint32_t b[2][BITS];
    const uint8_t* src = q + (size_t)o * BITS * N + n;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < BITS; ++i)
        b[h][i] = (o + h < n_oct && (h == 0 || r)) ? load_quad(src + (size_t)(h * BITS + i) * N, aligned & 1) : 0u;
    auto group_of = [&](int c) { return g_shift >= 0 ? c >> g_shift : c / G; };
    const int g = group_of(kc), split = (g + 1) * G - kc;       // codes 0 .. split - 1 belong to group g
    const bool whole = split >= n_codes;
    unsigned long long s0 = 0, s1 = 0;                          // the four rows' scales of groups g and g + 1
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n_codes > 0) s0 |= (unsigned long long)__half_as_ushort(scales[(size_t)g * N + n + j]) << (16 * j);
      if (!whole) s1 |= (unsigned long long)__half_as_ushort(scales[(size_t)(g + 1) * N + n + j]) << (16 * j);
    }
    uint32_t own = 0, second = 0;                               // columns that are cherries; that belong to group g + 1
    for (int t = 0; t < cnt; ++t) own |= 1u << (((int)idx[low + t] - k) & 7);
    if (!whole) {
#pragma unroll
      for (int e = 0; e < 8; ++e) second |= (e - __popc(own & ((1u << e) - 1)) >= split ? 1u : 0u) << e;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t w[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t sel = (uint32_t)j | ((uint32_t)(4 + j) << 4);
        const uint32_t lo = __byte_perm(b[h][0], b[h][1], sel);
        const uint32_t hi = BITS == 4 ? __byte_perm(b[h][2], b[h][BITS - 1], sel) : ((b[h][2] >> (8 * j)) & 0xFFu);
        w[h] = __byte_perm(lo, hi, 0x5410);
      }
      // the eight codes from column kc on
      uint32_t word;
      if (BITS == 4)
        word = __funnelshift_r(w[0], w[1], 4 * r);
      else
        word = ((w[0] & 0xFFFFFFu) >> (3 * r)) | (r ? w[1] << (24 - 3 * r) : 0u);
      for (uint32_t m = own; m; m &= m - 1) {                   // a gap at each cherry column
        const int at = BITS * (__ffs(m) - 1);
        const uint32_t below = (1u << at) - 1;
        word = (word & below) | ((word & ~below) << BITS);
      }
      const uint32_t sa = (uint32_t)(s0 >> (16 * j)) & 0xFFFFu, sb = (uint32_t)(s1 >> (16 * j)) & 0xFFFFu;
      uint32_t p[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t sc = whole ? (sa | (sa << 16))
                                  : (((second >> (2 * i)) & 1u ? sb : sa) | (((second >> (2 * i + 1)) & 1u ? sb : sa) << 16));
        const __half2 v = __hmul2(code_pair<BITS>(word, i), *reinterpret_cast<const __half2*>(&sc));
        p[i] = *reinterpret_cast<const uint32_t*>(&v);
      }
      tile[(4 * nq + j) * 16 + (oct ^ nq)] = make_uint4(p[0], p[1], p[2], p[3]);
    }
    for (int t = 0; t < cnt; ++t) {
      const int e = ((int)idx[low + t] - k) & 7;
#pragma unroll
      for (int j = 0; j < 4; ++j) reinterpret_cast<__half*>(&tile[(4 * nq + j) * 16 + (oct ^ nq)])[e] = cw[(size_t)(low + t) * N + n + j];
    }
    if (!whole && G < 8) {
      // groups narrower than 8 columns can put more than two into an octet: column by column
#pragma unroll 1
      for (int e = 0, m = low; e < 8; ++e) {
        if ((own >> e) & 1u) { ++m; continue; }
        const int c = k + e - m;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float a = (float)((int)cq_ref_code(q, BITS, c, n + j, N) - (1 << (BITS - 1))) + 0.5f;
          reinterpret_cast<__half*>(&tile[(4 * nq + j) * 16 + (oct ^ nq)])[e] =
              __float2half_rn(__fmul_rn(a, __half2float(scales[(size_t)group_of(c) * N + n + j])));
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int id = tid + 256 * i, rr = id >> 4, oo = id & 15;
    const int nn = n0 + rr, kk = k0 + 8 * oo;
    if (nn < N && kk < K) {
      const uint4 v = tile[rr * 16 + (oo ^ (rr >> 2))];
      __half* dst = dense + (size_t)nn * K + kk;
      if (aligned & 2) {
        *reinterpret_cast<uint4*>(dst) = v;
      } else {
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[e] = __ushort_as_half((unsigned short)(u[e >> 1] >> (16 * (e & 1))));
      }
    }
  }
}

// A block keeps its 128 columns and goes down the rows: what depends on the columns alone (the search for the cherry columns
// among it) is done once, the next rows' codes are on their way while these are written.  Pairs of codes become mantissa bits
// of 1024; one exact multiply-add and the product with the scale, rounded once, make the values.  Warps whose octets have
// neither a cherry column nor a group's end inside take a short path, the others a general one with a scale for each column.
// Bound by its instructions (15 a weight, 65 % of the issue slots busy): 11008 x 4096 3-bit 35.6 us (108 MB), 38.9 with the
// kernel above; 4096 x 11008 4-bit 36.9 and 40.6; 16384 x 28672 335 and 360.
// CHERRY = the layer has cherry columns
template <int BITS, bool CHERRY>
__global__ void __launch_bounds__(256, UP_BLOCKS) unpack_rows_kernel(
    const uint8_t* __restrict__ q, const __half* __restrict__ scales, const __half* __restrict__ cw,
    const uint16_t* __restrict__ idx, int K, int N, int C, int G, int g_shift, __half* __restrict__ dense, int aligned) {
  __shared__ __align__(16) uint4 tiles[2][UP_ROWS * (UP_COLS / 8)];
  const int tid = threadIdx.x, nq = tid & 15, oct = tid >> 4, lane = tid & 31;
  const int k0 = blockIdx.x * UP_COLS, k = k0 + 8 * oct, k_warp = k0 + 8 * (oct & ~1);       // a warp has two octets
  const int Kc = K - C, n_oct = Kc / 8;
  int low = 0, cnt = 0;                                         // cherry columns before the octet and inside it
  if (CHERRY) {
    int before[3] = {0, 0, 0};                                  // ... before the warp's first, second and the next octet
    for (int c = lane; c - lane < C; c += 32) {
      const int col = c < C ? (int)idx[c] : 0x7fffffff;
#pragma unroll
      for (int i = 0; i < 3; ++i) before[i] += __popc(__ballot_sync(0xffffffffu, col < k_warp + 8 * i));
    }
    low = before[oct & 1];
    cnt = max(0, min(8, before[(oct & 1) + 1] - low));
  }
  const int n_codes = 8 - cnt;
  const int kc = max(k - low, 0), o = kc >> 3, r = kc & 7;
  auto group_of = [&](int c) { return g_shift >= 0 ? c >> g_shift : c / G; };
  const int g = group_of(kc), split = (g + 1) * G - kc;         // codes 0 .. split - 1 belong to group g
  const bool whole = split >= n_codes;
  const bool plain = __all_sync(0xffffffffu, whole && cnt == 0);        // the whole warp's octets: eight codes of one group
  uint32_t own = 0, second = 0;                                 // columns that are cherries; that belong to group g + 1
  if (!plain && k < K) {
    for (int t = 0; t < cnt; ++t) own |= 1u << (((int)idx[low + t] - k) & 7);
    if (!whole) {
#pragma unroll
      for (int e = 0; e < 8; ++e) second |= (e - __popc(own & ((1u << e) - 1)) >= split ? 1u : 0u) << e;
    }
  }
  const bool in = k < K, more = r && o + 1 < n_oct, first = o < n_oct;
  // the bytes of compact octets o and o + 1, four rows in each word
  uint32_t b[2][BITS];
  uint2 ahead = make_uint2(0, 0);                               // the four rows' scales of group g
  const uint8_t* src = q + (size_t)o * BITS * N;
  const __half* own_scales = scales + (size_t)g * N;
  auto load = [&](int n) {
    const uint8_t* p = src + n;
    if (in && n < N && n_codes > 0) ahead = load_scales(own_scales + n, aligned & 4);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < BITS; ++i) {
        b[h][i] = (in && n < N && (h ? more : first)) ? load_quad(p, aligned & 1) : 0u;
        p += N;
      }
  };
  load(blockIdx.y * UP_ROWS + 4 * nq);
  uint4* tile = tiles[0];
  uint4* slot = tile + 64 * nq + (oct ^ nq);                    // rows 4 nq + j: 16 j slots on
  int other = UP_ROWS * (UP_COLS / 8);
  for (int n0 = blockIdx.y * UP_ROWS; n0 < N; n0 += gridDim.y * UP_ROWS) {
    const int n = n0 + 4 * nq;
    if (in && n < N) {
      const uint2 sc = ahead;
      // the four rows' words of both octets (a 4 x 4 transpose of bytes), then the eight codes from column kc on
      uint32_t words[4];
      {
        uint32_t w[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t b3 = BITS == 4 ? b[h][BITS - 1] : 0u;
          const uint32_t p0 = __byte_perm(b[h][0], b[h][1], 0x5140), p1 = __byte_perm(b[h][0], b[h][1], 0x7362);
          const uint32_t p2 = __byte_perm(b[h][2], b3, 0x5140), p3 = __byte_perm(b[h][2], b3, 0x7362);
          w[h][0] = __byte_perm(p0, p2, 0x5410);
          w[h][1] = __byte_perm(p0, p2, 0x7632);
          w[h][2] = __byte_perm(p1, p3, 0x5410);
          w[h][3] = __byte_perm(p1, p3, 0x7632);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (BITS == 4)
            words[j] = __funnelshift_r(w[0][j], w[1][j], 4 * r);
          else
            words[j] = (w[0][j] >> (3 * r)) | (r ? w[1][j] << (24 - 3 * r) : 0u);
        }
      }
      load(n + (int)gridDim.y * UP_ROWS);
      if (plain) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t s = __byte_perm(j < 2 ? sc.x : sc.y, 0, (j & 1) ? 0x3232 : 0x1010);
          const uint32_t s2[4] = {s, s, s, s};
          slot[16 * j] = scaled_octet<BITS>(words[j], s2);
        }
      } else {
        const uint2 sd = whole ? sc : load_scales(scales + (size_t)(g + 1) * N + n, aligned & 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t word = words[j];
          for (uint32_t m = own; m; m &= m - 1) {               // a gap at each cherry column
            const int at = BITS * (__ffs(m) - 1);
            const uint32_t below = (1u << at) - 1;
            word = (word & below) | ((word & ~below) << BITS);
          }
          const uint32_t sa = __byte_perm(j < 2 ? sc.x : sc.y, 0, (j & 1) ? 0x4432 : 0x4410);
          const uint32_t sb = __byte_perm(j < 2 ? sd.x : sd.y, 0, (j & 1) ? 0x4432 : 0x4410);
          uint32_t s2[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            s2[i] = ((second >> (2 * i)) & 1u ? sb : sa) | (((second >> (2 * i + 1)) & 1u ? sb : sa) << 16);
          slot[16 * j] = scaled_octet<BITS>(word, s2);
        }
        for (int t = 0; t < cnt; ++t) {
          const int e = ((int)idx[low + t] - k) & 7;
#pragma unroll
          for (int j = 0; j < 4; ++j) reinterpret_cast<__half*>(slot + 16 * j)[e] = cw[(size_t)(low + t) * N + n + j];
        }
      }
    }
    __syncthreads();                                            // (the other tile was read before this barrier)
    const int rr = tid >> 4, oo = tid & 15, kk = k0 + 8 * oo;
    if (kk < K) {
      __half* dst = dense + (size_t)(n0 + rr) * K + kk;
#pragma unroll
      for (int i = 0; i < 4; ++i) {                             // rows rr + 16 i
        if (n0 + rr + 16 * i < N) {
          const uint4 v = tile[(rr + 16 * i) * 16 + (oo ^ ((rr >> 2) + 4 * i))];
          if (aligned & 2) {
            *reinterpret_cast<uint4*>(dst) = v;
          } else {
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) dst[e] = __ushort_as_half((unsigned short)(u[e >> 1] >> (16 * (e & 1))));
          }
        }
        dst += 16 * (size_t)K;
      }
    }
    tile += other;
    slot += other;
    other = -other;
  }
}

// ------------------------------------------------------------------ Dequantize{3,4}Normal
__global__ void dequant_normal_kernel(const uint8_t* __restrict__ q, const float* __restrict__ sf,
                                      float* __restrict__ out, int bits, int Kc, int N, int G) {
  const long long total = (long long)Kc * N;
  const float off = (float)(1 << (bits - 1)) - 0.5f;
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total;
       id += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(id % N), kc = (int)(id / N);
    const float u = (float)cq_ref_code(q, bits, kc, n, N);
    out[id] = __fmul_rn(__fsub_rn(u, off), sf[(size_t)(kc / G) * N + n]);
  }
}

int nblocks(long long total, int threads) {
  long long b = (total + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 32) b = 148 * 32;
  return (int)b;
}

// Blocks over the rows for kernels whose blocks keep their columns and go down the rows, `per_sm` of them on an SM at once:
// about four waves, so that a last one that is nearly empty costs little (one wave and a bit took twice the time).
int row_blocks(int n_x, int n_tiles, int per_sm) {
  long long n = 4ll * per_sm * cq_sm_count() / n_x;
  if (n > n_tiles) n = n_tiles;
  return n < 1 ? 1 : (n > 65535 ? 65535 : (int)n);
}

int check_dims(int bits, int K, int N, int C, int* G) {
  if (bits != 3 && bits != 4) return CQ_ERR_BAD_BITS;
  if (*G == -1) *G = K;
  if (K <= 0 || N <= 0 || C < 0 || K % 8 || N % 8 || C % 8 || C >= K || K > 65534) return CQ_ERR_BAD_SHAPE;
  if (*G <= 0) return CQ_ERR_BAD_GROUP;
  return CQ_OK;
}

}  // namespace

extern "C" size_t cq_pack_tmp_bytes(int K) { (void)K; return 256; }

extern "C" int cq_pack(const void* weight, int weight_is_f32, const int32_t* cherry_unsorted, int bits,
                       int K, int N, int C, int G, uint8_t* qweight, void* scales, void* cherry_weight,
                       int16_t* cherry_indices, void* tmp, cq_stream_t stream) {
  (void)tmp;
  if (!weight || !qweight || !scales) return CQ_ERR_BAD_ARG;
  if (C > 0 && (!cherry_unsorted || !cherry_weight || !cherry_indices)) return CQ_ERR_BAD_ARG;
  const int rc = check_dims(bits, K, N, C, &G);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int T = 256;
  if (C > 0) pack_sort_kernel<<<nblocks(C, T), T, 0, st>>>(cherry_unsorted, C, cherry_indices);
  const uint16_t* idx = (const uint16_t*)cherry_indices;
  const int ng = (K - C + G - 1) / G;
  // From 12 million weights on a warp of pack_group_kernel has rows enough to go down (4096 x 11008 4-bit: 48.0 and 58.8 us;
  // 16384 x 28672 342 and 542; 4096 x 4096 22.9 and 24.9; 16384 x 1024 25.6 and 27.5; 4096 x 2048 16.5 and 16.5; 2048 x 1024
  // 12.3 and 10.3; 1032 x 1000 12.3 and 9.6).
  // Its weights come in 16 bytes at a time (off that alignment 4096 x 11008 would take 61 us, 55 with the other kernel), and each
  // cherry column among them moves the others: with more than a cherry column in 128 the other kernel is faster on matrices
  // below 25 million weights (2048 x 6144, one in 256 18.9 and 19.1, in 64 20.5 and 19.9, in 16 28 and 25, in 8 37 and 31) and on
  // narrow ones (1024 x 24576, one in 32 34 and 36, in 8 54 and 46; 4096 x 8192, in 8 78 and 86), but its last blocks copy the
  // cherry columns one after another (8192 x 1536, in 64 22 and 24, in 8 60 and 86; 1024 x 12288, in 4 26 and 38).
  const long long weights_all = (long long)K * N;
  const bool fits = (long long)C * 128 <= K || K >= 8192 || (long long)C * 5 >= K ||
                    (weights_all >= (3ll << 23) && ((long long)C * 32 <= K || K >= 4096));
  if (!weight_is_f32 && (G == 64 || G == PK_COLS) && weights_all >= (3ll << 22) && fits && ((uintptr_t)weight & 15) == 0) {
    const int n_x = (K - C + PK_COLS - 1) / PK_COLS, rows = PG_WARPS * PG_ROWS;
    auto kernel = bits == 4 ? pack_group_kernel<4> : pack_group_kernel<3>;
    kernel<<<dim3(n_x, row_blocks(n_x, (N + rows - 1) / rows, PG_BLOCKS)), PG_WARPS * 32, 0, st>>>(
        (const __half*)weight, idx, K, N, C, G, (__half*)scales, qweight, (__half*)cherry_weight);
    CQ_CUDA_TRY(cudaGetLastError());
    return CQ_OK;
  }
  const int span = G == 64 ? PK_COLS : (ng == 1 ? (K - C) : G);           // compact columns a block owns
  // A block walks a group of several chunks from end to end, twice, while the general pair spreads it over the chip: on
  // matrices of few rows the pair is faster.  Microseconds as measured over 256 .. 11008 columns, 64 .. 16384 rows (one
  // group per row, 4096 columns with cherries: 64 rows 65 and 98, 1024 rows 86 and 99, 2048 rows 111 and 100, 8192 rows
  // 301 and 112; without cherries 1024 rows 27 and 83, 8192 rows 155 and 85).
  const int chunks = (span + PK_COLS - 1) / PK_COLS;
  const double weights = (double)K * N;
  const double pair_us = C > 0 ? 8.0 + 0.0138 * span + 6.0e-6 * weights : 4.8 + 0.0013 * span + 4.4e-6 * weights;
  const double one_us = C > 0 ? (weight_is_f32 ? 4.0 + 3.7 * chunks : 3.0 + 3.0 * chunks) : 1.5 + (weight_is_f32 ? 3.3 : 2.6) * chunks;
  if ((G == 64 || G % PK_COLS == 0 || ng == 1) && (chunks == 1 || one_us <= pair_us)) {
    const int n_tiles = (N + PK_ROWS - 1) / PK_ROWS, n_spans = (K - C + span - 1) / span;
    const long long blocks = (long long)n_tiles * (n_spans + (C > 0));
    if (blocks <= 0x7fffffffll) {
      auto launch = [&](auto kernel, auto* wp) {
        kernel<<<(unsigned)blocks, PK_THREADS, 0, st>>>(wp, idx, K, N, C, G, span, n_tiles, n_spans,
                                                       (__half*)scales, qweight, (__half*)cherry_weight);
      };
      if (weight_is_f32)
        bits == 4 ? launch(pack_fused_kernel<float, 4>, (const float*)weight) : launch(pack_fused_kernel<float, 3>, (const float*)weight);
      else
        bits == 4 ? launch(pack_fused_kernel<__half, 4>, (const __half*)weight) : launch(pack_fused_kernel<__half, 3>, (const __half*)weight);
      CQ_CUDA_TRY(cudaGetLastError());
      return CQ_OK;
    }
  }
  if (C > 0)
    pack_cherry_kernel<<<nblocks((long long)C * N, T), T, 0, st>>>(weight, weight_is_f32, idx, K, N, C,
                                                                  (__half*)cherry_weight);
  pack_scales_kernel<<<nblocks((long long)ng * N * 32, T), T, 0, st>>>(weight, weight_is_f32, idx, bits,
                                                                      K, N, C, G, (__half*)scales);
  pack_codes_kernel<<<nblocks((long long)((K - C) / 8) * N, T), T, 0, st>>>(
      weight, weight_is_f32, idx, (const __half*)scales, bits, K, N, C, G, qweight);
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}

extern "C" int cq_unpack_dense(const uint8_t* qweight, const void* scales, const void* cherry_weight,
                               const int16_t* cherry_indices, int bits, int K, int N, int C, int G,
                               void* dense, cq_stream_t stream) {
  if (!qweight || !scales || !dense) return CQ_ERR_BAD_ARG;
  if (C > 0 && (!cherry_weight || !cherry_indices)) return CQ_ERR_BAD_ARG;
  const int rc = check_dims(bits, K, N, C, &G);
  if (rc) return rc;
  const int aligned = (((uintptr_t)qweight & 3) == 0 ? 1 : 0) | (((uintptr_t)dense & 15) == 0 ? 2 : 0) | (((uintptr_t)scales & 7) == 0 ? 4 : 0);
  int g_shift = -1;
  if ((G & (G - 1)) == 0)
    for (g_shift = 0; (1 << g_shift) < G;) ++g_shift;
  const int n_cols = (K + UP_COLS - 1) / UP_COLS, n_tiles = (N + UP_ROWS - 1) / UP_ROWS;
  auto launch = [&](auto kernel, int n_y) {
    kernel<<<dim3(n_cols, n_y), 256, 0, (cudaStream_t)stream>>>(qweight, (const __half*)scales, (const __half*)cherry_weight,
                                                               (const uint16_t*)cherry_indices, K, N, C, G, g_shift, (__half*)dense, aligned);
  };
  // From 25 million weights on, so that a block has rows to go down, up to a cherry column in 48, so that most octets have none,
  // and groups that put at most two into an octet.  New and old kernel: 4096 x 11008 4-bit, 16 cherry columns 36.9 us and 40.6, 64
  // 40.2 and 43.9, 128 44.6 and 46.2, groups of 4 66 and 62; 16384 x 1024, 64 cherry columns 18.4 and 18.6, 512 25.3 and 20.0; 2048
  // x 8192, groups of 96 17.3 and 17.0.  Matrices of few columns have no columns to spread over the chip but rows: 128 x 65536
  // 13.4 and 12.2.
  if ((long long)C * 48 <= K && G >= 8 && n_cols >= 8 && (long long)K * N >= (3ll << 23)) {
    const int n_y = row_blocks(n_cols, n_tiles, UP_BLOCKS);
    bits == 4 ? (C > 0 ? launch(unpack_rows_kernel<4, true>, n_y) : launch(unpack_rows_kernel<4, false>, n_y))
              : (C > 0 ? launch(unpack_rows_kernel<3, true>, n_y) : launch(unpack_rows_kernel<3, false>, n_y));
  } else {
    bits == 4 ? (C > 0 ? launch(unpack_dense_kernel<4, true>, n_tiles) : launch(unpack_dense_kernel<4, false>, n_tiles))
              : (C > 0 ? launch(unpack_dense_kernel<3, true>, n_tiles) : launch(unpack_dense_kernel<3, false>, n_tiles));
  }
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}

static int dequant_normal(int bits, const uint8_t* qweight, const float* sf, float* out, int qrows, int width,
                          int height, int cherry_size, int group_size, cq_stream_t stream) {
  if (!qweight || !sf || !out) return CQ_ERR_BAD_ARG;
  if (group_size == -1) group_size = height;
  if (width <= 0 || height <= 0 || cherry_size < 0 || cherry_size >= height || group_size <= 0)
    return CQ_ERR_BAD_SHAPE;
  const int Kc = height - cherry_size;
  if (Kc % 8 || qrows != Kc / 8 * bits) return CQ_ERR_BAD_SHAPE;
  dequant_normal_kernel<<<nblocks((long long)Kc * width, 256), 256, 0, (cudaStream_t)stream>>>(
      qweight, sf, out, bits, Kc, width, group_size);
  CQ_CUDA_TRY(cudaGetLastError());
  return CQ_OK;
}

extern "C" int cq_dequantize3_normal(const uint8_t* qweight, const float* sf, float* out, int qrows, int width,
                                     int height, int cherry_size, int group_size, cq_stream_t stream) {
  return dequant_normal(3, qweight, sf, out, qrows, width, height, cherry_size, group_size, stream);
}
extern "C" int cq_dequantize4_normal(const uint8_t* qweight, const float* sf, float* out, int qrows, int width,
                                     int height, int cherry_size, int group_size, cq_stream_t stream) {
  return dequant_normal(4, qweight, sf, out, qrows, width, height, cherry_size, group_size, stream);
}
