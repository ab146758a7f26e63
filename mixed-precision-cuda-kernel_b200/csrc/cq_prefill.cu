// Prefill GEMM of a tile-layout CherryQ layer for many activation rows ("tokens"):
//   y[m, n] (+)= sum_k' fp16((u[k', n] - off) * s[group(k'), n]) * x[m, orig(k')]
//              + sum_c  cherry_weight[c, n] * x[m, idx[c]]
// i.e. the reference's dense mode: QuantLinear.unpack() to fp16 followed by F.linear
// (llama/qlinear.py:120-162, 183-195 of the reference project), without ever writing the
// dequantised matrix to memory.  This is the only part of the path that is a dense
// contraction, so it runs on the 5th-generation tensor cores:
//
//   * A operand = weights, 256 rows per tile, 128 in each CTA of a pair, dequantised to fp16 by the
//     row's own thread (one thread = one weight row = one TENSOR MEMORY lane) and stored straight
//     into tensor memory with tcgen05.st: exponent-trick unpack (AND-OR into the bits of 1024.0), one
//     exact multiply-add and one multiplication by the group scale per fp16 pair, which reproduces
//     unpack()'s fp16 values bit for bit, whatever the scale;
//   * B operand = NT tokens of activations per tile (NT = 32 .. 256 in steps of 32), half of them in each CTA,
//     prepared once per call by a small pre-pass kernel (gather into compact column order, canonical
//     K-major UMMA layout) so that the main kernel moves them with plain bulk async copies;
//   * D = 256 rows x NT tokens fp32 in tensor memory (128 rows per CTA), accumulated over K by
//     tcgen05.mma.cta_group::2.kind::f16 (A from TMEM, M = 256, N = NT, K = 16 per instruction).
//
// Why pairs: a lone CTA with 128 x 256 tiles has to bring 64 KB of activations and 8 KB of weights into shared memory
// per 128 columns, about 70 bytes a cycle at the tensor core's rate, more than an SM gets from L2; in a pair each CTA
// brings half of the activations.
//
// Work: (token block, pair of row tiles) units x items (cherry items, then granules of 128 columns).  Clusters take
// whole units round-robin; the units that do not fill a last wave - all of them in a call of few tokens - are cut
// into equal runs of items, one run per cluster.  A unit that more than one cluster worked on is summed from fp32
// partial tiles, in item order, by the cluster that arrives last (no cluster waits for another; sums do not depend on
// timing).
//
// Warp roles (736 threads, one CTA per SM, persistent over its work list):
//   warps 0-15  four decode groups (items go round-robin), thread r of a group = row r
//   warp 16     MMA issuer (one lane, leader CTA); owns the tensor-memory allocation
//   warps 17-18 producers (one lane each): bulk copies of weight items / activation tiles; each issue costs its thread
//               a few hundred cycles, so they are two and keep their addresses and phases without a division
//   warps 19-22 epilogue: tcgen05.ld of a finished tile into shared memory (which frees the accumulator), then
//               16-byte stores to y
// Every wait is bounded and reports into the status word instead of hanging.  The kernel may be resident while kernels
// before the pre-pass still run (an exchange that waits for a late rank for seconds, say): the bounds only count once the
// activation producer has passed the dependency wait, which it notes in the CTA's state.  (A dependency wait in every
// role did the same and cost a call of 16 rows 0.3 us.)
//
// Bound and state: 4096 -> 11008 4-bit, 2048 rows: 140 us = 1.32 PFLOP/s (739 us through QuantLinear and 195 us by itself
// with lone CTAs of 128 x 256 tiles); 8192 -> 28672 3-bit, 2048 rows: 641 us = 1.50 PFLOP/s, tensor-bound.  16 rows: 18 and
// 49 us (31 and 76): an item then takes about 700 cycles, most of them the decode groups' instructions and waits, against
// 365 that its weights need to arrive from HBM.  (54 us while every decode warp walked over all items, polled without a
// hint and took every fourth; the hint without the stepping was slower, 61.  With six groups, or with lone CTAs that leave
// room for seven A slots, it was no faster.)
#include <algorithm>
#include <cmath>

#include "cq_tile.cuh"

namespace {

constexpr uint32_t WAIT_LIMIT = 1u << 22;
// How long one try of a wait may suspend its thread.  Every role but the decode groups mostly waits, and a call of few
// rows is bound by what the decode groups issue; without the hint its polls come back after some tens of cycles each.
constexpr uint32_t WAIT_HINT_NS = 20000;
constexpr int NGRP = 4;                 // decode groups of four warps
constexpr int NA = 4;                   // A slots in tensor memory (64 columns each), one per decode group
constexpr int A_COLS = 64;
constexpr int D_BASE = NA * A_COLS;
constexpr int TMEM_COLS = 512;
constexpr int SW_MAX = 12, SB_MAX = 12; // most weight / activation ring stages
constexpr int NTHREADS = (NGRP * 4 + 7) * 32;
constexpr int STAGE_THREADS = 128;     // a block of the pre-pass fits beside a CTA of the main kernel
constexpr int N_BARS = 2 * SW_MAX + 2 * SB_MAX + 2 * NA + 4;
// A CTA's half of the B operand of one K = 16 step: [token group of 8][k half][8 tokens][16 B] = NT / 2 * 32 bytes;
// a granule is 8 steps, a cherry item one.
__host__ __device__ constexpr int b_kstep_bytes(int nt) { return nt * 16; }
__host__ __device__ constexpr int b_gran_bytes(int nt) { return nt * 128; }

constexpr int MAX_LAYERS = 4;           // layers of one launch, which share an input

struct PrefillLayer {
  const uint8_t* stream;     // tile-layout weight stream
  const uint8_t* xb;         // staged activations: [token block][half][cherry items][granules]
  __half* y;
  const __half* bias;        // null: none
  float* partial;            // [cluster][first / last run][CTA of the pair][token][128 rows] fp32
  uint32_t* arrived;         // [cut unit][CTA of the pair] runs finished so far
  int N, n_tile, ldy;
  uint32_t n_units;          // token blocks x pairs of row tiles
  uint32_t sk_units, sk_clusters;   // the first sk_units units are cut into runs of items for sk_clusters clusters
};
struct PrefillParams {
  PrefillLayer layer[MAX_LAYERS];
  uint32_t* status;
  int n_layers, M, n_gran, n_cher, gran_bytes, tile_bytes, accumulate, vec_y;
  int nt;                    // tokens per block
  unsigned long long xb_half_bytes;
  int wstage_bytes, sw, sb, off_wring, off_bring, off_stage, off_bar;   // sw, sb = ring stages
};
// what the pre-pass needs of each layer
struct StageLayers {
  const uint32_t* osh[MAX_LAYERS];
  const uint16_t* cidx[MAX_LAYERS];
  uint8_t* xb[MAX_LAYERS];
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(WAIT_HINT_NS) : "memory");
  return ok != 0;
}
// State of a CTA: whether the kernels before this one have finished, and whether a wait ran out.
constexpr int RUNNING = 0, ABORTED = 1, PENDING = 2;
// Bounded wait: gives up after WAIT_LIMIT polls or about one second of the device's nanosecond timer (read once some polls
// have failed), at once when the CTA already gave up, records which wait failed in the status word and lets the caller run
// on to the common exit.  While the CTA is PENDING nothing counts: that time belongs to the kernels before.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* state,
                                            uint32_t* status, uint32_t code) {
  const uint32_t limit = *state == ABORTED ? 1u : WAIT_LIMIT;
  unsigned long long t0 = 0;
  for (uint32_t it = 0; it < limit;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*state == PENDING) continue;
    if ((++it & 15u) == 0u) {
      unsigned long long t1;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      if (t0 == 0) t0 = t1;
      else if (t1 - t0 > 1000000000ull) break;
    }
  }
  *state = ABORTED;
  if (status) atomicOr(status, code);
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* state, uint32_t* status,
                                          uint32_t code) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, state, status, code);
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// until the kernels before this one have finished and their writes are visible
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// What an arrival in the other CTA announces is read there by the tensor core only (tensor memory, ordered by the
// tcgen05 fences, and tiles written by the async proxy), so it needs no cluster-wide fence: release.cluster here and
// acquire.cluster in the waits made an item of 128 columns take 1500 cycles whatever its number of tokens.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrives on the barrier at this offset in both CTAs when every MMA issued so far has finished
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((unsigned short)3) : "memory");
}
// D[tmem_d] (+)= A[tmem_a] * B[desc_b] over the pair: fp16 inputs, fp32 accumulate, shape from the instruction descriptor
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float* v) {
  uint32_t r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr) : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major, unswizzled operand: rows of a core matrix 16 B
// apart, the two 8-column halves of a 16-column step `lbo` bytes apart, 8-row groups `sbo` apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo16, uint32_t sbo16) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)lbo16 << 16) | ((uint64_t)sbo16 << 32) | ((uint64_t)1 << 46);
}

// ------------------------------------------------------------------ dequantisation to fp16
// A code field at mantissa bit p OR-ed into the bits of fp16 1024.0 is the number 1024 + 2^p u.
// One multiply-add, times 2^-p less (1024 * 2^-p + off), makes it u - off: every constant and the result are
// exact.  The product with the scale s is then (u - off) * s rounded once to fp16: exactly the value unpack()
// computes as fp16(q + 0.5) * s (llama/qlinear.py:139-146 of the reference project).  (2^-p folded into the scale
// instead would round it where it becomes subnormal: s below 2^-8, weights of a deviation of about 0.01.)
constexpr uint32_t MAGIC = 0x64006400u;
__device__ __forceinline__ constexpr uint32_t dup16(uint32_t h) { return h | (h << 16); }
__device__ __forceinline__ constexpr uint32_t pow2_neg(int pbit) { return (uint32_t)(15 - pbit) << 10; }   // fp16 bits of 2^-p
// fp16 bits of -(1024 * 2^-p + off)
template <int BITS> __device__ __forceinline__ constexpr uint32_t center(int pbit) {
  return BITS == 4 ? (pbit == 2 ? 0xDC1Eu : 0xCDE0u)                       // -263.5, -23.5
                   : (pbit == 1 ? 0xE007u : (pbit == 4 ? 0xD438u : 0xC9C0u));   // -515.5, -67.5, -11.5
}
// the pair of codes at mantissa bit P of `word` -> (u - off) * s
template <int BITS, int P> __device__ __forceinline__ uint32_t code_pair(uint32_t word, uint32_t s) {
  return hmul2_u32(hfma2_u32(word | MAGIC, dup16(pow2_neg(P)), dup16(center<BITS>(P))), s);
}

// One 4-bit word (8 codes) -> 4 fp16 pairs; s = the scale, twice
__device__ __forceinline__ void dequant4(uint32_t w, uint32_t s, uint32_t* out) {
  const uint32_t v1 = w << 2, v2 = w >> 6;
  out[0] = code_pair<4, 2>(v1 & 0x003C003Cu, s);
  out[1] = code_pair<4, 6>(v1 & 0x03C003C0u, s);
  out[2] = code_pair<4, 2>(v2 & 0x003C003Cu, s);
  out[3] = code_pair<4, 6>(v2 & 0x03C003C0u, s);
}
// Three 3-bit words (32 codes) -> 16 fp16 pairs
__device__ __forceinline__ void dequant3(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t s, uint32_t* out) {
  const uint32_t w[3] = {w0, w1, w2};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t v = w[i] >> 6;
    out[5 * i + 0] = code_pair<3, 1>(w[i] & 0x000E000Eu, s);   // field at bit 1
    out[5 * i + 1] = code_pair<3, 4>(w[i] & 0x00700070u, s);   // bit 4
    out[5 * i + 2] = code_pair<3, 7>(w[i] & 0x03800380u, s);   // bit 7
    out[5 * i + 3] = code_pair<3, 4>(v & 0x00700070u, s);      // bit 10 -> 4
    out[5 * i + 4] = code_pair<3, 7>(v & 0x03800380u, s);      // bit 13 -> 7
  }
  uint32_t r = (w0 << 7) & 0x00800080u;     // pair 15: one bit from each word, at bits 7..9
  r |= (w1 << 8) & 0x01000100u;
  r |= (w2 << 9) & 0x02000200u;
  out[15] = code_pair<3, 7>(r, s);
}

// ------------------------------------------------------------------ activation pre-pass
// xb[token block][half of the block][item][...] in the layout the MMA reads from shared memory: per K = 16 step
// [token group of 8][k half][token in group][8 fp16]; cherry items (16 cherry columns) first, then the granules
// (128 compact columns = 8 steps).  A warp stages four octets of eight tokens (128 contiguous bytes per octet) and goes
// on to the next GROUPS - 1 token groups with the same columns, all their loads in flight together.  An octet without a
// cherry column inside is two aligned 16-byte loads and a shift by its position in them; the others are loaded column by
// column.  Bound by latency: where the columns are is found once, before the kernels before this one have finished (with a
// search for each token of an octet with a cherry column, after the wait, a call of 16 rows of 4096 x 11008 took 18.6 us
// instead of 17.1, 45 rows of 5120 x 5120 21.5 and 20.3).  Eight blocks an SM: with nine and ten, spilling registers at
// ten, 2048 rows of 5120 x 5120 took 2 to 3 us longer.
// Tokens past M are not written: the padding feeds accumulator columns that are never read back (each output
// column depends on its own token only).  Also clears the arrival counters of the main kernel.
// the eight halves that start `off` halves into the two vectors
__device__ __forceinline__ uint4 shift_halves(uint4 lo, uint4 hi, int off) {
  uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
  for (int i = 0; i < 6; ++i) w[i] = (off & 4) ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 5; ++i) w[i] = (off & 2) ? w[i + 1] : w[i];
  const uint32_t s = 16 * (off & 1);
  return make_uint4(__funnelshift_r(w[0], w[1], s), __funnelshift_r(w[1], w[2], s), __funnelshift_r(w[2], w[3], s),
                    __funnelshift_r(w[3], w[4], s));
}
template <int GROUPS>
__global__ void __launch_bounds__(STAGE_THREADS, 8) prefill_stage_x_kernel(
    const __half* __restrict__ x, int ldx, int M, const __grid_constant__ StageLayers layers, int C, int Kc, int n_gran, int n_cher,
    unsigned long long half_bytes, int NT, uint32_t* __restrict__ arrived, int n_arrived, int aligned16) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int n_oct = 2 * n_cher + 16 * n_gran;              // octets per token
  const int lane = threadIdx.x & 31, HT = NT >> 1;
  const int oi = (blockIdx.x * (STAGE_THREADS / 32) + (threadIdx.x >> 5)) * 4 + (lane >> 3);
  const unsigned short* xs = reinterpret_cast<const unsigned short*>(x);
  const uint32_t* __restrict__ osh = layers.osh[blockIdx.z];
  const uint16_t* __restrict__ cidx = layers.cidx[blockIdx.z];
  uint8_t* __restrict__ xb = layers.xb[blockIdx.z];
  // Where the octet's columns are (weights: no need to wait for the kernels before): a lane finds one of the eight.  (Shared
  // memory would keep the block from an SM that has a CTA of the main kernel.)
  constexpr uint32_t NONE = 0xFFFFu;
  uint32_t col = NONE;
  {
    const int oc = oi - 2 * n_cher, k = 8 * oc + (lane & 7);
    if (oc < 0) {
      if (k + 16 * n_cher < C) col = cidx[k + 16 * n_cher];
    } else if (k < Kc) {
      const uint32_t sh = osh[oc];
      if (sh != 0xFFFFFFFFu) {
        // cherry columns inside the octet: the shift grows from the first column's to the last one's
        int sft = (int)(sh & 0xFFFFu);
        while (sft < (int)(sh >> 16) && (int)cidx[sft] - sft <= k) ++sft;
        col = (uint32_t)(k + sft);
      }
    }
  }
  const int c0 = (int)__shfl_sync(0xffffffffu, col, lane & 24), c7 = (int)__shfl_sync(0xffffffffu, col, lane | 7), off = c0 & 7;
  const bool cherry = oi < 2 * n_cher;
  const int o = oi - 2 * n_cher;
  const size_t dst0 = cherry ? (size_t)(oi >> 1) * b_kstep_bytes(NT) + (oi & 1) * 128
                             : (size_t)n_cher * b_kstep_bytes(NT) + (size_t)(o >> 4) * b_gran_bytes(NT) +
                                   ((o & 15) >> 1) * b_kstep_bytes(NT) + (o & 1) * 128;
  const bool plain = !cherry && c7 != (int)NONE && c7 == c0 + 7 && aligned16;      // (the same for an octet's eight lanes)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
    for (int i = threadIdx.x; i < n_arrived; i += STAGE_THREADS) arrived[i] = 0u;
  if (oi >= n_oct) return;
  auto store = [&](int m, uint4 v) {
    const int mb = m / NT, ml = m - mb * NT, hf = ml >= HT, mt = ml - hf * HT;
    *reinterpret_cast<uint4*>(xb + (size_t)(2 * mb + hf) * half_bytes + dst0 + (mt >> 3) * 256 + (mt & 7) * 16) = v;
  };
  for (int tg0 = blockIdx.y * GROUPS; tg0 < (M + 7) >> 3; tg0 += gridDim.y * GROUPS) {
    const int m0 = tg0 * 8 + (lane & 7);
    if (plain) {
      uint4 v[GROUPS], v2[GROUPS];
#pragma unroll
      for (int u = 0; u < GROUPS; ++u) {
        const int m = m0 + 8 * u;
        v[u] = v2[u] = make_uint4(0, 0, 0, 0);
        if (m < M) {
          // (K is a multiple of 8 and all eight columns exist: the second vector, where needed, lies inside the row)
          const uint4* src = reinterpret_cast<const uint4*>(xs + (size_t)m * ldx + (c0 - off));
          v[u] = __ldg(src);
          if (off) v2[u] = __ldg(src + 1);
        }
      }
#pragma unroll
      for (int u = 0; u < GROUPS; ++u)
        if (m0 + 8 * u < M) store(m0 + 8 * u, shift_halves(v[u], v2[u], off));
    } else {
#pragma unroll 1
      for (int u = 0; u < GROUPS; u += 2) {
        uint32_t h[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int m = m0 + 8 * (u + i);
            const uint32_t ce = __shfl_sync(0xFFu << (lane & 24), col, (lane & 24) + e);
            h[i][e] = u + i < GROUPS && m < M && ce != NONE ? __ldg(xs + (size_t)m * ldx + ce) : 0u;
          }
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (u + i < GROUPS && m0 + 8 * (u + i) < M)
            store(m0 + 8 * (u + i), make_uint4(h[i][0] | (h[i][1] << 16), h[i][2] | (h[i][3] << 16), h[i][4] | (h[i][5] << 16),
                                               h[i][6] | (h[i][7] << 16)));
      }
    }
  }
}

// ------------------------------------------------------------------ work list of a cluster
struct Work {
  uint32_t layer, unit, j0, j1;     // items [j0, j1) of this unit of the layer
  int run;                   // -1: a whole unit; 0 / 1: the first / last run of this cluster, a part of its unit
};
// first item of cluster c's run over the cut units
__device__ __forceinline__ uint32_t run_begin(const PrefillLayer& L, uint32_t c, uint32_t total) {
  return c * total / L.sk_clusters;        // (74 clusters x 73 units x a few thousand items at most: fits 32 bits)
}
// Layer by layer, each divided as in a launch of its own: the sums are the same, and while the last of a layer is stored the
// next one's weights are on their way.  MANY: more than one layer (with the layer as a variable in launches of one, 45 rows of
// 5120 x 13824 took 1 us longer).
template <bool MANY> struct WorkList {
  const PrefillParams& p;
  uint32_t layer, b, e, b0, u, ipt, cluster, clusters;
  __device__ __forceinline__ WorkList(const PrefillParams& p_, uint32_t cluster_, uint32_t n_clusters, uint32_t ipt_)
      : p(p_), layer(0), ipt(ipt_), cluster(cluster_), clusters(n_clusters) {
    begin();
  }
  __device__ __forceinline__ void begin() {
    const PrefillLayer& L = p.layer[MANY ? layer : 0];
    u = L.sk_units + cluster;
    b = e = b0 = 0;
    if (cluster < L.sk_clusters) {
      const uint32_t total = L.sk_units * ipt;
      b0 = b = run_begin(L, cluster, total);
      e = run_begin(L, cluster + 1, total);
    }
  }
  __device__ __forceinline__ bool next(Work& w) {
    for (;;) {
      w.layer = MANY ? layer : 0;
      if (b < e) {
        w.unit = b / ipt;
        w.j0 = b - w.unit * ipt;
        w.j1 = min(ipt, w.j0 + (e - b));
        w.run = (w.j0 == 0 && w.j1 == ipt) ? -1 : (b == b0 ? 0 : 1);
        b += w.j1 - w.j0;
        return true;
      }
      if (u < p.layer[MANY ? layer : 0].n_units) {
        w.unit = u;
        w.j0 = 0;
        w.j1 = ipt;
        w.run = -1;
        u += clusters;
        return true;
      }
      if (!MANY || layer + 1 >= (uint32_t)p.n_layers) return false;
      ++layer;
      begin();
    }
  }
};

// position in a ring of stages: slot, parity of its current round, rounds completed
struct Ring {
  uint32_t slot = 0, phase = 0, round = 0;
  __device__ __forceinline__ void advance(uint32_t stages) {
    if (++slot == stages) {
      slot = 0;
      phase ^= 1;
      ++round;
    }
  }
  // `n` at once, at most the number of stages
  __device__ __forceinline__ void skip(uint32_t n, uint32_t stages) {
    if ((slot += n) >= stages) {
      slot -= stages;
      phase ^= 1;
      ++round;
    }
  }
  // the last use of every slot used so far
  template <typename F> __device__ __forceinline__ void each_last(uint32_t stages, F f) const {
    for (uint32_t s = 0; s < stages; ++s) {
      if (s < slot) f(s, phase);
      else if (round) f(s, phase ^ 1);
    }
  }
};

// ------------------------------------------------------------------ main kernel
template <int BITS, int SETS, bool MANY>
__global__ void __launch_bounds__(NTHREADS, 1) cq_prefill_kernel(const __grid_constant__ PrefillParams p) {
  constexpr int W_MMA = NGRP * 4, W_PROD_W = NGRP * 4 + 1, W_PROD_B = NGRP * 4 + 2;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_state;
  __shared__ uint32_t s_tmem;
  __shared__ int s_last;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const uint32_t cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const uint32_t NT = (uint32_t)p.nt;
  const uint32_t ND = NT <= 128 ? 2 : 1;                   // accumulator buffers of NT columns
  const uint32_t NCH = (uint32_t)p.n_cher, IPT = NCH + (uint32_t)p.n_gran;
  const uint32_t SW = (uint32_t)p.sw, SB = (uint32_t)p.sb;
  const uint32_t B_KSTEP_BYTES = b_kstep_bytes(NT), B_GRAN_BYTES = b_gran_bytes(NT), B_CHER_BYTES = B_KSTEP_BYTES;

  const uint32_t bar0 = smem_u32(smem + p.off_bar);
  auto B_WFULL = [&](uint32_t s) { return bar0 + 8 * s; };
  auto B_WEMPTY = [&](uint32_t s) { return bar0 + 8 * (SW_MAX + s); };
  auto B_BFULL = [&](uint32_t s) { return bar0 + 8 * (2 * SW_MAX + s); };
  // leader's: item ready in both CTAs (A in tensor memory, activations in shared memory)
  auto B_READY = [&](uint32_t a) { return bar0 + 8 * (2 * SW_MAX + 2 * SB_MAX + a); };
  auto B_AEMPTY = [&](uint32_t a) { return bar0 + 8 * (2 * SW_MAX + 2 * SB_MAX + NA + a); };
  // with as many activation stages as A slots one commit releases both
  auto B_BEMPTY = [&](uint32_t s) { return SB == NA ? B_AEMPTY(s) : bar0 + 8 * (2 * SW_MAX + SB_MAX + s); };
  auto B_DFULL = [&](uint32_t d) { return bar0 + 8 * (2 * SW_MAX + 2 * SB_MAX + 2 * NA + d); };
  auto B_DEMPTY = [&](uint32_t d) { return bar0 + 8 * (2 * SW_MAX + 2 * SB_MAX + 2 * NA + 2 + d); };

  if (tid == 0) {
    s_state = PENDING;
    for (uint32_t s = 0; s < SW; ++s) { mbar_init(B_WFULL(s), 1); mbar_init(B_WEMPTY(s), 4); }
    for (uint32_t s = 0; s < SB; ++s) {
      mbar_init(B_BFULL(s), 1);
      if (SB != NA) mbar_init(B_BEMPTY(s), 1);
    }
    for (uint32_t a = 0; a < NA; ++a) { mbar_init(B_READY(a), 8); mbar_init(B_AEMPTY(a), 1); }
    for (uint32_t d = 0; d < 2; ++d) { mbar_init(B_DFULL(d), 1); mbar_init(B_DEMPTY(d), 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                          // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == W_PROD_W) {
    // ================================================================ weight producer
    // (starts at once: the first ring of weights streams while the pre-pass still stages the activations)
    if (lane == 0) {
      const uint32_t wring = smem_u32(smem + p.off_wring);
      Ring ring;
      WorkList<MANY> wl(p, cluster, n_clusters, IPT);
      Work w;
      while (wl.next(w)) {
        // (an odd number of row tiles: the last pair's second CTA repeats the last tile, its results are dropped)
        const PrefillLayer& L = p.layer[MANY ? w.layer : 0];
        const uint32_t NTILE = (uint32_t)L.n_tile, NPAIR = (NTILE + 1) / 2;
        const uint32_t tile = min(2 * (w.unit % NPAIR) + rank, NTILE - 1);
        const uint32_t c0 = min(w.j0, NCH);
        const uint8_t* src = L.stream + (size_t)tile * p.tile_bytes + (size_t)c0 * CQT_CHER_BYTES + (size_t)(w.j0 - c0) * p.gran_bytes;
        for (uint32_t j = w.j0; j < w.j1; ++j) {
          const uint32_t bytes = j < NCH ? (uint32_t)CQT_CHER_BYTES : (uint32_t)p.gran_bytes;
          if (ring.round) mbar_wait(B_WEMPTY(ring.slot), ring.phase ^ 1, &s_state, p.status, 1u);
          if (*(volatile int*)&s_state == ABORTED) break;
          mbar_expect_tx(B_WFULL(ring.slot), bytes);
          bulk_g2s(wring + ring.slot * (uint32_t)p.wstage_bytes, src, bytes, B_WFULL(ring.slot));
          src += bytes;
          ring.advance(SW);
        }
      }
      // No copy is in flight when this thread leaves, also after a wait that ran out (bounded like every wait).
      int own = 0;
      ring.each_last(SW, [&](uint32_t slot, uint32_t phase) { mbar_wait(B_WFULL(slot), phase, &own, p.status, 512u); });
    }
  } else if (warp == W_PROD_B) {
    // ================================================================ activation producer
    if (lane == 0) {
      // the staged activations are written by the kernel launched just before this one
      dependency_wait();
      atomicCAS(&s_state, PENDING, RUNNING);
      const uint32_t bring = smem_u32(smem + p.off_bring);
      Ring ring;
      WorkList<MANY> wl(p, cluster, n_clusters, IPT);
      Work w;
      while (wl.next(w)) {
        const PrefillLayer& L = p.layer[MANY ? w.layer : 0];
        const uint32_t mb = w.unit / (((uint32_t)L.n_tile + 1) / 2);
        const bool real = (int)(mb * NT + rank * (NT >> 1)) < p.M;       // this half of the block holds tokens
        const uint32_t c0 = min(w.j0, NCH);
        const uint8_t* src = L.xb + (size_t)(2 * mb + rank) * p.xb_half_bytes + (size_t)c0 * B_CHER_BYTES +
                             (size_t)(w.j0 - c0) * B_GRAN_BYTES;
        for (uint32_t j = w.j0; j < w.j1; ++j) {
          const uint32_t bytes = j < NCH ? B_CHER_BYTES : B_GRAN_BYTES;
          if (ring.round) mbar_wait(B_BEMPTY(ring.slot), ring.phase ^ 1, &s_state, p.status, 2u);
          if (*(volatile int*)&s_state == ABORTED) break;
          if (real) {
            mbar_expect_tx(B_BFULL(ring.slot), bytes);
            bulk_g2s(bring + ring.slot * B_GRAN_BYTES, src, bytes, B_BFULL(ring.slot));
          } else {
            mbar_arrive(B_BFULL(ring.slot));
          }
          src += bytes;
          ring.advance(SB);
        }
      }
      // No copy and no arrival of a tcgen05.commit is in flight when this thread leaves: a late one would land in the
      // barriers of the next kernel's CTA (the decode groups wait for theirs below).
      int own = 0;
      ring.each_last(SB, [&](uint32_t slot, uint32_t phase) {
        mbar_wait(B_BFULL(slot), phase, &own, p.status, 512u);
        mbar_wait(B_BEMPTY(slot), phase, &own, p.status, 512u);
      });
    }
  } else if (warp == W_MMA) {
    if (rank == 0) {
      // ================================================================ MMA issuer (leader CTA)
      // The whole warp walks the list and one elected lane issues: addresses and descriptors then stay in uniform
      // registers, where the MMA takes them (all of tensor memory is allocated, so its base is column 0).
      // instruction descriptor: fp32 accumulate, fp16 A and B, both K-major, N = NT, M = 256
      const uint32_t IDESC = (1u << 4) | ((NT >> 3) << 17) | (16u << 24);
      const uint32_t bring = smem_u32(smem + p.off_bring);
      if (tmem != 0) {
        s_state = ABORTED;
        if (p.status && lane == 0) atomicOr(p.status, 1024u);
      }
      __syncwarp();
      uint32_t lu = 0;
      Ring rb, ra;
      WorkList<MANY> wl(p, cluster, n_clusters, IPT);
      Work w;
      for (; wl.next(w); ++lu) {
        const uint32_t dbuf = lu % ND;
        const uint32_t td = D_BASE + dbuf * NT;
        if (lu >= ND) mbar_wait(B_DEMPTY(dbuf), ((lu / ND) - 1) & 1, &s_state, p.status, 4u);
        tc_fence_after();
        for (uint32_t j = w.j0; j < w.j1; ++j) {
          // one wait an item: everything that stands between two items idles the tensor core
          const bool ok = mbar_wait(B_READY(ra.slot), ra.phase, &s_state, p.status, 8u);
          if (!__all_sync(0xffffffffu, ok)) break;           // nothing is issued on operands that never came
          tc_fence_after();
          const uint64_t bdesc = smem_desc(bring + rb.slot * B_GRAN_BYTES, 8, 16);
          const uint32_t ta = ra.slot * A_COLS;
          if (elect_one()) {
            if (j < NCH) {
              umma_ts(td, ta, bdesc, IDESC, j != w.j0);
            } else {
              umma_ts(td, ta, bdesc, IDESC, j != w.j0);
#pragma unroll
              for (uint32_t ks = 1; ks < 8; ++ks) umma_ts(td, ta + ks * 8, bdesc + ks * (B_KSTEP_BYTES >> 4), IDESC, 1u);
            }
            tc_commit_pair(B_AEMPTY(ra.slot));
            if (SB != NA) tc_commit_pair(B_BEMPTY(rb.slot));
          }
          __syncwarp();
          ra.advance(NA);
          rb.advance(SB);
        }
        if (elect_one()) tc_commit_pair(B_DFULL(dbuf));
        __syncwarp();
      }
      if (*(volatile int*)&s_state == ABORTED) __nanosleep(100000);     // (after a wait that ran out: let issued MMAs finish)
    }
  } else if (warp < W_MMA) {
    // ================================================================ decode groups
    const int grp = warp >> 2;
    const int row = (warp & 3) * 32 + lane;                 // row of the tile = tensor-memory lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint8_t* wring = smem + p.off_wring;
    static_assert(NA == NGRP, "a decode group owns one A slot");
    uint32_t n = 0, turn = 0;                               // items before this piece modulo NGRP; items of this group so far
    const uint32_t a = grp;
    // the group steps from one of its items to the next, every NGRP-th, in the rings too (both have NGRP stages and more)
    Ring ring, rb;
    ring.slot = rb.slot = grp;
    const uint32_t ready = rank == 0 ? B_READY(a) : cluster_addr(B_READY(a), 0);
    WorkList<MANY> wl(p, cluster, n_clusters, IPT);
    Work w;
    while (wl.next(w)) {
      const uint32_t first = w.j0 + (grp >= (int)n ? grp - n : grp + NGRP - n);
      n = (n + w.j1 - w.j0) % NGRP;
      for (uint32_t j = first; j < w.j1; j += NGRP) {
        const uint32_t sw = ring.slot, wphase = ring.phase, sb = rb.slot, bphase = rb.phase;
        ring.skip(NGRP, SW);
        rb.skip(NGRP, SB);
        mbar_wait(B_WFULL(sw), wphase, &s_state, p.status, 32u);
        const uint8_t* item = wring + (size_t)sw * p.wstage_bytes;
        const bool cherry = j < NCH;
        uint4 raw[BITS];
        uint32_t s0 = 0, s1 = 0;
        if (cherry) {
          raw[0] = *reinterpret_cast<const uint4*>(item + row * 16);
          raw[1] = *reinterpret_cast<const uint4*>(item + 2048 + row * 16);
        } else {
#pragma unroll
          for (int q = 0; q < BITS; ++q) raw[q] = *reinterpret_cast<const uint4*>(item + q * 2048 + row * 16);
          const unsigned short* sc = reinterpret_cast<const unsigned short*>(item + 2048 * BITS);
          s0 = dup16(sc[row]);
          s1 = (SETS == 2) ? dup16(sc[128 + row]) : s0;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(B_WEMPTY(sw));
        if (turn) mbar_wait(B_AEMPTY(a), (turn - 1) & 1, &s_state, p.status, 64u);
        ++turn;
        tc_fence_after();
        const uint32_t ta = tmem + lane_addr + a * A_COLS;
        if (cherry) {
          const uint32_t v[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
          tmem_st8(ta, v);
        } else {
          const uint32_t* wds = reinterpret_cast<const uint32_t*>(raw);
          if constexpr (BITS == 4) {
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              uint32_t v[16];
#pragma unroll
              for (int e = 0; e < 4; ++e) dequant4(wds[4 * c4 + e], (c4 < 2) ? s0 : s1, v + 4 * e);
              tmem_st16(ta + 16 * c4, v);
            }
          } else {
#pragma unroll
            for (int t3 = 0; t3 < 4; ++t3) {
              uint32_t v[16];
              dequant3(wds[3 * t3], wds[3 * t3 + 1], wds[3 * t3 + 2], (t3 < 2) ? s0 : s1, v);
              tmem_st16(ta + 16 * t3, v);
            }
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          // The group's first warp also answers for the activation tile.  (No wait by parity comes a round early: the
          // MMAs of item n - 4 are done, so the slot's last tile, of an item n - SB <= n - 4, has landed.)
          if ((warp & 3) == 0) mbar_wait(B_BFULL(sb), bphase, &s_state, p.status, 16u);
          if (rank == 0) mbar_arrive(ready);
          else mbar_arrive_cluster(ready);
        }
      }
    }
    if (turn) mbar_wait(B_AEMPTY(a), (turn - 1) & 1, &s_state, p.status, 64u);
  } else {
    // ================================================================ epilogue (last four warps)
    const int quad = warp & 3;                              // the tensor-memory lanes this warp may read
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const int etid = tid - (NGRP * 4 + 3) * 32;             // 0..127 among the epilogue threads
    const int ewarp = etid >> 5;
    __half* stage = reinterpret_cast<__half*>(smem + p.off_stage);      // [token][128 rows]
    auto epi_sync = [&]() { asm volatile("bar.sync 2, 128;" ::: "memory"); };
    dependency_wait();
    uint32_t lu = 0;
    WorkList<MANY> wl(p, cluster, n_clusters, IPT);
    Work w;
    for (; wl.next(w); ++lu) {
      const PrefillLayer& L = p.layer[MANY ? w.layer : 0];
      const uint32_t NPAIR = ((uint32_t)L.n_tile + 1) / 2;
      const uint32_t mb = w.unit / NPAIR, tile = 2 * (w.unit % NPAIR) + rank;
      const uint32_t dbuf = lu % ND;
      const uint32_t d_lu = tmem + lane_addr + D_BASE + dbuf * NT;
      const int tok0 = (int)(mb * NT), ntok = min((int)NT, p.M - tok0);
      const int n0 = (int)tile * 128, nrows = min(128, L.N - n0);       // <= 0: the repeated tile of an odd pair
      if (w.run < 0) {
        if (p.accumulate && nrows > 0) {
          // the old outputs into the staging area while the MMAs run
          for (int i = etid; i < ntok * 16; i += 128) {
            const int t = i >> 4, r8 = (i & 15) * 8;
            if (r8 < nrows) {
              const __half* yp = L.y + (size_t)(tok0 + t) * L.ldy + n0 + r8;
              if (p.vec_y) {
                *reinterpret_cast<uint4*>(stage + t * 128 + r8) = *reinterpret_cast<const uint4*>(yp);
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) stage[t * 128 + r8 + e] = yp[e];
              }
            }
          }
          epi_sync();
        }
        mbar_wait(B_DFULL(dbuf), (lu / ND) & 1, &s_state, p.status, 128u);
        tc_fence_after();
        // (NT is a multiple of 32: a 32-column step may read padding, never past the accumulator)
#pragma unroll 1
        for (int c = 0; c < ntok; c += 32) {
          float v[2][16];
          tmem_ld16(d_lu + c, v[0]);
          tmem_ld16(d_lu + c + 16, v[1]);
          tmem_wait_ld();
          __half* sp = stage + c * 128 + row;
          // (the bias meets the rounded output, as in a kernel after this one)
          if (p.accumulate) {
#pragma unroll
            for (int e = 0; e < 32; ++e) sp[e * 128] = __float2half(v[e >> 4][e & 15] + __half2float(sp[e * 128]));
          } else if (L.bias) {
            const __half b = row < nrows ? L.bias[n0 + row] : __float2half(0.f);
#pragma unroll
            for (int e = 0; e < 32; ++e) sp[e * 128] = __hadd(__float2half(v[e >> 4][e & 15]), b);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) sp[e * 128] = __float2half(v[e >> 4][e & 15]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(B_DEMPTY(dbuf), 0));
        epi_sync();
        for (int i = etid; i < ntok * 16; i += 128) {
          const int t = i >> 4, r8 = (i & 15) * 8;
          if (r8 < nrows) {
            __half* yp = L.y + (size_t)(tok0 + t) * L.ldy + n0 + r8;
            if (p.vec_y) {
              *reinterpret_cast<uint4*>(yp) = *reinterpret_cast<const uint4*>(stage + t * 128 + r8);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) yp[e] = stage[t * 128 + r8 + e];
            }
          }
        }
        epi_sync();
      } else {
        // a part of a unit: park the fp32 tile; the cluster that arrives last adds the parts in item order and
        // stores the outputs
        const size_t part_floats = (size_t)NT * 128;
        float* mine = L.partial + ((size_t)(cluster * 2 + w.run) * 2 + rank) * part_floats;
        mbar_wait(B_DFULL(dbuf), (lu / ND) & 1, &s_state, p.status, 128u);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < ntok; c += 32) {
          float v[2][16];
          tmem_ld16(d_lu + c, v[0]);
          tmem_ld16(d_lu + c + 16, v[1]);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) mine[(c + e) * 128 + row] = v[e >> 4][e & 15];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(B_DEMPTY(dbuf), 0));
        // clusters whose runs touch this unit
        const uint32_t total = L.sk_units * IPT, i0 = w.unit * IPT;
        const uint32_t c_first = ((i0 + 1) * L.sk_clusters - 1) / total, c_last = ((i0 + IPT) * L.sk_clusters - 1) / total;
        __threadfence();
        epi_sync();
        if (etid == 0) s_last = (atomicAdd(L.arrived + 2 * w.unit + rank, 1u) == c_last - c_first) ? 1 : 0;
        epi_sync();
        if (s_last && nrows > 0) {
          __threadfence();
          // a warp takes every fourth token, a lane four rows of it, four tokens' loads in flight; only the first
          // cluster's run can have begun in an earlier unit (its part is then that cluster's last)
          const uint32_t run0 = run_begin(L, c_first, total) >= i0 ? 0u : 1u;
          const float4* parts = reinterpret_cast<const float4*>(L.partial + (size_t)(c_first * 4 + rank) * part_floats) + lane;
          const size_t part_step = part_floats;               // one cluster's four parts, in float4
          for (int t0 = ewarp; t0 < ntok; t0 += 16) {
            float4 sum[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) sum[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t c = 0; c <= c_last - c_first; c += 2) {
              const bool two = c < c_last - c_first;
              const float4* src = parts + c * part_step + (c == 0 ? run0 * (part_floats / 2) : 0);
              const float4* src2 = parts + (c + 1) * part_step;
              float4 f[4], g[4];                            // two parts of four tokens in flight
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const size_t at = (size_t)min(t0 + 4 * u, ntok - 1) * 32;
                f[u] = __ldcg(src + at);
                g[u] = two ? __ldcg(src2 + at) : make_float4(0.f, 0.f, 0.f, 0.f);
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                sum[u].x += f[u].x; sum[u].y += f[u].y; sum[u].z += f[u].z; sum[u].w += f[u].w;
                sum[u].x += g[u].x; sum[u].y += g[u].y; sum[u].z += g[u].z; sum[u].w += g[u].w;
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int t = t0 + 4 * u;
              const float4 s = sum[u];
              if (t >= ntok) break;
              if (4 * lane < nrows) {
                __half* yp = L.y + (size_t)(tok0 + t) * L.ldy + n0 + 4 * lane;
                float r[4] = {s.x, s.y, s.z, s.w};
                if (p.accumulate) {
#pragma unroll
                  for (int e = 0; e < 4; ++e) r[e] += __half2float(yp[e]);
                } else if (L.bias) {
#pragma unroll
                  for (int e = 0; e < 4; ++e) r[e] = __half2float(__float2half(r[e])) + __half2float(L.bias[n0 + 4 * lane + e]);
                }
                if (p.vec_y) {
                  const __half2 a = __floats2half2_rn(r[0], r[1]), b = __floats2half2_rn(r[2], r[3]);
                  uint2 o;
                  o.x = *reinterpret_cast<const uint32_t*>(&a);
                  o.y = *reinterpret_cast<const uint32_t*>(&b);
                  *reinterpret_cast<uint2*>(yp) = o;
                } else {
#pragma unroll
                  for (int e = 0; e < 4; ++e) yp[e] = __float2half(r[e]);
                }
              }
            }
          }
        }
        epi_sync();
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync();              // no CTA leaves while the other may still signal its barriers or read its shared memory
  tc_fence_after();
  if (warp == W_MMA) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

struct PDeviceInfo { int sms = 0, max_smem = 0; bool ok = false; };
PDeviceInfo pdevice_info(int dev) {
  static PDeviceInfo cache[64];
  if (dev < 0 || dev >= 64) return PDeviceInfo();
  if (!cache[dev].ok) {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return PDeviceInfo();
    cache[dev].sms = prop.multiProcessorCount;
    cache[dev].max_smem = (int)prop.sharedMemPerBlockOptin - 256;     // (the kernel's static variables)
    cache[dev].ok = true;
  }
  return cache[dev];
}

int palign_up(int v, int a) { return (v + a - 1) / a * a; }

typedef void (*PKernelFn)(const PrefillParams);
template <bool MANY> PKernelFn ppick(int bits, int sets) {
  if (bits == 4) return sets == 1 ? cq_prefill_kernel<4, 1, MANY> : cq_prefill_kernel<4, 2, MANY>;
  return sets == 1 ? cq_prefill_kernel<3, 1, MANY> : cq_prefill_kernel<3, 2, MANY>;
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }
// the pair MMA takes N = 32 .. 256 in steps of 32; blocks of equal size, so that 300 rows are two of 160
int token_blocks(int M) { return (M + 255) / 256; }
int block_tokens(int M) {
  const int nb = token_blocks(M);
  return ((M + nb - 1) / nb + 31) & ~31;
}
unsigned long long xb_half_bytes(const cq_tlayer* L, int nt) {
  return (unsigned long long)L->n_cher * b_kstep_bytes(nt) + (unsigned long long)L->n_gran * b_gran_bytes(nt);
}
size_t part_bytes(int nt) { return (size_t)nt * 128 * sizeof(float); }

// Weight stages used of those that fit: a multiple of the decode groups.  Items go round the groups, so a slot then always
// belongs to one group, which has finished the slot's last round before it waits for the next: a wait by parity that
// comes a round early (another group's item of the slot not yet landed) would pass at once.
constexpr int weight_stages(int fit) { return (fit > SW_MAX ? SW_MAX : fit) / NGRP * NGRP; }
static_assert(SW_MAX % NGRP == 0 && weight_stages(5) == 4 && weight_stages(11) == 8 && weight_stages(30) == 12, "ring / group binding");

// Workspace: staged activations | fp32 partial tiles (two per CTA) | arrival counters.  Covers every smaller call too.
size_t xb_bytes_for(const cq_tlayer* L, int M) {
  const size_t per_token = (size_t)L->n_cher * 32 + (size_t)L->n_gran * 256;
  return align256(((size_t)M + 32 * (size_t)token_blocks(M)) * per_token);
}
size_t partial_bytes_for(int M, int clusters) {
  const int nt = M >= 256 ? 256 : (M + 31) & ~31;
  return (size_t)clusters * 4 * part_bytes(nt);
}

// Over how many clusters the `rem` units that do not fill a wave are cut, 0 = they stay whole.  In SM cycles, as measured:
// an item takes 4.5 NT, at least 740; a part costs about 20 NT and a fixed 500 (its fp32 tile is parked, and the last
// arriver reads it in steps of four tokens a warp, each a trip to L2).
int pick_runs(uint32_t rem, uint32_t items, int nt, int clusters) {
  const double t_item = 4.5 * nt > 740.0 ? 4.5 * nt : 740.0, t_part = 500.0 + 20.0 * nt;
  double best = (double)items * t_item;
  int runs = 0;
  for (int g = (int)rem + 1; g <= clusters; ++g) {
    const double t = std::ceil((double)rem * items / g) * t_item + ((double)g / rem + 1.0) * t_part;
    if (t < best) { best = t; runs = g; }
  }
  return runs;
}

}  // namespace

// Workspace of n layers: staged activations of each | partial tiles of each | arrival counters of each
extern "C" size_t cq_tlayers_gemm_workspace_bytes(const cq_tlayer* L, int n_layers, int M) {
  if (!L || M < 1 || n_layers < 1 || n_layers > MAX_LAYERS) return 0;
  int dev = 0;
  PDeviceInfo di;
  if (cudaGetDevice(&dev) == cudaSuccess) di = pdevice_info(dev);
  else (void)cudaGetLastError();
  const int clusters = (di.ok ? di.sms : 148) / 2;
  return n_layers * (xb_bytes_for(L, M) + partial_bytes_for(M, clusters) + align256((size_t)clusters * 2 * sizeof(uint32_t)));
}
extern "C" size_t cq_tlayer_gemm_workspace_bytes(const cq_tlayer* L, int M) { return cq_tlayers_gemm_workspace_bytes(L, 1, M); }

extern "C" int cq_tlayer_gemm(const cq_tlayer* L, const void* x, int ldx, void* y, int ldy, int M, int accumulate,
                              void* workspace, uint32_t* status_word, cq_stream_t stream) {
  return cq_tlayers_gemm(&L, 1, x, ldx, &y, &ldy, nullptr, M, accumulate, workspace, status_word, stream);
}

extern "C" int cq_tlayers_gemm(const cq_tlayer* const* layers, int n_layers, const void* x, int ldx, void* const* ys, const int* ldys,
                               const void* const* biases, int M, int accumulate, void* workspace, uint32_t* status_word, cq_stream_t stream) {
  if (!layers || n_layers < 1 || n_layers > MAX_LAYERS || !ys || !ldys || !x || !workspace) return CQ_ERR_BAD_ARG;
  const cq_tlayer* L = layers[0];
  if (!L || M < 1 || ldx < L->K || ((uintptr_t)x & 1) || ((uintptr_t)workspace & 127)) return CQ_ERR_BAD_ARG;
  for (int i = 0; i < n_layers; ++i) {
    const cq_tlayer* l = layers[i];
    if (!l || !l->blob || !ys[i] || ldys[i] < l->N || ((uintptr_t)ys[i] & 1)) return CQ_ERR_BAD_ARG;
    if (biases && biases[i] && (accumulate || ((uintptr_t)biases[i] & 1))) return CQ_ERR_BAD_ARG;
    if (l->K != L->K || l->C != L->C || l->G != L->G || l->bits != L->bits) return CQ_ERR_BAD_SHAPE;
  }
  int dev = 0;
  CQ_CUDA_TRY(cudaGetDevice(&dev));
  const PDeviceInfo di = pdevice_info(dev);
  if (!di.ok) return CQ_ERR_NO_DEVICE;
  cudaStream_t st = (cudaStream_t)stream;
  const int NT = block_tokens(M), n_mblk = (M + NT - 1) / NT;
  const int clusters = di.sms / 2;
  const uint32_t items = (uint32_t)(L->n_cher + L->n_gran);

  PrefillParams p = {};
  StageLayers stage = {};
  p.status = status_word;
  p.n_layers = n_layers;
  p.M = M; p.n_gran = L->n_gran; p.n_cher = L->n_cher;
  p.gran_bytes = L->gran_bytes; p.tile_bytes = L->tile_bytes; p.accumulate = accumulate;
  p.vec_y = 1;
  p.nt = NT;
  p.xb_half_bytes = xb_half_bytes(L, NT);
  uint8_t* xb = (uint8_t*)workspace;
  uint8_t* partial = xb + n_layers * xb_bytes_for(L, M);
  uint32_t* arrived = (uint32_t*)(partial + n_layers * partial_bytes_for(M, clusters));
  uint32_t used = 0, n_arrived = 0;
  for (int i = 0; i < n_layers; ++i) {
    const cq_tlayer* l = layers[i];
    const uint8_t* blob = (const uint8_t*)l->blob;
    PrefillLayer& d = p.layer[i];
    d.stream = blob + l->off_stream;
    d.xb = stage.xb[i] = xb + i * xb_bytes_for(L, M);
    d.y = (__half*)ys[i];
    d.bias = biases ? (const __half*)biases[i] : nullptr;
    d.N = l->N; d.n_tile = l->n_tile; d.ldy = ldys[i];
    d.n_units = (uint32_t)n_mblk * (uint32_t)((l->n_tile + 1) / 2);
    const uint32_t rem = d.n_units % (uint32_t)clusters;
    d.sk_clusters = rem ? (uint32_t)pick_runs(rem, items, NT, clusters) : 0;
    d.sk_units = d.sk_clusters ? rem : 0;
    d.partial = (float*)(partial + i * partial_bytes_for(M, clusters));
    d.arrived = arrived + n_arrived;
    n_arrived += 2 * d.sk_units;                     // (fewer than the clusters, for which there is room)
    used = std::max(used, d.n_units >= (uint32_t)clusters ? (uint32_t)clusters : (d.sk_clusters ? d.sk_clusters : d.n_units));
    if (((uintptr_t)ys[i] & 15) || ldys[i] % 8) p.vec_y = 0;
    stage.osh[i] = (const uint32_t*)(blob + l->off_osh);
    stage.cidx[i] = (const uint16_t*)(blob + l->off_cidx);
  }

  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = attr;
  {
    const int quads = (2 * L->n_cher + 16 * L->n_gran + 3) / 4, groups = (M + 7) / 8;
    // four token groups a thread once that still fills the SMs (2048 rows of 5120: 10 us against 18), one below it
    // (64 rows of 4096: four would add 4 us of latency to a 24 us call)
    const int gx = (quads + STAGE_THREADS / 32 - 1) / (STAGE_THREADS / 32);
    const bool four = (long long)gx * n_layers * ((groups + 3) / 4) >= 10ll * di.sms;
    const int gy = four ? (groups + 3) / 4 : groups;
    cfg.gridDim = dim3(gx, gy < 65535 ? gy : 65535, n_layers);
    cfg.blockDim = dim3(STAGE_THREADS);
    cfg.numAttrs = 1;
    const int aligned16 = ((uintptr_t)x & 15) == 0 && ldx % 8 == 0;
    CQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, four ? prefill_stage_x_kernel<4> : prefill_stage_x_kernel<1>, (const __half*)x, ldx, M,
                                   stage, (int)L->C, (int)L->Kc, (int)L->n_gran, (int)L->n_cher, p.xb_half_bytes, NT, arrived,
                                   (int)n_arrived, aligned16));
  }

  // shared memory: barriers, output staging tile, activation ring, and weights in what is left
  p.wstage_bytes = palign_up(L->gran_bytes > CQT_CHER_BYTES ? L->gran_bytes : CQT_CHER_BYTES, 128);
  int off = 0;
  p.off_bar = off;   off = palign_up(off + N_BARS * 8, 128);
  p.off_stage = off; off += NT * 128 * 2;
  p.sb = (di.max_smem - off - NGRP * p.wstage_bytes) / b_gran_bytes(NT);
  if (p.sb > NA) {
    const int even = (di.max_smem - off) / (p.wstage_bytes + b_gran_bytes(NT));       // about as many stages of both
    p.sb = even < NA ? NA : (even > SB_MAX ? SB_MAX : even);
  }
  p.off_bring = off; off += p.sb * b_gran_bytes(NT);
  p.off_wring = off;
  p.sw = weight_stages((di.max_smem - off) / p.wstage_bytes);
  if (p.sb < NA || p.sw < NGRP) return CQ_ERR_TOO_LARGE;
  const int smem = off + p.sw * p.wstage_bytes;

  PKernelFn fn = n_layers > 1 ? ppick<true>(L->bits, L->sets) : ppick<false>(L->bits, L->sets);
  CQ_CUDA_TRY(cq_grant_smem((const void*)fn, smem));
  cfg.gridDim = dim3(2 * used);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.numAttrs = 2;
  CQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, p));
  return CQ_OK;
}
