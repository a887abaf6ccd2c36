// Decode path, row-owning form: y[M<=16, N] = x[M, K] * dequant(W[N, K])^T, bf16 and f16, HBM-bound.
//
// Replaces cu::qmv_kernel / the small-M use of cu::qmm_sm80_kernel of the reference
// (mlx/backend/cuda/quantized/qmm/qmv.cu:84-209, quantized.cpp:106-136).
//
// Design (one persistent CTA per SM; 16 consumer warps, a loader, a scales and two reducer warps; no
// scratch in global memory):
//  * Every CTA owns a contiguous range of 8-row blocks of W for the WHOLE of K, so no output is
//    shared between CTAs: no global atomics, no arrival counters, no workspace.
//  * A stage is 16 weight rows x one K phase.  The loader warp brings it in with one untiled bulk copy per two rows (where the
//    phase is all of K they are contiguous; else per row) into pairs of rows whose pitch is an odd multiple of 16 bytes, so that eight
//    pairs are read without bank conflicts: the MMA's upper rows are the stage's even rows.  No tensor map: nothing to encode per call,
//    no descriptor to fetch before the first byte, and no rule on K beyond rows of whole 16 bytes.  (A copy costs the issuing warp
//    about 100 cycles whatever its size; an SM's share of HBM delivers 16 rows of 2 KB in 1500.)
//  * The scales warp copies the rows' scales and biases with cp.async in the widest pieces that their alignment allows.  Its
//    instructions count, since every warp of a scheduler gets one in five to ten cycles: a loop with cases inside it, or half the lanes
//    along a row, made it the slowest part of short stages; the consumers fetching their own cost them 10 % and more.
//  * K is cut into 16 slices, one per consumer warp.  A warp keeps the x values of its slice in
//    registers for the whole phase, as mma.sync B fragments in the order the unpack produces the
//    weights: x is read from L2 once per CTA and never touches shared memory.
//  * A field masked in place and read as a bf16 (or f16) number with an empty exponent is the subnormal number
//    field * 2^(offset - 133) (2^(offset - 24)), exactly, and the tensor cores take subnormal inputs exactly.  Two fields whose
//    distance brings them into the two halves of a register within the subnormal's 8 bits are unpacked by one AND (and a shift
//    that several pairs share); the offsets' powers of two go into x.  The integer pipe, which issues at half rate, bounds the
//    unpacking: 5 operations per 8 four-bit weights, 3 per 4 eight-bit, 9 per 16 two-bit, 26 to 34 per 32 of 3, 5 and 6 bits.
//    To keep the products inside fp32's range whatever the magnitude of x, every token row of a
//    warp's K slice is multiplied by a power of two, 2^126 at most, that brings its largest element to about 2^126
//    (less where the field sits some bits up) when it is put into registers, and the warp's sums
//    are multiplied back by the matching power of two before they leave the warp: exact.
//  * Scales are applied per group to fp32 group sums:  y = sum_g s_g * (sum_k x_k q_k) + sum_g b_g * (sum_k x_k).
//    Two forms, by how fields lie in memory:
//      units   2, 4 and 8 bits: 16 bytes of a row, of which ldmatrix gives every lane of a quad one word, lie inside one group, so
//              an MMA sums inside a group; two groups at a time keep two accumulation chains going.
//      runs    3, 5 and 6 bits (fields straddle words) and 2 bits in groups of 32: a lane owns 32 consecutive fields of each
//              128, so the four lanes of a quad hold different groups.  The groups are kept apart in the MMA's columns: column
//              (token, group of the 128) has x in the lanes of its group and zeros in the others.  M = 1 fills one tile of 8 columns
//              for any group size.
//  * The consumer warps leave fp32 partial sums in shared memory; a reducer warp adds them in
//    warp order (the result does not depend on timing), converts and stores y.  What is not finite (an infinite x: the
//    factored form cannot give the sign) is computed again from the weights themselves at the end, unless its token's x has a NaN.
//  * Grouped launches (mixture-of-experts decode) walk a table of (expert, up to 8 rows) tiles: blocks take contiguous
//    ranges of (tile, 16-row group) units, x and y rows are found through the sort's slot tables.
#pragma once
#include <type_traits>

#include "bounded_wait.h"
#include "common.cuh"
#include "kernels.h"
#include "qmv_rows.h"
#include "tc_ptx.cuh"

namespace b200q {
namespace rows {

using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_test;
using tc::smem_u32;

// Registers are handed out per group of four warps; the two kinds of warps re-balance their register budgets at entry.
constexpr int kThreads = (kConsumers + 4) * 32;
// (WIDE in groups of 64, with eight groups' sums beside 64 registers of x, wants 112 and leaves the others 32: one row through
// [28672, 8192] 24.4 us, 27.9 with 104; in groups of 128 23.1 with 104, 24.2 with 112.)
__host__ __device__ constexpr int regs_consumer(bool more) { return more ? 112 : 104; }
__host__ __device__ constexpr int regs_service(bool more) { return more ? 32 : 64; }
// setmaxnreg only moves registers inside what the block was launched with (96 per thread at this
// block size): a request beyond that pool would wait forever.
constexpr bool in_pool(bool more) { return regs_consumer(more) * kConsumers * 32 + regs_service(more) * 4 * 32 <= 96 * kThreads; }
static_assert(in_pool(false) && in_pool(true), "register budgets exceed the launch allocation");

template <typename T>
constexpr bool is_bf16 = std::is_same<T, __nv_bfloat16>::value;

template <typename T>
__device__ __forceinline__ uint32_t mul_x2(uint32_t a, uint32_t b) {
  uint32_t d;
  if constexpr (is_bf16<T>) asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  else asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
template <typename T>
__device__ __forceinline__ uint32_t pack_x2(float lo, float hi) {
  uint32_t d;
  if constexpr (is_bf16<T>) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
template <typename T>
__device__ __forceinline__ void mma16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (is_bf16<T>)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same with nothing to add to.
template <typename T>
__device__ __forceinline__ void mma16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (is_bf16<T>)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
// Four 8x8 matrices of 16-bit elements; lane l supplies the address of row l%8 of matrix l/8 and
// receives, from matrix m, the 32-bit word (l%4) of row l/4.
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr)
               : "memory");
}
// `bytes` (a multiple of 16) from global to shared memory, both 16-byte aligned, counted on `bar`.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// N bytes, of which the first `n` are read and the rest are zeros.
template <int N>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(n) : "memory");
}
__device__ __forceinline__ uint4 ldg_nc_u128(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ldg_nc_u64(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
template <typename T>
__device__ __forceinline__ float lo_f(uint32_t v) {
  if constexpr (is_bf16<T>) return __uint_as_float(v << 16);
  else return __half2float(__ushort_as_half((unsigned short)(v & 0xFFFFu)));
}
template <typename T>
__device__ __forceinline__ float hi_f(uint32_t v) {
  if constexpr (is_bf16<T>) return __uint_as_float(v & 0xFFFF0000u);
  else return __half2float(__ushort_as_half((unsigned short)(v >> 16)));
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void lds_u64(uint32_t addr, uint32_t& a, uint32_t& b) {
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr));
}
__device__ __forceinline__ void sts_rows(uint32_t addr, float a, float b) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

// Bounded wait (0.65 s) that never parks the thread (try_wait may suspend it for a hardware-chosen time) and leaves issue slots to
// the warps that share the scheduler.  For a whole warp: all lanes go on or none.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xFFFFFFFFu, bounded_wait([=] { return mbar_test(bar, parity); }, [] { __nanosleep(20); }, [] { return false; }, 1u << 23,
                                              abort_flag));
}
// The same for the loader and the scales warp, which start before the others and count from when those go: the word after the flag.
// (Hardware barriers for that, before their first wait, cost decode 5 to 10 %.)
__device__ __forceinline__ bool early_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xFFFFFFFFu, bounded_wait([=] { return mbar_test(bar, parity); }, [] { __nanosleep(20); }, [=] { return abort_flag[1] == 0; },
                                              1u << 23, abort_flag));
}

// ---- units: one packed word -> NP registers of two subnormals each; register i holds fields (i, i + NP) of the word
template <int BITS>
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t* P) {
  const uint32_t u = w >> 8;
  if constexpr (BITS == 4) {
    P[0] = w & 0x000F000Fu; P[1] = w & 0x00F000F0u; P[2] = u & 0x000F000Fu; P[3] = u & 0x00F000F0u;
  } else if constexpr (BITS == 8) {
    P[0] = w & 0x00FF00FFu; P[1] = u & 0x00FF00FFu;
  } else {
    P[0] = w & 0x00030003u; P[1] = w & 0x000C000Cu; P[2] = w & 0x00300030u; P[3] = w & 0x00C000C0u;
    P[4] = u & 0x00030003u; P[5] = u & 0x000C000Cu; P[6] = u & 0x00300030u; P[7] = u & 0x00C000C0u;
  }
}
// Binary places by which field i of a word sits above bit 0 of its byte: x pair i is scaled down by
// as many powers of two.
template <int BITS>
__host__ __device__ constexpr int field_shift(int i) {
  return BITS == 4 ? ((i & 1) ? 4 : 0) : (BITS == 8 ? 0 : 2 * (i & 3));
}

// ---- runs: pair j (0..15) of a lane's 32 fields.  Fields a and b sit at bits oa and 16 + ob of the 32 bits from bit `at` on
// (both within the 8 bits of a bf16 subnormal); joined: the pair comes from two shifts instead (a at 0, b at 16).
struct RunPair { int a, b, at, oa, ob; bool joined; };
template <int BITS>
__host__ __device__ constexpr RunPair run_pair(int j) {
  if (BITS == 2) {          // fields i and i + 8 of a word are 16 bits apart
    const int w = j >> 3, i = j & 7;
    return {16 * w + i, 16 * w + i + 8, 32 * w + (i & 4 ? 8 : 0), 2 * (i & 3), 2 * (i & 3), false};
  }
  if (BITS == 3) {
    if (j < 12) {           // 18 bits apart; one window serves two pairs
      const int f = 12 * (j / 6) + 2 * ((j % 6) >> 1), odd = j & 1;
      return {f + odd, f + odd + 6, 3 * f, 3 * odd, 3 * odd + 2, false};
    }
    const int f = 24 + (j - 12);   // the last eight: 12 bits apart
    return {f, f + 4, 3 * f - 4, 4, 0, false};
  }
  // 5 and 6 bits: 15 or 18 bits apart, six fields after six, and two left over
  if (j < 15) {
    const int f = 6 * (j / 3) + j % 3;
    return BITS == 5 ? RunPair{f, f + 3, 5 * f - 1, 1, 0, false} : RunPair{f, f + 3, 6 * f, 0, 2, false};
  }
  return {30, 31, 0, 0, 0, true};
}
template <int BITS, int J>
__device__ __forceinline__ uint32_t run_bits(const uint32_t (&w)[BITS]) {
  constexpr RunPair p = run_pair<BITS>(J);
  constexpr uint32_t m = (1u << BITS) - 1u;
  if constexpr (p.joined) {
    constexpr int pa = p.a * BITS - 32 * (BITS - 1), pb = p.b * BITS - 32 * (BITS - 1);   // both in the last word
    static_assert(pa >= 0 && pb >= 16, "fields of the last word");
    return ((w[BITS - 1] >> pa) & m) | ((w[BITS - 1] >> (pb - 16)) & (m << 16));
  } else {
    constexpr int wi = p.at < 0 ? 0 : p.at >> 5, sh = p.at < 0 ? 0 : p.at & 31;
    uint32_t v;
    if constexpr (p.at < 0) v = w[0] << -p.at;
    else if constexpr (sh == 0) v = w[wi];
    else if constexpr (sh + 16 + p.ob + BITS <= 32) v = w[wi] >> sh;
    else v = __funnelshift_r(w[wi], w[(wi + 1) % BITS], sh);
    return v & (m << p.oa | m << (16 + p.ob));
  }
}
template <int BITS>
__device__ __forceinline__ void run_words(uint32_t addr, uint32_t (&w)[BITS]) {   // pitches make these free of bank conflicts
  if constexpr (BITS % 2 == 0) {
#pragma unroll
    for (int i = 0; i < BITS; i += 2) lds_u64(addr + 4 * i, w[i], w[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < BITS; ++i) w[i] = lds_u32(addr + 4 * i);
  }
}

// A run of consecutive 16-row groups of one tile.  Units of grouped work are (tile, row group) pairs in that order; a
// block takes a contiguous range of them, which spans two tiles at most while there are fewer tiles than blocks.
struct Segment {
  int row0;        // first row of the run inside the matrix
  int base;        // rows of the stack before the matrix
  int n;           // row groups
  int x0, rows;    // first sorted row and number of rows of the tile
};
__device__ __forceinline__ Segment segment_at(const RowsParams& p, int u, int u_end) {
  const int tile = u / p.rgs, rg = u - tile * p.rgs;
  const int4 t = p.tiles[tile];
  return Segment{rg * 16, t.x * p.N, min(p.rgs - rg, u_end - u), t.y, t.z};
}
// Row of x or y that sorted row r stands for.
__device__ __forceinline__ long long slot_row(const int* table, int r, int per) {
  if (table == nullptr) return r;
  const int q = r / per;
  return (long long)table[q] * per + (r - q * per);
}

// One element from the weights themselves, in fp32, by a warp, until a lane's sum is a NaN.
template <typename T, int BITS>
__device__ __forceinline__ float exact_dot(const RowsParams& p, int which, long long row, const uint16_t* x, int lane) {
  const uint32_t* w = p.wq[which] + row * (p.row_bytes / 4);
  const uint16_t *s = p.scales[which] + row * p.groups, *b = p.biases[which] + row * p.groups;
  const int sh = 31 - __clz(p.K / p.groups);   // (32 neighbouring k are of one group)
  float sum = 0.0f;
#pragma unroll 1
  for (int k = lane; k < p.K; k += 32) {
    const int gi = k >> sh;
    sum = fmaf(lo_f<T>(x[k]), fmaf((float)stream_get<BITS>(w, k), lo_f<T>(s[gi]), lo_f<T>(b[gi])), sum);
    if (__any_sync(0xFFFFFFFFu, sum != sum)) break;
  }
#pragma unroll
  for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
  return sum;
}
template <typename T>
__device__ __forceinline__ bool not_finite(uint16_t v) {
  constexpr uint16_t kExp = is_bf16<T> ? 0x7F80 : 0x7C00;
  return (v & kExp) == kExp;
}
__device__ __forceinline__ float gated(float a, float b) { return __fdividef(a, 1.f + __expf(-a)) * b; }
// Whether K values at x, a whole number of 128 on a 16-byte boundary, have a NaN among them, by a warp.
template <typename T>
__device__ __forceinline__ bool has_nan(const uint16_t* x, int K, int lane) {
  constexpr uint32_t kInf = is_bf16<T> ? 0x7F807F80u : 0x7C007C00u;
  uint32_t found = 0;
#pragma unroll 1
  for (int k = 8 * lane; k < K; k += 256) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + k);
    found |= __vcmpgtu2(v.x & 0x7FFF7FFFu, kInf) | __vcmpgtu2(v.y & 0x7FFF7FFFu, kInf) | __vcmpgtu2(v.z & 0x7FFF7FFFu, kInf) |
             __vcmpgtu2(v.w & 0x7FFF7FFFu, kInf);
  }
  return __any_sync(0xFFFFFFFFu, found != 0);
}

// SHAPE: units: the group size; runs: tiles of 8 columns.  MT: units: tiles of 8 tokens.
template <typename T, int BITS, bool RUNS, int SHAPE, int MT, Work W, bool WIDE>
__global__ void __launch_bounds__(kThreads, 1)
qmv_rows_kernel(const __grid_constant__ RowsParams p) {
  constexpr bool kGrouped = W != Work::Plain;
  constexpr int NW = W == Work::Gated ? 2 : 1;
  constexpr bool kMoreRegs = WIDE && SHAPE == 64;
  static_assert(!kGrouped || MT == 1, "grouped tiles have up to 8 rows");
  extern __shared__ __align__(1024) unsigned char smem[];
  // header: [0, 128) "stage landed" barriers | [128, 256) "stage consumed" barriers |
  //         [256, 288) "partial buffer free" barriers | [288, 320) "partial buffer full" | 320: abort flag, "all go"
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t full0 = smem_base, done0 = smem_base + 128, pfree0 = smem_base + 256, pfull0 = smem_base + 288;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 320);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  asm volatile("griddepcontrol.launch_dependents;");

  const int nst = p.nst;
  // The range of this CTA: plain, 8-row blocks [b0, b1) as one segment; grouped, units [b0, b1), which are known only
  // once the table has been written.
  int b0 = 0, b1 = 0;
  Segment seg{};
  auto find_range = [&]() {
    if constexpr (kGrouped) {
      const long long n = (long long)*p.n_tiles * p.rgs;
      b0 = (int)(blockIdx.x * n / gridDim.x);
      b1 = (int)((blockIdx.x + 1) * n / gridDim.x);
    } else {   // (no division: it took part of every launch's start)
      b0 = (int)blockIdx.x * p.blk_each + min((int)blockIdx.x, p.blk_more);
      b1 = b0 + p.blk_each + ((int)blockIdx.x < p.blk_more ? 1 : 0);
    }
  };
  if constexpr (!kGrouped) {
    find_range();
    seg = Segment{b0 * 8, 0, (b1 - b0 + 1) >> 1, 0, p.M};
  }
  const int row_end = kGrouped ? p.N : min(b1 * 8, p.N);
  // Grouped: on to the segment that starts at unit `at`; false when there is none.  (A plain launch has its one segment
  // from the start, and every role's loop over segments folds away.)
  auto next_segment = [&](int& at) -> bool {
    if (at >= b1) return false;
    seg = segment_at(p, at, b1);
    at += seg.n;
    return true;
  };

  // Which partial buffer a row group's sums go into.  One token tile: that of the reducer warp which takes the row group (each
  // has one or, gated, two of its own, so neither can miss a phase of a barrier while it is busy); two: in turn.
  auto buffer_of = [&](int rg, int nth) { return MT == 2 ? nth & 1 : (NW == 2 ? rg & 3 : rg & 1); };

  // Barriers are set up by the loader warp, which then starts requesting weights at once; the
  // other warps meet it at a named barrier (id 1) only when they first need the barriers - the
  // consumers after their x values are in registers.
  if (warp >= kConsumers) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(regs_service(kMoreRegs)));
    if (warp == kConsumers) {
      if (lane < nst) {
        mbar_init(full0 + 8 * lane, 33);           // the loader's announcement and the scales warp's lanes
        mbar_init(done0 + 8 * lane, p.n_active);
      }
      if (lane < partial_bufs(W)) {
        mbar_init(pfree0 + 8 * lane, MT);
        mbar_init(pfull0 + 8 * lane, p.n_active);
      }
      if (lane == 0) abort_flag[0] = abort_flag[1] = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      __syncwarp();
      asm volatile("bar.arrive 2, 64;" ::: "memory");   // the scales warp does not wait for the others
      if (MT == 1) asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
      // ================================= loader warp ==========================================
      // Without the caller's promise the weights may have been written by the previous kernel.
      if (kGrouped || !p.early) asm volatile("griddepcontrol.wait;" ::: "memory");
      if constexpr (kGrouped) find_range();
      int slot = 0, use = 0, at = b0;
      // one phase: lanes 0..7, two rows each; several: lanes 0..15, a row's part each
      const bool pairs = p.nph == 1;
      const int lane_row = pairs ? 2 * lane : lane;
      uint32_t dst = smem_base + p.off_slots + (lane_row >> 1) * p.pitch + (lane_row & 1) * p.phase_bytes;
      bool more = !kGrouped || next_segment(at), ok = true, met = false;
      while (more) {
        const int nrg = seg.n * NW;
        for (int ph = 0; ok && ph < p.nph; ++ph) {
          const uint32_t off = (uint32_t)ph * p.phase_bytes, bytes = min(p.phase_bytes, p.row_bytes - off);
          for (int rg = 0; rg < nrg; ++rg) {
            // slot free: all consumer warps arrived for the stage that used it last
            if (use > 0 && !early_wait(done0 + 8 * slot, (use - 1) & 1, abort_flag)) { ok = false; break; }
            const int row = seg.row0 + (NW == 2 ? rg >> 1 : rg) * 16, rows = min(16, p.N - row);
            const uint32_t bar = full0 + 8 * slot;
            if (lane == 0) mbar_expect_tx(bar, rows * bytes);
            __syncwarp();
            // (rows past the end keep what is there: their products are never stored)
            if (lane_row < rows)
              bulk_copy(dst, reinterpret_cast<const char*>(p.wq[NW == 2 ? rg & 1 : 0]) + (long long)(seg.base + row + lane_row) * p.row_bytes + off,
                        pairs && lane_row + 1 < rows ? 2 * bytes : bytes, bar);
            dst += p.slot_bytes;
            if (++slot == nst) { slot = 0; ++use; dst -= nst * p.slot_bytes; }
            // One stage; the rest once the consumers have asked for x, which would else wait behind a ring full of weights (one row of
            // x through [14336, 4096]: 8400 cycles instead of 3000), or, with x of 9 to 16 tokens, once they have it (16 rows: 14.1 us
            // against 15.1; 3 rows of f16 through [11008, 4096] at 8 bits the other way, 12.3 and 11.65).
            if (!met) {
              met = true;
              if (MT == 2) asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
              else asm volatile("bar.sync 4, %0;" ::"r"(32 * (p.n_active + 1)) : "memory");
            }
          }
        }
        more = kGrouped && ok && next_segment(at);
      }
      if (!ok) {   // the copies in flight still write to this block's shared memory
        for (int i = 0; i < nst; ++i) {
          const int n = use + (i < slot ? 1 : 0);
          for (int k = 0; n > 0 && k < (1 << 14) && !mbar_test(full0 + 8 * i, (n - 1) & 1); ++k) {}
        }
      }
    } else if (warp == kConsumers + 3) {
      // ================================= scales warp ==========================================
      asm volatile("bar.sync 2, 64;" ::: "memory");
      asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
      if (kGrouped || !p.early) asm volatile("griddepcontrol.wait;" ::: "memory");
      if constexpr (kGrouped) find_range();
      int slot = 0, use = 0, at = b0;
      const int r = lane >> 1;   // two lanes per row, pieces in turn
      uint32_t ds = smem_base + p.off_slots + p.off_scales + (r >> 1) * p.spitch + (r & 1) * p.shalf;
      const uint32_t db = 8 * p.spitch;
      bool more = !kGrouped || next_segment(at), ok = true;
      while (more) {
        const int nrg = seg.n * NW;
        for (int ph = 0; ok && ph < p.nph; ++ph) {
          const int g0 = ph * p.phase_groups, bytes = 2 * min(p.phase_groups, p.groups - g0), all = p.s_bytes;   // (zeros beyond the row)
          for (int rg = 0; rg < nrg; ++rg) {
            if (use > 0 && !early_wait(done0 + 8 * slot, (use - 1) & 1, abort_flag)) { ok = false; break; }
            const int row = seg.row0 + (NW == 2 ? rg >> 1 : rg) * 16, which = NW == 2 ? rg & 1 : 0;
            const long long src = ((long long)(seg.base + min(row + r, p.N - 1)) * p.groups + g0) * 2;
            const char* s = reinterpret_cast<const char*>(p.scales[which]) + src;
            const char* b = reinterpret_cast<const char*>(p.biases[which]) + src;
            if (p.s_piece == 16 && bytes == all) {
              for (int o = (lane & 1) * 16; o < all; o += 32) { cp_async<16>(ds + o, s + o, min(16, all - o)); cp_async<16>(ds + db + o, b + o, min(16, all - o)); }
            } else {
              const int piece = p.s_piece;
              for (int o = (lane & 1) * piece; o < all; o += 2 * piece) {
                const int n = max(min(piece, bytes - o), 0), at_o = n > 0 ? o : 0;
                if (piece == 16) { cp_async<16>(ds + o, s + at_o, n); cp_async<16>(ds + db + o, b + at_o, n); }
                else if (piece == 8) { cp_async<8>(ds + o, s + at_o, n); cp_async<8>(ds + db + o, b + at_o, n); }
                else if (piece == 4) { cp_async<4>(ds + o, s + at_o, n); cp_async<4>(ds + db + o, b + at_o, n); }
                else {
                  asm volatile("st.shared.u16 [%0], %1;" ::"r"(ds + o), "h"(n ? *reinterpret_cast<const unsigned short*>(s + o) : (unsigned short)0) : "memory");
                  asm volatile("st.shared.u16 [%0], %1;" ::"r"(ds + db + o), "h"(n ? *reinterpret_cast<const unsigned short*>(b + o) : (unsigned short)0) : "memory");
                }
              }
            }
            if (p.s_piece > 2) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + 8 * slot) : "memory");
            else tc::mbar_arrive(full0 + 8 * slot);
            ds += p.slot_bytes;
            if (++slot == nst) { slot = 0; ++use; ds -= nst * p.slot_bytes; }
          }
        }
        more = kGrouped && ok && next_segment(at);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
      // ================================= reducer warps ========================================
      // Add the consumer warps' partial sums of a finished stage in warp order, free the partial buffer, and store y (or
      // keep running sums while K is walked in phases).  A lane has four consecutive rows of a token.  Each of the two warps takes
      // every other row group, or (MT = 2) eight of the tokens: one warp took longer per stage than the products.
      const int mine = warp - (kConsumers + 1), mt = MT == 2 ? mine : 0;
      asm volatile("griddepcontrol.wait;" ::: "memory");   // y may still be in use by the previous kernel
      if (lane == 0) peer_wait_previous(p.sig, p.status);  // ... or by a peer's consumer of the step before
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
      abort_flag[1] = 1;   // all go: every role that waits for something outside the block has done so (a store in the consumers: 10 %)
      if constexpr (kGrouped) find_range();
      constexpr int kLoads = kMoreRegs ? 2 : 8;   // partial sums under way at a time
      const int r4 = 4 * (lane & 3), tok = mt * 8 + g;
      int red = 0, uses = 0, at = b0;
      bool more = !kGrouped || next_segment(at), odd = false;   // odd: a sum of this lane's was not finite
      while (more) {
        int rph = 0, rrg = 0;
        const int nrg = seg.n * NW, end = red + nrg * p.nph;
        [[maybe_unused]] uint2 gate = make_uint2(0, 0);
        const long long y_off = (kGrouped ? slot_row(p.dst_slot, seg.x0 + min(tok, seg.rows - 1), p.per_slot) : (long long)tok) * p.ld + p.col0;
        for (; red < end; ++red) {
          const int pbi = buffer_of(rrg, red);
          if (MT == 2 || (NW == 2 ? pbi >> 1 : pbi) == mine) {
            if (!warp_wait(pfull0 + 8 * pbi, (MT == 2 || NW == 2 ? uses >> 1 : uses) & 1, abort_flag)) break;
            ++uses;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tok < seg.rows) {
              const unsigned char* pb = smem + p.off_pbuf + (size_t)pbi * p.pbuf_bytes + (tok * tok_pitch(W) + r4) * 4;
#pragma unroll
              for (int w = 0; w < kConsumers; w += kLoads) {   // independent loads, then the additions in warp order
                float4 v[kLoads];
#pragma unroll
                for (int i = 0; i < kLoads; ++i)
                  v[i] = w + i < p.n_active ? *reinterpret_cast<const float4*>(pb + (size_t)(w + i) * p.pwarp_bytes) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < kLoads; ++i) { sum.x += v[i].x; sum.y += v[i].y; sum.z += v[i].z; sum.w += v[i].w; }
              }
            }
            __syncwarp();   // every lane holds its sums: the partial buffer may be written again
            if (lane == 0) tc::mbar_arrive(pfree0 + 8 * pbi);
            bool final_phase = true;
            if (p.nph > 1) {   // long K: running sums of this CTA's rows, touched by this warp only
              float4* tl = reinterpret_cast<float4*>(smem + p.off_run + (size_t)rrg * (MT * 512) + mt * 512) + lane;
              final_phase = rph == p.nph - 1;
              if (rph > 0) {
                const float4 v = *tl;
                sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
              }
              if (!final_phase) *tl = sum;
            }
            if (final_phase) {
              const int row0 = seg.row0 + (NW == 2 ? rrg >> 1 : rrg) * 16, r = row0 + r4;
              const bool live = tok < seg.rows && r < row_end;
              odd = odd || (live && !(fabsf(sum.x) + fabsf(sum.y) + fabsf(sum.z) + fabsf(sum.w) < INFINITY));
              uint2 v = make_uint2(pack_x2<T>(sum.x, sum.y), pack_x2<T>(sum.z, sum.w));
              bool store = live;
              if constexpr (W == Work::Gated) {
                if ((rrg & 1) == 0) {   // the gate's product waits, rounded
                  gate = v;
                  store = false;
                } else {
                  v.x = pack_x2<T>(gated(lo_f<T>(gate.x), lo_f<T>(v.x)), gated(hi_f<T>(gate.x), hi_f<T>(v.x)));
                  v.y = pack_x2<T>(gated(lo_f<T>(gate.y), lo_f<T>(v.y)), gated(hi_f<T>(gate.y), hi_f<T>(v.y)));
                }
              }
              if (store) {
                const long long off = y_off + r;
                for (int q = 0; q < p.n_out; ++q) {
                  uint16_t* dst = p.y[q] + off;
                  if (r + 4 <= row_end && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
                    *reinterpret_cast<uint2*>(dst) = v;
                  } else {
                    const uint16_t* e = reinterpret_cast<const uint16_t*>(&v);
                    for (int i = 0; i < 4 && r + i < row_end; ++i) dst[i] = e[i];
                  }
                }
              }
            }
          }
          if (++rrg == nrg) { rrg = 0; ++rph; }
        }
        more = kGrouped && red == end && next_segment(at);
      }
      // What this warp has stored that is not finite, once more from the weights: here, where no role waits for it any more.
      // (In the loop above one row of x with a NaN was N sums of K products that the block's other roles waited for.)
      if (__any_sync(0xFFFFFFFFu, odd)) {
        at = b0;
        more = !kGrouped || next_segment(at);
        while (more) {
          uint32_t looked = 0, nans = 0;   // a bit per token of the warp's eight: x has been looked at, has a NaN
          const long long y_off = (kGrouped ? slot_row(p.dst_slot, seg.x0 + min(tok, seg.rows - 1), p.per_slot) : (long long)tok) * p.ld + p.col0;
          for (int rg = MT == 2 ? 0 : mine; rg < seg.n; rg += MT == 2 ? 1 : 2) {
            const int row0 = seg.row0 + rg * 16;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              const int r = row0 + r4 + c;
              bool again = tok < seg.rows && r < row_end;
              if (again) again = not_finite<T>(p.y[0][y_off + r]);
#pragma unroll 1
              for (uint32_t bad = __ballot_sync(0xFFFFFFFFu, again); bad; bad &= bad - 1) {
                const int who = __ffs(bad) - 1;
                const uint32_t bit = 1u << (who >> 2);
                const uint16_t* x = p.x + (kGrouped ? slot_row(p.src_slot, seg.x0 + (who >> 2), p.per_slot) : mt * 8 + (who >> 2)) * p.K;
                if (!(looked & bit)) {
                  looked |= bit;
                  if (has_nan<T>(x, p.K, lane)) nans |= bit;
                }
                if (nans & bit) continue;   // a NaN, as it stands
                const long long row = seg.base + row0 + 4 * (who & 3) + c;
                float v = 0.0f;
#pragma unroll 1
                for (int i = 0; i < NW; ++i) {
                  const float before = v;
                  v = lo_f<T>(pack_x2<T>(exact_dot<T, BITS>(p, i, row, x, lane), 0.0f));
                  if (i == 1) v = gated(before, v);
                }
                if (lane == who)
                  for (int q = 0; q < p.n_out; ++q) p.y[q][y_off + r] = (uint16_t)pack_x2<T>(v, 0.0f);
              }
            }
          }
          more = kGrouped && next_segment(at);
        }
        __syncwarp();
      }
      if (p.sig.n > 0) {   // all of this block's stores to y were issued by these two warps
        __threadfence_system();
        asm volatile("bar.sync 3, 64;" ::: "memory");
      }
      if (lane == 0) end_of_role([&] { if (mine == 0) peer_signal_tail(p.sig); }, abort_flag, p.status, 7u);
    }
    return;
  }

  // ================================= consumer warps ===========================================
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(regs_consumer(kMoreRegs)));
  auto meet = [&]() {   // before the first stage: the barriers exist from here on
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
  };
  if (warp >= p.n_active) {   // fewer slices than warps
    meet();
    return;
  }
  {
    // The first mma.sync of a kernel is slow (the tensor pipe wakes up): issue one now.  Its result is never used.
    float d[4];
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%4,%4,%4}, {%4,%4}, {%5,%5,%5,%5};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(0u), "f"(0.0f));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (p.sig.wait_flag != nullptr && p.sig.wait_x) {   // x is the gathered output of the previous exchange step
    if (lane == 0) peer_wait_previous(p.sig, p.status);
    __syncwarp();
  }
  if constexpr (kGrouped) find_range();
  int at = b0;
  if (kGrouped && !next_segment(at)) {   // no work for this block
    meet();
    return;
  }
  constexpr uint32_t kOne = is_bf16<T> ? 0x00800080u : 0x04000400u;      // one binary place of both halves
  constexpr uint32_t kOnes = is_bf16<T> ? 0x3F803F80u : 0x3C003C00u;     // (1, 1)
  constexpr float kOut = is_bf16<T> ? 0x1p8f : 1.0f;
  // x is multiplied by 2^E, E up to 126, so that its largest element, whose bits are `m`, lands at or below 2^127 (f16: 2^15): with the
  // weights' 2^-133 the sums are within 2^-7 of true units for x up to 1, and results down to the smallest numbers keep their bits.
  // (The powers of two below that the fields ask for stay normal numbers; sums beyond fp32 end up infinite and are computed again.)
  auto exponent = [](uint32_t m) -> int {
    if constexpr (is_bf16<T>) {
      const int E = 253 - (int)(m >> 7);
      return E < -2 ? -2 : (E > 126 ? 126 : E);
    } else {
      const int E = 29 - (int)(m >> 10);
      return E < -8 ? -8 : (E > 15 ? 15 : E);
    }
  };
  // the larger of two positive numbers of either type, twice
  auto max_x2 = [](uint32_t a, uint32_t b) {   // (abs and max of packed numbers; a NaN among them changes nothing that matters)
    uint32_t d;
    if constexpr (is_bf16<T>) asm("{.reg .b32 t; abs.bf16x2 t, %2; max.bf16x2 %0, %1, t;}" : "=r"(d) : "r"(a), "r"(b));
    else asm("{.reg .b32 t; abs.f16x2 t, %2; max.f16x2 %0, %1, t;}" : "=r"(d) : "r"(a), "r"(b));
    return d;
  };
  // the largest of a quad's (both halves)
  auto quad_max = [](uint32_t m) {
    m = __vmaxu2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
    m = __vmaxu2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
    return max(m & 0xFFFFu, m >> 16);
  };
  // The weights come out as field * 2^-133 (f16: 2^-24): sums are true value * 2^(E - 133).  2^(125 - E) is applied when they
  // leave the warp, 2^8 with it (f16: 2^(24 - E)).
  auto unscale_of = [](int E) { return __uint_as_float((uint32_t)(127 + (is_bf16<T> ? 125 : 24) - E) << 23); };

  int slot = 0, use = 0, nth = 0;
  uint32_t pphase = 0;   // per partial buffer: parity of its uses so far
  uint32_t sb = smem_base + p.off_slots;   // stage the warp works on
  const uint32_t pb_mine = smem_base + p.off_pbuf + warp * p.pwarp_bytes;
  bool first = true, more = true;
  while (more) {
    const int nrg = seg.n * NW;
    for (int ph = 0; ph < p.nph; ++ph) {
      const int i0 = warp * p.cnt;                                                       // first item of this warp in the phase
      const int lim = min(p.cnt, min(p.phase_items, p.items - ph * p.phase_items) - i0);   // items that it has (may be negative)
      if constexpr (!RUNS) {
        // ---------------------------------------------------------------------- units
        using C = UnitsCfg<BITS, SHAPE, MT, WIDE>;
        constexpr int NGW = C::NGW, NP = C::NP, UG = C::UG, UW = C::UW, KW = C::KW;
        uint32_t X[UW][MT][NP];         // B fragments of this warp's K slice, pre-scaled
        uint32_t sx_hi[MT], sx_lo[MT];  // scaled group sums of x for groups 2t, 2t+1 of the slice (hi / lo parts)
        float unscale[MT][2];           // per output token (2t, 2t+1 of tile mt): what brings the warp's sums back to true units / kOut
        const uint16_t* xr[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int tok = mt * 8 + g;
          xr[mt] = p.x + (kGrouped ? slot_row(p.src_slot, seg.x0 + min(tok, seg.rows - 1), p.per_slot) : (long long)min(tok, seg.rows - 1)) * p.K +
                   (long long)(ph * p.phase_items + i0) * SHAPE + t * KW;
        }
        // unit i of the slice: 4 * KW consecutive k, of which this lane owns KW starting at t * KW
#pragma unroll
        for (int i = 0; i < UW; ++i) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const bool live = i < lim * UG && mt * 8 + g < seg.rows;
            const uint16_t* xp = xr[mt] + i * (4 * KW);
            // pair q = (x_q, x_{q + NP}), the order the unpack delivers the fields in
            if constexpr (BITS == 8) {
              uint2 v = make_uint2(0, 0);
              if (live) v = ldg_nc_u64(xp);
              X[i][mt][0] = __byte_perm(v.x, v.y, 0x5410); X[i][mt][1] = __byte_perm(v.x, v.y, 0x7632);
            } else if constexpr (BITS == 4) {
              uint4 v = make_uint4(0, 0, 0, 0);
              if (live) v = ldg_nc_u128(xp);
              X[i][mt][0] = __byte_perm(v.x, v.z, 0x5410); X[i][mt][1] = __byte_perm(v.x, v.z, 0x7632);
              X[i][mt][2] = __byte_perm(v.y, v.w, 0x5410); X[i][mt][3] = __byte_perm(v.y, v.w, 0x7632);
            } else {
              uint4 a = make_uint4(0, 0, 0, 0), b = make_uint4(0, 0, 0, 0);
              if (live) { a = ldg_nc_u128(xp); b = ldg_nc_u128(xp + 8); }
              X[i][mt][0] = __byte_perm(a.x, b.x, 0x5410); X[i][mt][1] = __byte_perm(a.x, b.x, 0x7632);
              X[i][mt][2] = __byte_perm(a.y, b.y, 0x5410); X[i][mt][3] = __byte_perm(a.y, b.y, 0x7632);
              X[i][mt][4] = __byte_perm(a.z, b.z, 0x5410); X[i][mt][5] = __byte_perm(a.z, b.z, 0x7632);
              X[i][mt][6] = __byte_perm(a.w, b.w, 0x5410); X[i][mt][7] = __byte_perm(a.w, b.w, 0x7632);
            }
          }
        }
        if (MT == 1 && first) asm volatile("bar.arrive 4, %0;" ::"r"(32 * (p.n_active + 1)) : "memory");   // x is on its way
        // Group sums of x by MMAs with x as the other operand (tokens as rows, times ones; summing by adds took 9 instructions
        // per register, most of the 3000 cycles between a launch's start and its first product).  Lane t keeps groups 2t, 2t+1.
        float e[MT][2];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) e[mt][0] = e[mt][1] = 0.0f;
#pragma unroll
        for (int j = 0; j < NGW; ++j) {
          float d[4];
#pragma unroll
          for (int iu = 0; iu < UG; ++iu)
#pragma unroll
            for (int st = 0; st < NP / 2; ++st) {
              const uint32_t(&x0)[NP] = X[j * UG + iu][0];
              const uint32_t(&x1)[NP] = X[j * UG + iu][MT - 1];
              const uint32_t a1 = MT == 2 ? x1[2 * st] : 0u, a3 = MT == 2 ? x1[2 * st + 1] : 0u;
              if (iu == 0 && st == 0) mma16_first<T>(d, x0[2 * st], a1, x0[2 * st + 1], a3, kOnes, kOnes);
              else mma16<T>(d, x0[2 * st], a1, x0[2 * st + 1], a3, kOnes, kOnes);
            }
          if ((j >> 1) == t) {
            e[0][j & 1] = d[0];
            if constexpr (MT == 2) e[1][j & 1] = d[2];
          }
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          uint32_t m = 0;
#pragma unroll
          for (int i = 0; i < UW; ++i)
#pragma unroll
            for (int q = 0; q < NP; ++q) m = max_x2(m, X[i][mt][q]);
          const int E = exponent(quad_max(m));
          const uint32_t sc2 = (uint32_t)((is_bf16<T> ? 127 : 15) + E) * kOne;   // 2^E twice
#pragma unroll
          for (int i = 0; i < UW; ++i)
#pragma unroll
            for (int q = 0; q < NP; ++q) X[i][mt][q] = mul_x2<T>(X[i][mt][q], sc2 - (uint32_t)field_shift<BITS>(q) * kOne);
          const float un = unscale_of(E);
          unscale[mt][0] = __shfl_sync(0xFFFFFFFFu, un, (2 * t) * 4);
          unscale[mt][1] = __shfl_sync(0xFFFFFFFFu, un, (2 * t + 1) * 4);
          // the group sums in the sums' units (f16: times 2^(E - 9): 128 of the largest element stay finite, and what the lower
          // part loses is 2^-30 of the largest element)
          const float down = is_bf16<T> ? __uint_as_float((uint32_t)(127 + E - 64) << 23) : __uint_as_float((uint32_t)(118 + E) << 23);
          constexpr float kDown = is_bf16<T> ? 0x1p-69f : 1.0f;   // (a factor of its own: 2^(E - 133) may be no number)
          const float e0 = e[mt][0] * down * kDown, e1 = e[mt][1] * down * kDown;
          const uint32_t hi = pack_x2<T>(e0, e1);
          sx_hi[mt] = hi;
          sx_lo[mt] = pack_x2<T>(e0 - lo_f<T>(hi), e1 - hi_f<T>(hi));
        }
        if (first) { meet(); first = false; }
        // ldmatrix roles of this lane: matrix m = lane / 8 covers rows (m & 1) * 8 .. +7 of unit (m >> 1)
        // (row i of the MMA's upper half is row 2i of the stage, of its lower half row 2i + 1)
        const uint32_t w_off = (lane & 7) * p.pitch + ((lane >> 3) & 1) * p.phase_bytes + (i0 * UG + (lane >> 4)) * 16;
        const uint32_t s_off = p.off_scales + g * p.spitch + 2 * i0, s8 = p.shalf;
        for (int rg = 0; rg < nrg; ++rg) {
          if (!warp_wait(full0 + 8 * slot, use & 1, abort_flag)) return;
          float out[MT][4];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int c = 0; c < 4; ++c) out[mt][c] = 0.0f;
          const uint32_t wa = sb + w_off, sa = sb + s_off;
#pragma unroll
          for (int gq = 0; gq < NGW; gq += 2) {
            if (gq < lim) {
              float acc[2][MT][4];
              // (a group past the row's end multiplies what is there with x registers that are zero, and with a zero scale)
              uint32_t sl2, sh2;
              auto read_scales = [&]() { sl2 = lds_u32(sa + 2 * gq); sh2 = lds_u32(sa + s8 + 2 * gq); };
              if constexpr (BITS == 8) read_scales();   // (4 bits: after the words)
              // units iu, iu + 1 of both groups (of one unit each: both at once); a few words at a time, for registers
              constexpr int UB = UG == 1 ? 1 : 2;
#pragma unroll
              for (int i0u = 0; i0u < UG; i0u += UB) {
                // packed words: lane (g, t) gets word t of a unit for rows g (wl) and g + 8 (wh)
                uint32_t wl[2][UB], wh[2][UB];
                if constexpr (UG == 1) {
                  ldmatrix_x4(wa + gq * 16, wl[0][0], wh[0][0], wl[1][0], wh[1][0]);
                } else {
#pragma unroll
                  for (int u = 0; u < 2; ++u) ldmatrix_x4(wa + ((gq + u) * UG + i0u) * 16, wl[u][0], wh[u][0], wl[u][UB - 1], wh[u][UB - 1]);
                }
                if (BITS != 8 && i0u == 0) read_scales();
#pragma unroll
                for (int iu = i0u; iu < i0u + UB; ++iu) {
#pragma unroll
                  for (int u = 0; u < 2; ++u) {
                    uint32_t Pl[NP], Ph[NP];
                    unpack_word<BITS>(wl[u][iu - i0u], Pl);
                    unpack_word<BITS>(wh[u][iu - i0u], Ph);
#pragma unroll
                    for (int st = 0; st < NP / 2; ++st)
#pragma unroll
                      for (int mt = 0; mt < MT; ++mt) {
                        const uint32_t(&x)[NP] = X[(gq + u) * UG + iu][mt];
                        if (iu == 0 && st == 0) mma16_first<T>(acc[u][mt], Pl[2 * st], Ph[2 * st], Pl[2 * st + 1], Ph[2 * st + 1], x[2 * st], x[2 * st + 1]);
                        else mma16<T>(acc[u][mt], Pl[2 * st], Ph[2 * st], Pl[2 * st + 1], Ph[2 * st + 1], x[2 * st], x[2 * st + 1]);
                      }
                  }
                }
              }
              const float s_l[2] = {lo_f<T>(sl2), hi_f<T>(sl2)}, s_h[2] = {lo_f<T>(sh2), hi_f<T>(sh2)};
#pragma unroll
              for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                  for (int c = 0; c < 4; ++c) out[mt][c] = fmaf(c < 2 ? s_l[u] : s_h[u], acc[u][mt][c], out[mt][c]);
            }
          }
          // biases: b_g * sum_k x_k through one MMA, k slots 2t, 2t+1 (hi part of the sum) / +8 (lo part)
          {
            const uint32_t ba = sa + 8 * p.spitch + 4 * t;
            uint32_t bl = 0, bh = 0;
            if (2 * t < p.cnt) { bl = lds_u32(ba); bh = lds_u32(ba + s8); }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              if constexpr (is_bf16<T>) {
                mma16<T>(out[mt], bl, bh, bl, bh, sx_hi[mt], sx_lo[mt]);
              } else {
                float ob[4];   // in units of 2^(E - 9); out: 2^(E - 24)
                mma16_first<T>(ob, bl, bh, bl, bh, sx_hi[mt], sx_lo[mt]);
#pragma unroll
                for (int c = 0; c < 4; ++c) out[mt][c] = fmaf(ob[c], 0x1p-15f, out[mt][c]);
              }
            }
          }
          // the partial buffer has been read by its reducer
          const int pbi = buffer_of(rg, nth);
          if (!warp_wait(pfree0 + 8 * pbi, (pphase >> pbi & 1) ^ 1, abort_flag)) return;
          pphase ^= 1u << pbi;
          ++nth;
          const uint32_t pa = pb_mine + (uint32_t)pbi * p.pbuf_bytes;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {   // back to true units on the way out (exact multiplications)
              const int tok = mt * 8 + 2 * t + h;
              if (tok < seg.rows) sts_rows(pa + (tok * tok_pitch(W) + 2 * g) * 4, out[mt][h] * kOut * unscale[mt][h], out[mt][2 + h] * kOut * unscale[mt][h]);
            }
          __syncwarp();
          if (lane == 0) {   // only here: the stores have consumed what was read from the slot, which the copies may now overwrite
            tc::mbar_arrive(pfull0 + 8 * pbi);
            tc::mbar_arrive(done0 + 8 * slot);
          }
          sb += p.slot_bytes;
          if (++slot == nst) { slot = 0; ++use; sb = smem_base + p.off_slots; }
        }
      } else {
        // ---------------------------------------------------------------------- runs
        constexpr int NT = SHAPE, CW = run_chunks(NT);   // chunks of 128 k per warp and phase
        const int ng = p.ng, sh = ng == 4 ? 2 : ng - 1;   // groups per chunk, log2 of it
        const int need = (seg.rows * ng + 7) >> 3;       // column tiles in use
        uint32_t X[CW][NT][16];
        float xs[CW][NT][2], unscale[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const int col = nt * 8 + g, tok = col >> sh;
          const bool mine = tok < seg.rows && ((t * ng) >> 2) == (col & (ng - 1));   // this lane's 32 k are of the column's group
          const uint16_t* xr = p.x + (kGrouped ? slot_row(p.src_slot, seg.x0 + min(tok, seg.rows - 1), p.per_slot) : (long long)min(tok, seg.rows - 1)) * p.K +
                               (long long)(ph * p.phase_items + i0) * 128 + t * 32;
          uint32_t m = 0;
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            uint4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              v[i] = make_uint4(0, 0, 0, 0);
              if (mine && j < lim) v[i] = ldg_nc_u128(xr + j * 128 + 8 * i);
            }
            const uint32_t R[16] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w,
                                    v[2].x, v[2].y, v[2].z, v[2].w, v[3].x, v[3].y, v[3].z, v[3].w};
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              m = max_x2(m, R[q]);
              const RunPair rp = run_pair<BITS>(q);
              X[j][nt][q] = __byte_perm(R[rp.a >> 1], R[rp.b >> 1], (rp.a & 1 ? 0x32 : 0x10) | (rp.b & 1 ? 0x7600 : 0x5400));
            }
            float d[4];   // sums of x over the lane's columns 2t, 2t+1
#pragma unroll
            for (int st = 0; st < 8; ++st) {
              if (st == 0) mma16_first<T>(d, kOnes, kOnes, kOnes, kOnes, X[j][nt][0], X[j][nt][1]);
              else mma16<T>(d, kOnes, kOnes, kOnes, kOnes, X[j][nt][2 * st], X[j][nt][2 * st + 1]);
            }
            xs[j][nt][0] = d[0];
            xs[j][nt][1] = d[1];
          }
          if (MT == 1 && nt == 0 && first) asm volatile("bar.arrive 4, %0;" ::"r"(32 * (p.n_active + 1)) : "memory");   // x is on its way
          const int E = exponent(quad_max(m));
          const uint32_t e1 = (uint32_t)((is_bf16<T> ? 127 : 15) + E);
#pragma unroll
          for (int j = 0; j < CW; ++j)
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const RunPair rp = run_pair<BITS>(q);
              constexpr int kExp = is_bf16<T> ? 7 : 10;
              X[j][nt][q] = mul_x2<T>(X[j][nt][q], e1 * kOne - ((uint32_t)rp.oa << kExp) - ((uint32_t)rp.ob << (16 + kExp)));
            }
          const float un = unscale_of(E);
          const float down = __uint_as_float((uint32_t)(127 + E - (is_bf16<T> ? 64 : 24)) << 23);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            unscale[nt][h] = __shfl_sync(0xFFFFFFFFu, un, (2 * t + h) * 4);
            const float dn = __shfl_sync(0xFFFFFFFFu, down, (2 * t + h) * 4);
#pragma unroll
            for (int j = 0; j < CW; ++j) xs[j][nt][h] = xs[j][nt][h] * dn * (is_bf16<T> ? 0x1p-69f : 1.0f);
          }
        }
        if (first) { meet(); first = false; }
        const uint32_t w_off = g * p.pitch + i0 * (16 * BITS) + t * (4 * BITS), w8 = p.phase_bytes;
        const uint32_t c0 = 2 * ((2 * t) & (ng - 1)), c1 = 2 * ((2 * t + 1) & (ng - 1));   // byte offsets of the columns' groups in a chunk
        const uint32_t s_off = p.off_scales + g * p.spitch + 2 * (i0 << sh), s8 = p.shalf;
        for (int rg = 0; rg < nrg; ++rg) {
          if (!warp_wait(full0 + 8 * slot, use & 1, abort_flag)) return;
          float out[NT][4];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) out[nt][c] = 0.0f;
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            if (j < lim) {
              const uint32_t wa = sb + w_off + j * (16 * BITS), sa = sb + s_off + 2 * (j << sh), ba = sa + 8 * p.spitch;
              uint32_t wl[BITS], wh[BITS];
              run_words<BITS>(wa, wl);
              run_words<BITS>(wa + w8, wh);
              const float sl0 = lo_f<T>(lds_u16(sa + c0)), sl1 = lo_f<T>(lds_u16(sa + c1));
              const float sh0 = lo_f<T>(lds_u16(sa + s8 + c0)), sh1 = lo_f<T>(lds_u16(sa + s8 + c1));
              const float bl0 = lo_f<T>(lds_u16(ba + c0)), bl1 = lo_f<T>(lds_u16(ba + c1));
              const float bh0 = lo_f<T>(lds_u16(ba + s8 + c0)), bh1 = lo_f<T>(lds_u16(ba + s8 + c1));
              float acc[NT][4];
              auto step = [&](auto stag) {
                constexpr int st = decltype(stag)::value;
                const uint32_t a0 = run_bits<BITS, 2 * st>(wl), a1 = run_bits<BITS, 2 * st>(wh);
                const uint32_t a2 = run_bits<BITS, 2 * st + 1>(wl), a3 = run_bits<BITS, 2 * st + 1>(wh);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                  if (nt > 0 && nt >= need) continue;
                  if constexpr (st == 0) mma16_first<T>(acc[nt], a0, a1, a2, a3, X[j][nt][0], X[j][nt][1]);
                  else mma16<T>(acc[nt], a0, a1, a2, a3, X[j][nt][2 * st], X[j][nt][2 * st + 1]);
                }
              };
              step(std::integral_constant<int, 0>{}); step(std::integral_constant<int, 1>{});
              step(std::integral_constant<int, 2>{}); step(std::integral_constant<int, 3>{});
              step(std::integral_constant<int, 4>{}); step(std::integral_constant<int, 5>{});
              step(std::integral_constant<int, 6>{}); step(std::integral_constant<int, 7>{});
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                if (nt > 0 && nt >= need) continue;
                out[nt][0] = fmaf(sl0, acc[nt][0], fmaf(bl0, xs[j][nt][0], out[nt][0]));
                out[nt][1] = fmaf(sl1, acc[nt][1], fmaf(bl1, xs[j][nt][1], out[nt][1]));
                out[nt][2] = fmaf(sh0, acc[nt][2], fmaf(bh0, xs[j][nt][0], out[nt][2]));
                out[nt][3] = fmaf(sh1, acc[nt][3], fmaf(bh1, xs[j][nt][1], out[nt][3]));
              }
            }
          }
          // the partial buffer has been read by its reducer
          const int pbi = buffer_of(rg, nth);
          if (!warp_wait(pfree0 + 8 * pbi, (pphase >> pbi & 1) ^ 1, abort_flag)) return;
          pphase ^= 1u << pbi;
          ++nth;
          const uint32_t pa = pb_mine + (uint32_t)pbi * p.pbuf_bytes;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = out[nt][c] * kOut * unscale[nt][c & 1];
            if (ng == 1) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int tok = nt * 8 + 2 * t + h;
                if (tok < seg.rows) sts_rows(pa + (tok * tok_pitch(W) + 2 * g) * 4, v[h], v[2 + h]);
              }
            } else {   // the groups of a token lie in neighbouring columns
              float l = v[0] + v[1], h = v[2] + v[3];
              int tok = nt * 4 + t;
              if (ng == 4) {
                l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
                h += __shfl_xor_sync(0xFFFFFFFFu, h, 1);
                tok = (t & 1) ? seg.rows : nt * 2 + (t >> 1);
              }
              if (tok < seg.rows) sts_rows(pa + (tok * tok_pitch(W) + 2 * g) * 4, l, h);
            }
          }
          __syncwarp();
          if (lane == 0) {   // only here: the stores have consumed what was read from the slot, which the copies may now overwrite
            tc::mbar_arrive(pfull0 + 8 * pbi);
            tc::mbar_arrive(done0 + 8 * slot);
          }
          sb += p.slot_bytes;
          if (++slot == nst) { slot = 0; ++use; sb = smem_base + p.off_slots; }
        }
      }
    }
    more = kGrouped && next_segment(at);
  }
}

// B200Q_PDL=0 turns programmatic dependent launch off (plain stream order).
bool pdl_on();

template <typename T, int BITS, bool RUNS, int SHAPE, int MT, Work W, bool WIDE = false>
int launch(const RowsPlan& pl, cudaStream_t st) {
  auto kern = qmv_rows_kernel<T, BITS, RUNS, SHAPE, MT, W, WIDE>;
  if (pl.smem > 48 * 1024)
    B200Q_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_on() ? 1 : 0;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, pl.prm));
  B200Q_LAUNCH_OK("qmv_rows_kernel");
  return B200Q_OK;
}
template <typename T, int BITS, bool RUNS, int SHAPE>
int launch_shape(const RowsPlan& pl, cudaStream_t st) {
  if constexpr (is_bf16<T>) {
    if (pl.work == Work::Grouped) return launch<T, BITS, RUNS, SHAPE, 1, Work::Grouped>(pl, st);
    if (pl.work == Work::Gated) return launch<T, BITS, RUNS, SHAPE, 1, Work::Gated>(pl, st);
  }
  if constexpr (!RUNS || (SHAPE == 2 && BITS != 2))   // (runs: more than 8 tokens only in groups of 128 and two column tiles)
    if (pl.mt == 2) return launch<T, BITS, RUNS, SHAPE, 2, Work::Plain>(pl, st);
  if constexpr (BITS == 2 && !RUNS)
    if (pl.wide) return launch<T, BITS, RUNS, SHAPE, 1, Work::Plain, true>(pl, st);
  return launch<T, BITS, RUNS, SHAPE, 1, Work::Plain>(pl, st);
}
template <typename T, int BITS>
int launch_width(const RowsPlan& pl, cudaStream_t st) {
  if (pl.runs) {
    if constexpr (BITS != 4 && BITS != 8) {
      switch (pl.shape) {
        case 1: return launch_shape<T, BITS, true, 1>(pl, st);
        default: return launch_shape<T, BITS, true, 2>(pl, st);
      }
    }
  } else {
    if constexpr (BITS == 2 || BITS == 4 || BITS == 8) {
      if constexpr (BITS != 2)
        if (pl.shape == 32) return launch_shape<T, BITS, false, 32>(pl, st);
      return pl.shape == 64 ? launch_shape<T, BITS, false, 64>(pl, st) : launch_shape<T, BITS, false, 128>(pl, st);
    }
  }
  return fail(B200Q_ERR_UNSUPPORTED, "[quantized_matmul] qmv_rows: unsupported problem");
}
template <int BITS>
int launch_rows(const RowsPlan& pl, cudaStream_t st) {
  return pl.f16 ? launch_width<__half, BITS>(pl, st) : launch_width<__nv_bfloat16, BITS>(pl, st);
}

}  // namespace rows
}  // namespace b200q
