// Decode path: y[M, N] = x[M, K] * dequant(W[N, K])^T for a few token rows, and its grouped form (a few rows per
// expert of a mixture-of-experts layer).  Bound by reading W once; what keeps a call from that bound is the
// instructions per weight and everything before the first and after the last byte:
//
//  * A cluster of thread blocks splits K: a block loads only its part of x.  Inside a block every warp owns
//    one "super-slice" of 128 * SPW k for ALL output rows of the cluster: its x values sit in registers as
//    mma.sync B fragments for the whole kernel.
//  * Every warp streams its columns of W, 16 rows at a time, through a ring of its own filled with cp.async:
//    no thread-block barrier, no mbarrier and no polling in the loop.  Scales and biases of the 16 rows
//    ride in the same stage.
//  * Weights are the M side of mma.sync.m16n8k16 (16 rows), tokens the N side (8 or 16).
//  * Two forms of unpacking.
//    Exact (2, 4 and 8 bits): a masked field, read as a 16-bit float, is the subnormal number q * 2^-133 (bf16) or
//    q * 2^-24 (f16), and the tensor cores take subnormals exactly: one AND per two weights, one shift per
//    four.  Scales are applied to fp32 group sums; y = sum_g s_g (sum_k x_k q_k) + sum_g b_g (sum_k x_k).
//    bf16 x is pre-scaled per (warp, token) by a power of two so that nothing leaves fp32's range, and by
//    2^-off for fields that sit `off` bits up in their byte; f16 x is used as it is, with all fields
//    shifted down.
//    Rounded (3, 5, 6 bits, and 2 bits in groups of 32; bf16): a lane holds 32 consecutive fields of a row, and
//    byte permutes bring fields e and e + 16 into the two halves of a register at the same bit offset; one
//    fma.rn.bf16x2 makes s*q+b of the pair, rounded once to bf16 as the register-path kernel does.
//  * Partial sums of the warps go to shared memory, are added in warp order, and the blocks of the cluster
//    exchange their sums through distributed shared memory, added in rank order: deterministic.
//
// Measured (device time, weights from HBM): M=1 28672x8192 6 bits g 32 80 -> 51 us (register-path kernel before),
// 3 bits 64 -> 42; M=3 11008x4096 8 bits f16 33 -> 14 (tensor-core tile before).
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace b200q {
namespace {

constexpr int kStages = 3;          // ring of 16-row stages per warp
constexpr int kMaxWarps = 8;
constexpr size_t kSmemSm = 227 * 1024;

struct StreamParams {
  const void* x;
  const uint8_t* wq;
  const uint16_t* scales;
  const uint16_t* biases;
  void* y;
  int M, N, K;
  long long ld;             // row pitch of y
  int tiles;                // ceil(N / 16) of one matrix
  int n_ss;                 // super-slices of K
  int passes;               // trips over K (1 unless K is longer than the cluster's super-slices)
  int rc;                   // tiles per chunk: partial sums in shared memory
  int mp;                   // token columns of a partial tile: 2, 8 or 16
  int row_bytes, row_groups;
  int csz;                  // bytes per copy of scales (4, 8 or 16)
  int early;                // weights may be read before the previous kernel of the stream has ended
  int entries;              // dense: groups of 16 token rows
  // grouped form: entry e multiplies up to 16 rows with matrix ent[e].expert (device data; nullptr: dense)
  const QmvEntry* ent;
  const int* n_ent;
  int x_is_y;               // grouped: activation rows are the entry's y_row (the second product of a chain), not its x_row
  uint32_t off_part, off_sum, off_sx;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// N bytes, of which the first `n` are read and the rest are zeros.
template <int N>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int n) {
  if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(n) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
  if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// (not .nc: in the grouped form x may be written by the kernel before this one, under programmatic launch)
__device__ __forceinline__ uint4 ldg128(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ldg64(const void* p) {
  uint2 v;
  asm volatile("ld.global.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
template <typename T>
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same with a zero accumulator (no registers to clear).
template <typename T>
__device__ __forceinline__ void mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
template <typename T>
__device__ __forceinline__ float to_f(uint32_t bits16) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float(bits16 << 16);
  else return __half2float(__ushort_as_half((unsigned short)bits16));
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {   // (not .aligned: the lanes of a warp come out of loops of unequal length)
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
  uint32_t r;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r) : "memory");
  return v;
}
__device__ __forceinline__ void add4(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

// ---------------------------------------------------------------------------- shapes
__host__ __device__ constexpr bool exact_form(int bits, int group) { return bits == 4 || bits == 8 || (bits == 2 && group > 32); }
// 128-k slices per warp: two wherever the x fragments leave registers for it (a trip's fixed instructions are
// then shared by twice the weights)
__host__ __device__ constexpr int spw_of(int bits, int mt) { return bits <= 4 || mt == 1 ? 2 : 1; }

template <int BITS, int SPW>
struct Stage {
  static constexpr int kRowB = SPW * 16 * BITS;                // packed bytes per row
  static constexpr int kChunks = kRowB / 16;                   // 16-byte copies per row
  static constexpr int kW = 16 * kRowB;
  // position of 16-byte chunk c of row r: 128- and 64-byte rows are swizzled for ldmatrix, the others lie
  // slice by slice as they come (reads of 3, 5 and 6 words per lane do not conflict)
  static __device__ __forceinline__ uint32_t at(int r, int c) {
    if constexpr (kRowB % 128 == 0 && (BITS == 4 || BITS == 8)) return (c >> 3) * 2048 + r * 128 + (((c & 7) ^ (r & 7)) << 4);
    else if constexpr (BITS == 2) return r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
    else return (c / BITS) * (256 * BITS) + r * (16 * BITS) + (c % BITS) * 16;
  }
};

// Exact form: one packed word -> NP registers; register i holds fields (i, i + NP) of the word.  bf16: in place
// (fields field_off(i) bits up in their byte); f16: shifted down.
template <int BITS, typename T>
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t* P) {
  constexpr bool kPlace = std::is_same<T, __nv_bfloat16>::value;
  constexpr int NP = 16 / BITS;
  constexpr uint32_t kM = ((1u << BITS) - 1u) * 0x00010001u;
  const uint32_t u = w >> 8;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int bit = i * BITS, off = bit & 7;
    const uint32_t v = bit >= 8 ? u : w;
    if constexpr (kPlace) P[i] = v & (kM << off);
    else P[i] = off ? (w >> bit) & kM : v & kM;
  }
}
template <int BITS>
__host__ __device__ constexpr int field_off(int i) { return (i * BITS) & 7; }

// Rounded form: fields e and e + 16 of a 32-field chunk (BITS words).
// Window at byte `by`: bytes by, by+1 in the low half, the same 2*BITS bytes further on in the high half.
template <int BITS>
__device__ __forceinline__ uint32_t window(const uint32_t (&w)[BITS], int by, bool one_byte) {
  const int b2 = by + 2 * BITS, i0 = by >> 2, i1 = b2 >> 2, r0 = by & 3, r1 = b2 & 3;
  if (r0 != 3 && r1 != 3) return __byte_perm(w[i0], w[i1], r0 | (r0 + 1) << 4 | (r1 + 4) << 8 | (r1 + 5) << 12);
  if (one_byte) return __byte_perm(w[i0], w[i1], r0 | r0 << 4 | (r1 + 4) << 8 | (r1 + 4) << 12);
  const uint32_t lo = r0 == 3 ? __funnelshift_r(w[i0], w[(i0 + 1) % BITS], 24) : w[i0];
  const uint32_t hi = r1 == 3 ? __funnelshift_r(w[i1], w[(i1 + 1) % BITS], 24) : w[i1];
  const int q0 = r0 == 3 ? 0 : r0, q1 = r1 == 3 ? 0 : r1;
  return __byte_perm(lo, hi, q0 | (q0 + 1) << 4 | (q1 + 4) << 8 | (q1 + 5) << 12);
}
// s*q+b of the 16 pairs of a chunk, rounded once to bf16.  A field read as bf16 is q * 2^(off - 133), which one
// fma with s * 2^(133 - off) turns into s*q+b exactly rounded; scales whose exponent leaves no room
// for that take the general form (one branch per warp).
__device__ __forceinline__ bool scale_has_room(uint32_t s) { return (s & 0x7FFFu) - 0x80u < (122u << 7) - 0x80u; }   // biased exponent 1..121
template <int BITS>
__device__ __forceinline__ void dequant_chunk(const uint32_t (&w)[BITS], uint32_t s, uint32_t b, bool fast, uint32_t (&P)[16]) {
  constexpr uint32_t kM = ((1u << BITS) - 1u) * 0x00010001u;
  const uint32_t b2 = b * 0x00010001u;
  if (fast) {
    const uint32_t s0 = (s + (133u << 7)) * 0x00010001u;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int by = (BITS * e) >> 3, off = (BITS * e) & 7;
      const bool direct = off + BITS <= 8;
      const uint32_t v = window<BITS>(w, by, direct);
      if (direct) P[e] = fma_bf16x2(v & (kM << off), s0 - (uint32_t)off * 0x00800080u, b2);
      else P[e] = fma_bf16x2((v >> off) & kM, s0, b2);
    }
  } else {
    const float sf = __uint_as_float(s << 16), bf = __uint_as_float(b << 16);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int by = (BITS * e) >> 3, off = (BITS * e) & 7;
      const uint32_t v = (window<BITS>(w, by, off + BITS <= 8) >> off) & kM;
      P[e] = pack_bf16x2(fmaf((float)(v & 0xFFFFu), sf, bf), fmaf((float)(v >> 16), sf, bf));
    }
  }
}

// ---------------------------------------------------------------------------- kernel
// G: group size of the exact form (compile time: it shapes the accumulators), 0 for the rounded form.
template <int BITS, typename T, int MT, int G>
__global__ void __launch_bounds__(kMaxWarps * 32, 2)
qmv_stream_kernel(const StreamParams p, const int group) {
  constexpr bool kExact = G != 0;
  constexpr bool kBf = std::is_same<T, __nv_bfloat16>::value;
  constexpr int SPW = spw_of(BITS, MT);
  using St = Stage<BITS, SPW>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rank = (int)cluster_rank(), cs = (int)cluster_size();
  const int cl = blockIdx.x / cs, ncl = gridDim.x / cs;
  const int gs = kExact ? G : group;
  const int sb = SPW * 256 / gs;                     // bytes of scales per row and stage
  const int sbp = sb < 4 ? 4 : sb;
  const uint32_t stage_bytes = St::kW + 32 * sbp;
  const uint32_t ring = smem_u32(smem) + warp * kStages * stage_bytes;
  const uint32_t part0 = smem_u32(smem) + p.off_part, sum0 = smem_u32(smem) + p.off_sum;
  asm volatile("griddepcontrol.launch_dependents;");
  // Everything may have been written by the previous kernel of the stream, unless the caller has promised
  // that weights are constant: then the first of them are requested before that kernel has ended.
  if (!p.early || p.ent) asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t TT = (uint32_t)(p.ent ? *p.n_ent : p.entries) * p.tiles, per = TT / (uint32_t)ncl, odd = TT - per * ncl;
  const int T0 = (int)(cl * per + min((uint32_t)cl, odd)), T1 = T0 + (int)per + ((uint32_t)cl < odd ? 1 : 0);

  // ---- the warp's copies: 16-byte pieces of 16 rows, lanes along a row.  The address of a copy is a base per
  // tile, the same for the whole block, plus a 32-bit offset of the lane.
  constexpr int kCopies = (16 * St::kChunks + 31) / 32;
  int ss = rank * nw + warp;                         // super-slice of this pass
  uint32_t w_off[kCopies], s_off = 0;
  bool full = true;
  int s_have = 0, w_have = 0;
  const uint16_t* s_ptr = lane < 16 ? p.scales : p.biases;
  auto set_slice = [&]() {                           // ss has changed
    const int k_bytes = ss * SPW * 16 * BITS;
#pragma unroll
    for (int i = 0; i < kCopies; ++i) {
      const int idx = lane + 32 * i, r = idx / St::kChunks, c = idx % St::kChunks;
      w_off[i] = (uint32_t)(r * p.row_bytes + k_bytes + c * 16);
    }
    w_have = p.row_bytes - k_bytes;                  // bytes of a row from here on (past K: zeros)
    const int g0 = ss * SPW * 128 / gs;
    s_off = (uint32_t)((lane & 15) * p.row_groups + (sb == 2 ? (g0 & ~1) : g0));
    s_have = (p.row_groups - g0) * 2;
    full = (ss + 1) * SPW * 128 <= p.K;
  };
  auto issue = [&](int tile, int e, int slot) {
    const long long row0 = (p.ent ? (long long)p.ent[e].expert * p.N : 0) + tile * 16;
    const int rows = p.N - tile * 16;                // rows past N: zeros
    const uint8_t* wb = p.wq + row0 * p.row_bytes;
    const uint32_t dst = ring + slot * stage_bytes;
    const uint32_t d = dst + St::kW + lane * sbp;    // 16 rows of scales, 16 of biases
    if (rows >= 16 && full) {                        // nothing to cut off
      const uint16_t* src = s_ptr + row0 * p.row_groups + s_off;
#pragma unroll
      for (int i = 0; i < kCopies; ++i) {
        const int idx = lane + 32 * i, r = idx / St::kChunks, c = idx % St::kChunks;
        if (kCopies * 32 == 16 * St::kChunks || idx < 16 * St::kChunks) cp_async<16>(dst + St::at(r, c), wb + w_off[i]);
      }
      if (p.csz == 16) {
        cp_async<16>(d, src);
      } else if (p.csz == 8) {
        cp_async<8>(d, src);
        if (sbp == 16) cp_async<8>(d + 8, src + 4);
      } else {
        for (int j = 0; j < sbp; j += 4) cp_async<4>(d + j, src + j / 2);
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < kCopies; ++i) {
      const int idx = lane + 32 * i, r = idx / St::kChunks, c = idx % St::kChunks;
      if (kCopies * 32 == 16 * St::kChunks || idx < 16 * St::kChunks) {
        const bool in = c * 16 < w_have && r < rows;
        cp_async<16>(dst + St::at(r, c), in ? wb + w_off[i] : p.wq, in ? 16 : 0);
      }
    }
    const bool s_in = (lane & 15) < rows;
    const uint16_t* src = s_in ? s_ptr + row0 * p.row_groups + s_off : s_ptr;
    const int have = s_in ? s_have : 0;
    if (p.csz == 16) {
      cp_async<16>(d, have > 0 ? src : s_ptr, have > 0 ? 16 : 0);   // (whole by alignment)
    } else if (p.csz == 8) {
      for (int j = 0; j < sbp; j += 8) cp_async<8>(d + j, j < have ? src + j / 2 : s_ptr, j < have ? 8 : 0);
    } else {
      for (int j = 0; j < sbp; j += 4) cp_async<4>(d + j, j < have ? src + j / 2 : s_ptr, j < have ? 4 : 0);
    }
  };
  int pf = T0, pf_e = T0 / p.tiles, pf_t = T0 - pf_e * p.tiles, pf_slot = 0, pf_end = T1;
  auto issue_next = [&]() {
    if (pf < pf_end) {
      issue(pf_t, pf_e, pf_slot);
      ++pf;
      if (++pf_t == p.tiles) { pf_t = 0; ++pf_e; }
    }
    cp_commit();
    if (++pf_slot == kStages) pf_slot = 0;
  };
  set_slice();
  if (p.passes == 1 && ss < p.n_ss) {
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) issue_next();
  }
  if (p.early && !p.ent) asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- x fragments of the warp's super-slice
  constexpr int NP = kExact ? 16 / BITS : 16;        // registers a word (exact) or a chunk (rounded) unpacks to
  constexpr int KW = 32 / BITS;                      // k per word (exact)
  constexpr int NX = 16 * SPW;                       // x registers per token tile
  constexpr int NG = kExact ? SPW * 128 / (G ? G : 1) : 1;   // groups per stage (exact)
  constexpr int UPS = SPW * BITS;                    // 16-byte units per row and stage (exact)
  constexpr int UG = kExact ? UPS / NG : 1;          // units per group
  uint32_t X[MT][NX];
  uint32_t sx_hi[MT] = {}, sx_lo[MT] = {};           // bf16: group sums of x for groups 2t, 2t+1 (hi / lo parts)
  float unscale[MT][2] = {};                         // bf16: what brings the sums of tokens 2t, 2t+1 back to true units / 2^69
  const uint32_t sx_mem = smem_u32(smem) + p.off_sx + warp * (8 * 16 * 4);   // group sums [group][token]
  auto load_x = [&](int e) {
    const T* x = static_cast<const T*>(p.x);
    const int ntok = p.ent ? p.ent[e].n : min(p.M - e * 16, 16);
    const int k0 = ss * SPW * 128;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const int tok = mt * 8 + g;
      const bool have = tok < ntok;
      const long long xrow = !have ? 0 : (p.ent ? (p.x_is_y ? p.ent[e].y_row[tok] : p.ent[e].x_row[tok]) : e * 16 + tok);
      const T* xp = x + xrow * p.K + k0;
      if constexpr (kExact) {
#pragma unroll
        for (int u = 0; u < UPS; ++u) {              // unit u: 4 * KW consecutive k, of which this lane owns KW
          const int k = u * 4 * KW + t * KW;
          const bool live = have && k0 + k < p.K;
          uint32_t* X0 = &X[mt][u * NP];
          if constexpr (BITS == 8) {
            uint2 v = make_uint2(0, 0);
            if (live) v = ldg64(xp + k);
            X0[0] = __byte_perm(v.x, v.y, 0x5410); X0[1] = __byte_perm(v.x, v.y, 0x7632);
          } else if constexpr (BITS == 4) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (live) v = ldg128(xp + k);
            X0[0] = __byte_perm(v.x, v.z, 0x5410); X0[1] = __byte_perm(v.x, v.z, 0x7632);
            X0[2] = __byte_perm(v.y, v.w, 0x5410); X0[3] = __byte_perm(v.y, v.w, 0x7632);
          } else {
            uint4 a = make_uint4(0, 0, 0, 0), b = a;
            if (live) { a = ldg128(xp + k); b = ldg128(xp + k + 8); }
            X0[0] = __byte_perm(a.x, b.x, 0x5410); X0[1] = __byte_perm(a.x, b.x, 0x7632);
            X0[2] = __byte_perm(a.y, b.y, 0x5410); X0[3] = __byte_perm(a.y, b.y, 0x7632);
            X0[4] = __byte_perm(a.z, b.z, 0x5410); X0[5] = __byte_perm(a.z, b.z, 0x7632);
            X0[6] = __byte_perm(a.w, b.w, 0x5410); X0[7] = __byte_perm(a.w, b.w, 0x7632);
          }
        }
        if constexpr (kBf) {
          // x is multiplied by 2^E so that the token's largest element in the slice lands in [2^64, 2^65), the sums by
          // 2^69 and then 2^(64 - E) on their way out (both exact)
          uint32_t top = 0;                          // largest |x|, per half of a register
#pragma unroll
          for (int i = 0; i < NX; ++i) top = __vmaxu2(top, X[mt][i] & 0x7FFF7FFFu);
          top = max(top & 0xFFFFu, top >> 16);
          top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
          top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
          int E = 191 - (int)(top >> 7);
          E = E < -62 ? -62 : (E > 120 ? 120 : E);
          const uint32_t sc = ((uint32_t)(127 + E) << 7) * 0x00010001u;
#pragma unroll
          for (int i = 0; i < NX; ++i) X[mt][i] = mul_bf16x2(X[mt][i], sc - (uint32_t)field_off<BITS>(i % NP) * 0x00800080u);
          const float un = __uint_as_float((uint32_t)(127 + 64 - E) << 23);
          unscale[mt][0] = __shfl_sync(0xFFFFFFFFu, un, (2 * t) * 4);
          unscale[mt][1] = __shfl_sync(0xFFFFFFFFu, un, (2 * t + 1) * 4);
        }
        // Group sums of x on the tensor cores: the A side holds 2^off for every k, which takes the pre-scaling of
        // its register back.  They pass through shared memory as [group][token].
#pragma unroll
        for (int j = 0; j < NG; ++j) {
          float d[4];
#pragma unroll
          for (int i = 0; i < UG * NP; i += 2) {
            const uint32_t one = kBf ? 0x3F803F80u : 0x3C003C00u;
            const uint32_t c0 = one + (kBf ? (uint32_t)field_off<BITS>(i % NP) * 0x00800080u : 0u);
            const uint32_t c1 = one + (kBf ? (uint32_t)field_off<BITS>((i + 1) % NP) * 0x00800080u : 0u);
            if (i == 0) mma0<T>(d, c0, c0, c1, c1, X[mt][j * UG * NP + i], X[mt][j * UG * NP + i + 1]);
            else mma<T>(d, c0, c0, c1, c1, X[mt][j * UG * NP + i], X[mt][j * UG * NP + i + 1]);
          }
          if (g == 0)
            asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(sx_mem + (j * 16 + mt * 8 + 2 * t) * 4), "f"(d[0]), "f"(d[1]) : "memory");
        }
        __syncwarp();
        if constexpr (kBf) {
          // in units of 2^(E - 133) like the products; lane t keeps groups 2t and 2t+1 of token g, in two bf16 parts
          float e0 = 0.0f, e1 = 0.0f;
          if (2 * t < NG) e0 = __uint_as_float(lds32(sx_mem + (2 * t * 16 + tok) * 4)) * 0x1p-133f;
          if (2 * t + 1 < NG) e1 = __uint_as_float(lds32(sx_mem + ((2 * t + 1) * 16 + tok) * 4)) * 0x1p-133f;
          sx_hi[mt] = pack_bf16x2(e0, e1);
          sx_lo[mt] = pack_bf16x2(e0 - __uint_as_float(sx_hi[mt] << 16), e1 - __uint_as_float(sx_hi[mt] & 0xFFFF0000u));
          __syncwarp();   // (a later entry writes the sums again)
        }
      } else {
#pragma unroll
        for (int sl = 0; sl < SPW; ++sl) {           // 32 consecutive k per lane and slice; pairs (k, k + 16)
          const int k = sl * 128 + t * 32;
          const bool live = have && k0 + k < p.K;
          uint4 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = live ? ldg128(xp + k + 8 * i) : make_uint4(0, 0, 0, 0);
          const uint32_t* lo = reinterpret_cast<const uint32_t*>(&v[0]);
          const uint32_t* hi = reinterpret_cast<const uint32_t*>(&v[2]);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            X[mt][sl * 16 + 2 * i] = __byte_perm(lo[i], hi[i], 0x5410);
            X[mt][sl * 16 + 2 * i + 1] = __byte_perm(lo[i], hi[i], 0x7632);
          }
        }
      }
    }
  };

  // ldmatrix roles of this lane (exact): matrix m = lane / 8 covers rows (m & 1) * 8 .. + 7 of unit (m >> 1)
  const int lm_row = (lane & 7) + ((lane >> 3) & 1) * 8, lm_hi = lane >> 4;

  // ---- one 16-row tile: out[mt][0..3] = (row g, tokens 2t, 2t+1), (row g + 8, the same)
  auto tile_sums = [&](uint32_t base, float (&out)[MT][4]) {
    const uint32_t sa = base + St::kW + g * sbp;     // scales of row g; row g + 8: 8 * sbp on; biases: 16 * sbp on
    const uint32_t odd_value = SPW == 1 && sb == 2 ? (uint32_t)(ss & 1) * 2 : 0u;   // one value per stage: which half of the word
    if constexpr (kExact) {
      uint32_t sl_w[(NG + 1) / 2], sh_w[(NG + 1) / 2];   // scales of the stage's groups: row g, row g + 8
      if constexpr (NG == 8) {
        const uint4 a = lds128(sa), b = lds128(sa + 8 * sbp);
        sl_w[0] = a.x; sl_w[1] = a.y; sl_w[2] = a.z; sl_w[3] = a.w; sh_w[0] = b.x; sh_w[1] = b.y; sh_w[2] = b.z; sh_w[3] = b.w;
      } else if constexpr (NG == 4) {
        const uint2 a = lds64(sa), b = lds64(sa + 8 * sbp);
        sl_w[0] = a.x; sl_w[1] = a.y; sh_w[0] = b.x; sh_w[1] = b.y;
      } else {
        sl_w[0] = lds32(sa); sh_w[0] = lds32(sa + 8 * sbp);
        if (NG == 1 && odd_value) { sl_w[0] >>= 16; sh_w[0] >>= 16; }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 4; ++c) out[mt][c] = 0.0f;
      // Groups go in pairs: with MT token tiles and SPLIT partial accumulators that makes four independent chains
      // of mma.sync, whose results come back after many cycles.
      constexpr int GP = NG < 2 ? 1 : 2;
      constexpr int STEPS = UG * NP / 2;             // mma k steps per group
      constexpr int SPLIT = 4 / (MT * GP) < 1 ? 1 : (4 / (MT * GP) < STEPS ? 4 / (MT * GP) : STEPS);
#pragma unroll
      for (int gq = 0; gq < NG; gq += GP) {
        uint32_t wl[GP * UG], wh[GP * UG];
        if constexpr (GP * UG >= 2) {
#pragma unroll
          for (int i = 0; i < GP * UG; i += 2) ldmatrix_x4(base + St::at(lm_row, gq * UG + i + lm_hi), wl[i], wh[i], wl[i + 1], wh[i + 1]);
        } else {
          wl[0] = lds32(base + St::at(g, gq * UG) + 4 * t); wh[0] = lds32(base + St::at(g + 8, gq * UG) + 4 * t);
        }
        float acc[GP][MT][SPLIT][4];
#pragma unroll
        for (int iu = 0; iu < UG; ++iu)
#pragma unroll
          for (int u = 0; u < GP; ++u) {
            uint32_t Pl[NP], Ph[NP];
            unpack_word<BITS, T>(wl[u * UG + iu], Pl);
            unpack_word<BITS, T>(wh[u * UG + iu], Ph);
#pragma unroll
            for (int st = 0; st < NP / 2; ++st)
#pragma unroll
              for (int mt = 0; mt < MT; ++mt) {
                const int step = iu * (NP / 2) + st, i = ((gq + u) * UG + iu) * NP + 2 * st;
                if (step < SPLIT) mma0<T>(acc[u][mt][step], Pl[2 * st], Ph[2 * st], Pl[2 * st + 1], Ph[2 * st + 1], X[mt][i], X[mt][i + 1]);
                else mma<T>(acc[u][mt][step % SPLIT], Pl[2 * st], Ph[2 * st], Pl[2 * st + 1], Ph[2 * st + 1], X[mt][i], X[mt][i + 1]);
              }
          }
#pragma unroll
        for (int u = 0; u < GP; ++u) {
          const int j = gq + u;
          const float s_l = to_f<T>(j & 1 ? sl_w[j / 2] >> 16 : sl_w[j / 2] & 0xFFFFu), s_h = to_f<T>(j & 1 ? sh_w[j / 2] >> 16 : sh_w[j / 2] & 0xFFFFu);
          float b_l = 0.0f, b_h = 0.0f;
          if constexpr (!kBf) {
            const uint32_t so = NG == 1 ? odd_value : 2 * j;
            b_l = to_f<T>(lds16(sa + 16 * sbp + so)); b_h = to_f<T>(lds16(sa + 24 * sbp + so));
          }
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
            for (int q = 1; q < SPLIT; ++q)
#pragma unroll
              for (int c = 0; c < 4; ++c) acc[u][mt][0][c] += acc[u][mt][q][c];
            if constexpr (kBf) {
              out[mt][0] = fmaf(s_l, acc[u][mt][0][0], out[mt][0]);
              out[mt][1] = fmaf(s_l, acc[u][mt][0][1], out[mt][1]);
              out[mt][2] = fmaf(s_h, acc[u][mt][0][2], out[mt][2]);
              out[mt][3] = fmaf(s_h, acc[u][mt][0][3], out[mt][3]);
            } else {
              const uint2 sx = lds64(sx_mem + (j * 16 + mt * 8 + 2 * t) * 4);
              const float x0 = __uint_as_float(sx.x), x1 = __uint_as_float(sx.y);
              const float sl = s_l * 0x1p24f, sh = s_h * 0x1p24f;
              out[mt][0] = fmaf(sl, acc[u][mt][0][0], fmaf(b_l, x0, out[mt][0]));
              out[mt][1] = fmaf(sl, acc[u][mt][0][1], fmaf(b_l, x1, out[mt][1]));
              out[mt][2] = fmaf(sh, acc[u][mt][0][2], fmaf(b_h, x0, out[mt][2]));
              out[mt][3] = fmaf(sh, acc[u][mt][0][3], fmaf(b_h, x1, out[mt][3]));
            }
          }
        }
      }
      if constexpr (kBf) {
        // biases: b_g * sum_k x_k through one MMA, k slots 2t, 2t+1 (hi part of the sum) / + 8 (lo part)
        uint32_t bl = 0, bh = 0;
        const uint32_t ba = sa + 16 * sbp;
        if constexpr (NG >= 2) {
          if (2 * t < NG) { bl = lds32(ba + 4 * t); bh = lds32(ba + 8 * sbp + 4 * t); }
        } else if (t == 0) {
          bl = lds16(ba + odd_value); bh = lds16(ba + 8 * sbp + odd_value);
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma<T>(out[mt], bl, bh, bl, bh, sx_hi[mt], sx_lo[mt]);
#pragma unroll
          for (int c = 0; c < 4; ++c) out[mt][c] = out[mt][c] * 0x1p69f * unscale[mt][c & 1];
        }
      }
    } else {
      const int gsh = group == 32 ? 0 : (group == 64 ? 1 : 2);
      constexpr int SPLIT = MT == 2 ? 2 : 4;
      float acc[MT][SPLIT][4];
#pragma unroll
      for (int sl = 0; sl < SPW; ++sl) {
        const uint32_t so = sb == 2 ? odd_value : 2 * ((4 * sl + t) >> gsh);
        uint32_t P[2][16], w[2][BITS], s[2], b[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = g + 8 * h;
          const uint32_t at = base + sl * (256 * BITS) + r * (16 * BITS) + t * (4 * BITS);
          if constexpr (BITS == 2) {
            const uint2 v = lds64(base + St::at(r, 2 * sl + (t >> 1)) + 8 * (t & 1));
            w[h][0] = v.x; w[h][1] = v.y;
          } else if constexpr (BITS == 6) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const uint2 v = lds64(at + 8 * i);
              w[h][2 * i] = v.x; w[h][2 * i + 1] = v.y;
            }
          } else {
#pragma unroll
            for (int i = 0; i < BITS; ++i) w[h][i] = lds32(at + 4 * i);
          }
          s[h] = lds16(sa + h * 8 * sbp + so);
          b[h] = lds16(sa + (16 + h * 8) * sbp + so);
        }
        const bool fast = __all_sync(0xFFFFFFFFu, scale_has_room(s[0]) && scale_has_room(s[1]));
        dequant_chunk<BITS>(w[0], s[0], b[0], fast, P[0]);
        dequant_chunk<BITS>(w[1], s[1], b[1], fast, P[1]);
#pragma unroll
        for (int st = 0; st < 8; ++st)
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const int i = sl * 16 + 2 * st;
            if (sl == 0 && st < SPLIT) mma0<T>(acc[mt][st], P[0][2 * st], P[1][2 * st], P[0][2 * st + 1], P[1][2 * st + 1], X[mt][i], X[mt][i + 1]);
            else mma<T>(acc[mt][st % SPLIT], P[0][2 * st], P[1][2 * st], P[0][2 * st + 1], P[1][2 * st + 1], X[mt][i], X[mt][i + 1]);
          }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float v = acc[mt][0][c];
#pragma unroll
          for (int q = 1; q < SPLIT; ++q) v += acc[mt][q][c];
          out[mt][c] = v;
        }
    }
  };

  // ---- chunks of up to rc tiles of one entry
  const int na = min(max(p.n_ss - rank * nw, 0), nw);   // warps of this block with a slice in the first pass
  int e = T0 / p.tiles, lt = T0 - e * p.tiles, e_x = -1, slot = 0, buf = 0;
  for (int tt = T0; tt < T1;) {
    const int n = min(min(p.rc, T1 - tt), p.tiles - lt);
    for (int ps = 0; ps < p.passes; ++ps) {
      ss = ps * cs * nw + rank * nw + warp;
      if (ss >= p.n_ss) continue;
      if (p.passes > 1) {
        pf = tt; pf_end = tt + n; pf_e = e; pf_t = lt;
        set_slice();
        slot = pf_slot;
        __syncwarp();   // the last tile of the pass before has been read by all lanes
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i) issue_next();
      }
      if (p.passes > 1 || e != e_x) { load_x(e); e_x = e; }
      for (int i = 0; i < n; ++i) {
        cp_wait<kStages - 2>();
        __syncwarp();   // the stage is visible to the warp, and the one before it has been read by all lanes
        issue_next();
        float out[MT][4];
        tile_sums(ring + slot * stage_bytes, out);
        if (++slot == kStages) slot = 0;
        if (p.mp == 2) {
          const uint32_t a = part0 + ((warp * p.rc + i) * 32 + g * 2) * 4;
          if (t == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float2 v = make_float2(out[0][2 * h], out[0][2 * h + 1]);
              if (ps > 0) { const uint2 o = lds64(a + h * 64); v.x += __uint_as_float(o.x); v.y += __uint_as_float(o.y); }
              asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a + h * 64), "f"(v.x), "f"(v.y) : "memory");
            }
          }
        } else {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const uint32_t a = part0 + (((warp * p.rc + i) * MT + mt) * 128 + g * 8 + 2 * t) * 4;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float2 v = make_float2(out[mt][2 * h], out[mt][2 * h + 1]);
              if (ps > 0) { const uint2 o = lds64(a + h * 256); v.x += __uint_as_float(o.x); v.y += __uint_as_float(o.y); }
              asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a + h * 256), "f"(v.x), "f"(v.y) : "memory");
            }
          }
        }
      }
    }
    __syncthreads();
    // ---- add the warps' partial tiles in order, then the blocks', and store: four sums per thread and turn
    const int ntok = p.ent ? p.ent[e].n : min(p.M - e * 16, 16);
    const int fsh = p.mp == 2 ? 3 : (MT == 2 ? 6 : 5);   // log2 of the float4 per tile
    const int nf = n << fsh;
    const uint32_t pitch = (uint32_t)p.rc << (fsh + 4);
    auto local_sum = [&](int f) {
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      for (int w = 0; w < na; ++w) {
        const uint4 v = lds128(part0 + w * pitch + f * 16);
        add4(s, make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)));
      }
      return s;
    };
    auto put = [&](int tok, int col, float v) {
      if (tok < ntok && col < p.N) {
        const long long yr = p.ent ? p.ent[e].y_row[tok] : e * 16 + tok;
        static_cast<T*>(p.y)[yr * p.ld + col] = Elem<T>::from_float(v);
      }
    };
    auto store = [&](int f, const float4& v) {
      const int c0 = (lt + (f >> fsh)) * 16;
      if (p.mp == 2) {                                   // [16 rows][2 tokens]
        const int col = c0 + (f & 7) * 2;
        put(0, col, v.x); put(1, col, v.y); put(0, col + 1, v.z); put(1, col + 1, v.w);
      } else {                                           // [token tile][16 rows][8 tokens]
        const int r = f & ((1 << fsh) - 1), col = c0 + ((r >> 1) & 15), tok = (r >> 5) * 8 + (r & 1) * 4;
        put(tok, col, v.x); put(tok + 1, col, v.y); put(tok + 2, col, v.z); put(tok + 3, col, v.w);
      }
    };
    if (cs == 1) {
      for (int f = tid; f < nf; f += blockDim.x) store(f, local_sum(f));
      __syncthreads();   // the partial tiles may be written again
    } else {
      const uint32_t sum = sum0 + buf * ((uint32_t)p.rc << (fsh + 4));
      for (int f = tid; f < nf; f += blockDim.x) {
        const float4 v = local_sum(f);
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(sum + f * 16), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
      }
      cluster_sync();    // (its release and acquire also order the next chunk's partial tiles behind the reads above)
      const int f1 = (rank + 1) * nf / cs;
      for (int f = rank * nf / cs + tid; f < f1; f += blockDim.x) {
        float4 v = ld_cluster(sum + f * 16, 0);
        for (int r = 1; r < cs; ++r) add4(v, ld_cluster(sum + f * 16, r));
        store(f, v);
      }
      buf ^= 1;          // the other blocks read this one until they arrive at the next chunk's barrier
    }
    tt += n;
    lt += n;
    if (lt == p.tiles) { lt = 0; ++e; }
  }
  if (cs > 1) cluster_sync();   // no block leaves while its sums may still be read
}

// ---------------------------------------------------------------------------- host side
struct StreamPlan {
  bool ok;
  int nw, cs, grid, mt;
  size_t smem;
  StreamParams prm;
};

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

bool pdl_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("B200Q_PDL");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

using StreamKernel = void (*)(const StreamParams, const int);

template <int BITS, typename T>
StreamKernel pick_group(int group, int mt) {
  auto mt_of = [&](auto gtag) -> StreamKernel {
    constexpr int G = decltype(gtag)::value;
    return mt == 2 ? (StreamKernel)qmv_stream_kernel<BITS, T, 2, G> : (StreamKernel)qmv_stream_kernel<BITS, T, 1, G>;
  };
  if constexpr (exact_form(BITS, 64)) {
    if (group == 64) return mt_of(std::integral_constant<int, 64>{});
    if (group == 128) return mt_of(std::integral_constant<int, 128>{});
    if constexpr (exact_form(BITS, 32)) return mt_of(std::integral_constant<int, 32>{});
  }
  if constexpr (std::is_same<T, __nv_bfloat16>::value && BITS != 4 && BITS != 8) return mt_of(std::integral_constant<int, 0>{});
  else return nullptr;
}
StreamKernel pick_kernel(int dtype, int bits, int group, int mt) {
  StreamKernel k = nullptr;
  if (dtype == B200Q_BF16) {
    B200Q_DISPATCH_BITS(bits, BITS, { k = pick_group<BITS, __nv_bfloat16>(group, mt); });
  } else if (dtype == B200Q_F16 && exact_form(bits, group)) {
    if (bits == 2) k = pick_group<2, __half>(group, mt);
    if (bits == 4) k = pick_group<4, __half>(group, mt);
    if (bits == 8) k = pick_group<8, __half>(group, mt);
  }
  return k;
}

// Clusters that the device holds at once (the GPCs' leftover slots are lost to large clusters), remembered per
// thread: the query costs more than a launch.
int resident_clusters(StreamKernel k, int cs, int nw, size_t smem) {
  struct Known { StreamKernel k; int dev, cs, nw; size_t smem; int n; };
  constexpr int kMost = 64;
  static thread_local Known known[kMost];
  static thread_local int count = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  for (int i = 0; i < (count < kMost ? count : kMost); ++i) {
    const Known& q = known[i];
    if (q.k == k && q.dev == dev && q.cs == cs && q.nw == nw && q.smem == smem) return q.n;
  }
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemSm));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(nw * 32);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = sm_count() / cs > 0 ? sm_count() / cs : 1;
  }
  known[count % kMost] = Known{k, dev, cs, nw, smem, n};
  if (++count == 2 * kMost) count = kMost;
  return n;
}

// How K is cut (warps per block, blocks per cluster) and how many blocks share an SM: the combination with
// the least estimated time.  The constants are fitted to sweeps of all combinations over 26 shapes (1024 x 4096 to
// 28672 x 8192, every width, 1 to 16 rows): a trip over a tile takes `work` cycles times the warps per scheduler
// and one more; clusters of four and eight leave 4 and 11 % of the SMs' slots empty.
StreamPlan stream_plan(int dtype, int64_t M, int64_t N, int64_t K, int group, int bits, int64_t entries, int rows_max) {
  StreamPlan best{};
  const int mt = rows_max > 8 ? 2 : 1, spw = spw_of(bits, mt);
  if (!pick_kernel(dtype, bits, group, mt)) return best;
  const int mp = rows_max <= 2 ? 2 : 8 * mt;
  const int n_ss = (int)((K + 128 * spw - 1) / (128 * spw));
  const int tiles = (int)((N + 15) / 16);
  const int sb = spw * 256 / group, sbp = sb < 4 ? 4 : sb;
  const size_t stage = (size_t)256 * spw * bits + 32 * sbp;
  const double work = (exact_form(bits, group) ? 270 : 390) * spw * (mt == 2 ? 1.5 : 1.0);
  double best_t = 1e300;
  const int sms = sm_count();
  for (int cs = 1; cs <= 8; cs *= 2) {
    for (int nw = 4; nw <= kMaxWarps; ++nw) {
      const int passes = (n_ss + cs * nw - 1) / (cs * nw);
      if (passes == 1 && cs > 1 && (n_ss + nw - 1) / nw <= cs / 2) continue;   // half of the blocks would be idle
      for (int occ = 16 / nw; occ >= 1; --occ) {
        const size_t budget = (kSmemSm + 1024) / occ - 1024;
        const size_t fixed = nw * (kStages * stage + 512) + 256;
        const size_t per_tile = (size_t)nw * 16 * mp * 4 + (cs > 1 ? 2 * 16 * mp * 4 : 0);
        if (budget < fixed + per_tile) continue;
        const int ncl = (int)(sms * occ / cs * (cs == 8 ? 0.89 : (cs == 4 ? 0.96 : 1.0)));
        if (ncl < 1) continue;
        const int64_t per_cl = (entries * tiles + ncl - 1) / ncl;
        int64_t rc = (int64_t)((budget - fixed) / per_tile);
        if (rc > per_cl) rc = per_cl;
        if (rc > 64) rc = 64;
        const double chunks = (double)((per_cl + rc - 1) / rc);
        const double trip = (occ * nw / 4.0 + 0.9) * work;
        const double time = passes * per_cl * trip + chunks * (600 + 250.0 * rc * mp / 16) +
                            (cs > 1 ? 800 + 300 * cs : 0) * chunks + (passes - 1) * chunks * 900 + 200 * occ;
        if (time < best_t) {
          best_t = time;
          best.ok = true;
          best.nw = nw; best.cs = cs; best.mt = mt; best.grid = sms * occ / cs * cs;
          StreamParams& p = best.prm;
          p.n_ss = n_ss; p.passes = passes; p.rc = (int)rc; p.mp = mp; p.tiles = tiles;
          p.off_part = (uint32_t)((nw * kStages * stage + 127) / 128 * 128);
          p.off_sum = p.off_part + (uint32_t)(nw * rc * 16 * mp * 4);
          p.off_sx = p.off_sum + (cs > 1 ? (uint32_t)(2 * rc * 16 * mp * 4) : 0);
          best.smem = p.off_sx + nw * 512;
        }
      }
    }
  }
  StreamParams& p = best.prm;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.row_bytes = (int)(K * bits / 8);
  p.row_groups = (int)(K / group);
  p.csz = sbp > 16 ? 16 : sbp;
  while (p.csz > 4 && (2 * p.row_groups) % p.csz != 0) p.csz /= 2;
  return best;
}

bool shape_ok(int dtype, int64_t N, int64_t K, int group, int bits, const void* x, const void* wq, const void* s, const void* b) {
  if (dtype != B200Q_BF16 && dtype != B200Q_F16) return false;
  if (N < 1 || K < 128 || K % 128 != 0 || (K / group) % 2 != 0 || N > (1ll << 28) || K > (1ll << 24)) return false;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(b)) & 15) != 0) return false;
  return pick_kernel(dtype, bits, group, 1) != nullptr;
}

int launch_stream(StreamPlan& pl, int dtype, int bits, int group, cudaStream_t st) {
  StreamKernel k = pick_kernel(dtype, bits, group, pl.mt);
  const int res = resident_clusters(k, pl.cs, pl.nw, pl.smem) * pl.cs;
  if (pl.grid > res) pl.grid = res;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(pl.nw * 32);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = pl.cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, k, (const StreamParams)pl.prm, group));
  B200Q_LAUNCH_OK("qmv_stream_kernel");
  return B200Q_OK;
}

}  // namespace

bool qmv_stream_supported(const QmmArgs& a) {
  if (!a.transpose || a.w_batched || a.batch != 1 || a.peers.n > 0 || a.M < 1 || a.M > 32) return false;
  return shape_ok(a.dtype, a.N, a.K, a.group, a.bits, a.x, a.wq, a.scales, a.biases);
}

int qmv_stream(const QmmArgs& a, cudaStream_t st) {
  const int entries = (int)((a.M + 15) / 16);
  StreamPlan pl = stream_plan(a.dtype, a.M, a.N, a.K, a.group, a.bits, entries, (int)(a.M < 16 ? a.M : 16));
  if (!pl.ok) return fail(B200Q_ERR_UNSUPPORTED, "[quantized_matmul] qmv_stream: unsupported problem");
  StreamParams& p = pl.prm;
  p.x = a.x;
  p.wq = reinterpret_cast<const uint8_t*>(a.wq);
  p.scales = static_cast<const uint16_t*>(a.scales);
  p.biases = static_cast<const uint16_t*>(a.biases);
  p.y = a.y;
  p.ld = a.N;
  p.early = weights_constant() ? 1 : 0;
  p.entries = entries;
  return launch_stream(pl, a.dtype, a.bits, a.group, st);
}

}  // namespace b200q
