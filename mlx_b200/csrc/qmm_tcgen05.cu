// Products with many token rows on the 5th-generation tensor cores:
//   y[M, N] = x[M, K] * dequant(W[N, K])^T      (transpose)
//   y[M, N] = x[M, K] * dequant(W[K, N])        (no transpose: the gradient of the first with respect to x)
//
// Replaces cu::qmm_sm80_kernel / qmm_naive_kernel of the reference
// (mlx/backend/cuda/device/qmm_sm80.cuh:70-356, quantized/qmm/qmm.cu:20-185), which run
// Ampere-style mma.sync code on this GPU.
//
// Formulation (swap-AB): D[256 output columns, NT tokens], so that the operand that has to be
// dequantised (W) is the A operand and is re-used by up to 256 tokens per instruction, and the operand
// that streams unchanged (x) is B.  A tile belongs to a PAIR of thread blocks (a cluster of two,
// tcgen05 cta_group::2): each block unpacks and accumulates 128 of the 256 output columns and holds half
// of the tokens.  At 256 tokens a stage of 128 k takes 1024 cycles on the tensor pipe; one block alone
// would have to fetch 64 KB of x in that time, the SM's whole L2 bandwidth (64 bytes per clock), and was
// bound by it.  A pair fetches every x tile once: 32 bytes per clock and SM.
//
//   warp 0: TMA  --two x sub-tiles [NT/2 tokens x 64 k], 128B-swizzled K-major-->  smem ring B
//   warp 1: tcgen05.mma.cta_group::2.kind::f16 (leader block only; one elected thread: under
//        elect.sync an MMA issues at its own rate, N/2 cycles, under "lane == 0" it cost 85)
//   warp 2: TMA  --packed W tile [128 rows x 16*bits bytes]-->  smem ring P (swizzled where the row is
//        32, 64 or 128 bytes: the unpack threads' 16-byte reads are then free of bank conflicts)
//   warp 3: cp.async --scales and biases of the same tile--> smem ring S.  A value of each is needed per row
//        and group, from as many cache lines as rows: one warp fetches every value once per block
//        where sixteen unpack warps fetched it four times.
//   warps 4-19: unpack W into the A operand, in sets that take A slots in turn: a warp's trip through a
//        slot is a chain of dependent latencies, and four sets (two for SplitT) give each trip as many
//        slot times
//   warps 20-27: tcgen05.ld the accumulator, round, store y (scattered through a row table in grouped
//        mode); with at most 128 tokens per tile there are two accumulators and the store of one tile
//        runs under the next
//
// How W becomes the A operand (Form):
//   Round   bf16, transpose: s*q+b rounded once to bf16 (one fma.rn.bf16x2 per pair), in tensor memory
//   Split   f16, transpose: s*q+b in fp32, split into two f16 numbers hi + lo, two MMAs per k step: the
//           product keeps the weights' fp32 value (split32 says how closely), as the CUDA-core kernel did
//   SplitT  no transpose, bf16 and f16: W is packed along the output columns, so A is written to shared
//           memory M-major (hi and lo)
// In two parts a weight beyond 65504 (f16), an infinite one and an infinite x give NaN where the weight itself gives a number
// or an infinity.  Where the epilogue warps of a block of the split forms have stored a result that is not finite, they go over
// the block's tiles once more at the end, when nobody waits for them any more, and compute such elements in fp32 from the weights
// themselves (repair).
//
// Tiles are dealt to the pairs in whole waves; the K stages of the tiles that are left over are laid end to end and cut
// into equal ranges, one per pair, so that the last wave is as short as its work (or, with few tiles, all SMs have
// work).  A tile that is cut leaves fp32 partial sums in the workspace and the last pair to arrive adds them in order;
// no block ever waits for another pair.  With the last wave uneven instead, 512 tokens through [28672, 8192] took four
// waves for 3.03 waves' work.
//
// Grouped mode (gather_qmm): a device-side table lists (expert, first row, valid rows) for
// every slice of up to NT rows of the expert-sorted activations; the weight tensor map spans the
// stacked experts [E*N, K*bits/8].
//
// The token width of a tile is rounded up to 32, not to NT: ragged token counts and experts with few rows
// pay for what they have.
//
// Every mbarrier wait is bounded.  When a wait expires the role sets the block's abort
// flag and the device status word, all roles leave their loops, TMEM is released and
// the kernel ends normally (its results are then invalid and the host reports it).
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

namespace b200q {
namespace {

using namespace tc;

enum class Form { Round, Split, SplitT };

constexpr int kTileRows = 128;    // output columns per block and tile (MMA M = 256 over the pair)
constexpr int kStageK = 128;      // k per pipeline stage of x, W, scales
constexpr int kMaxStagesB = 6;
constexpr int kMaxStagesP = 8;
constexpr int kMaxSlotsA = 4;
constexpr int kMaxSlotsS = 8;     // chunks of scales and biases
constexpr int kDoneRing = 16;     // one commit per A slot; longer than any distance a waiter can be behind
constexpr int kTmemCols = 512;    // [0, 256) accumulators, [256, 512) A ring (4 slots of 64 columns)
constexpr int kAccCols = 256;
constexpr int kUnpackWarps = 16;
constexpr int kEpilogueWarps = 8;
constexpr int kFirstUnpack = 4, kFirstEpilogue = kFirstUnpack + kUnpackWarps;
constexpr int kThreads = 32 * (kFirstEpilogue + kEpilogueWarps);   // 896
constexpr size_t kSmemMax = 227 * 1024;

template <int BITS, Form F>
struct Shape {
  static constexpr bool kT = F == Form::SplitT;
  static constexpr int kSub = F == Form::Round ? 1 : 2;        // A slots per stage (64 k each when split)
  static constexpr int kSlotsA = kT ? 3 : 4;
  static constexpr int kSets = kT ? 2 : 4;                     // sets of unpack warps, on A slots in turn
  // Packed stages: four sets hold one each while they unpack; with no more than that every set would wait for a
  // whole TMA latency after each slot.
  // 8 bits: 16 KB a stage.  Eight where the tile's x leaves room (up to 128 tokens), else four; both whole turns of the
  // sets.  Against single blocks with two packed stages and whole tiles, which bf16 ran on before (us): 64 rows through
  // [4096, 4096] 40 -> 20, 512 42 -> 23, 4096 141 -> 105; 35 through [1280, 22784] 196 -> 27; against CUDA cores: f16, 512
  // rows through [4096, 3584] 1090 -> 35, transpose=False, 300 through [4096, 4096] 1415 -> 56 (errors against 64 bits equal
  // to three digits: f16 2.08e-4, bf16 1.66e-3).
  static constexpr int kStagesP = kT ? (BITS == 8 ? 2 : 3) : (BITS <= 4 || BITS == 8 ? 8 : 6);
  static constexpr int kFewStagesP = BITS == 8 && !kT ? 4 : kStagesP;
  static constexpr int kPRowBytes = 16 * BITS;                 // 128 fields
  static constexpr int kPStageBytes = kTileRows * kPRowBytes;
  static constexpr int kSmemA = kT ? kSlotsA * 32768 : 0;      // 64 k x 128 columns, hi and lo
  // Tokens (x 32 columns, 64 bytes) of the epilogue's staging tile per warp.  SplitT, whose A ring takes 96 KB: half as many, so that
  // 256 tokens of x have two stages at 5, 6 and 8 bits too.
  static constexpr int kOutTok = kT ? 32 : 64;
  static constexpr int kStageOut = kOutTok * 64;
  static constexpr int kPArrivals = kSub * kUnpackWarps / kSets;   // of a packed stage: every set that takes one of its slots
};

// Shared-memory matrix descriptor of a 128-byte-swizzled operand tile, descriptor version 1 (sm_100).
// K-major (x): rows of 64 k, 8-row groups 1024 bytes apart (sbo); `addr` may point 32*j bytes into the
// first row to select the j-th 16-element K slice.  M-major (A of SplitT): rows of 64 columns, one per k,
// 8-k groups `sbo` apart, 64-column blocks `lbo` apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}
// Instruction descriptor: D f32, A and B of the same 16-bit type, B K-major, M = 256, N = n.
template <typename T, Form F>
__device__ __forceinline__ uint32_t make_idesc(int n) {
  constexpr uint32_t fmt = sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (F == Form::SplitT ? 1u << 15 : 0u) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(2 * kTileRows >> 4) << 24);
}

// One entry per group of up to NT consecutive rows of the (expert-sorted) activation matrix.
struct MTile {
  int expert;     // weight matrix the rows multiply
  int row0;       // first row in the activation matrix
  int rows;       // valid rows: what follows in the TMA box belongs to another expert
  int pad;
};

struct TcMaps {
  CUtensorMap x[4];   // boxes of 128, 64, 32 and 16 tokens x 64 k
  CUtensorMap w;
};

struct TcParams {
  // grouped (gather_qmm) mode: device-side tile table, else nullptr
  const MTile* mtiles;
  const int* n_mtiles;      // device scalar: entries of `mtiles`
  const int* dst_row;       // output row of every activation row
  const unsigned short* scales;
  const unsigned short* biases;
  const void* x;            // split forms, for `repair`: x and the packed weights
  const uint32_t* wq;
  // output buffers (one, or one per GPU of an N-sharded layer), row pitch and first column
  void* y_out[kMaxPeers];
  int n_out;
  long long ld, col0;
  int y_align;       // bytes that the start of every row of every output is a multiple of: 16, 8 or 2
  PeerSignal sig;    // completion signal towards the ranks that receive y (n == 0: none)
  uint32_t* status;
  int M, N, K;
  int NT;            // most tokens per tile (multiple of 32, <= 256)
  int nsb;           // x stages in shared memory (1 .. kMaxStagesB)
  int nsp;           // packed stages, 8 bits only: 8 or 4
  int n_tiles, m_tiles;
  int full;          // tiles in whole waves (all of them in grouped mode)
  int rem, cut;      // tiles left over, and the number of pairs their stages are cut for
  float* partial;    // [cut range, tile by tile][block of the pair][NT tokens][128 columns]
  uint32_t* counters;   // [tile left over][block of the pair]
  int g4;            // groups per 128 fields of a row: 4, 2, 1
  int row_groups;    // groups per packed row
  int s_slots;       // chunks of scales in their ring (a power of two)
  int spc, cb;       // stages per chunk of scales, bytes per row of a chunk (4, 8 or 16)
  int narrow;        // scales or biases are not aligned to cb: 2-byte loads
  long long n_scales;   // elements of `scales`
};

struct __align__(8) Barriers {
  uint64_t full_p[kMaxStagesP], empty_p[kMaxStagesP];
  uint64_t full_s[kMaxSlotsS], empty_s[kMaxSlotsS];
  // Of the pair's leader: x tiles of both blocks have landed; both blocks' unpack warps have filled an A slot
  uint64_t full_b[kMaxStagesB];
  uint64_t full_a[kMaxSlotsA];
  // One commit per A slot, to both blocks: slot use `ia` (counted across tiles) arrives on
  // done[ia % kDoneRing] when its MMAs have completed.  Whatever it read (A slot, with the last slot
  // of a stage the x stage too) is free again from then on.
  uint64_t done[kDoneRing];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag, last;
  int help;        // the pair's last unit is a tile that this block is the last to add up: all warps that can take part
  int odd;         // split forms: a result was not finite
  uint32_t ended;  // pieces of cut tiles (by their number among this pair's) that this block has summed
  int landed[2];   // of a tile (even, odd): its accumulator is complete, as the epilogue warp that waits for it found
};

// ------------------------------------------------------------------------------------ unpacking
__device__ __forceinline__ uint32_t lds_u16(uint32_t at) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t at) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ void lds_v2(uint32_t at, uint32_t& a, uint32_t& b) {
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(at));
}
__device__ __forceinline__ void lds_v4(uint32_t at, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at));
}
// The 32 fields of unit u (0..3) of row r of a packed tile: BITS words.
template <int BITS>
__device__ __forceinline__ void load_fields(uint32_t tile, int r, int u, uint32_t (&w)[BITS]) {
  if constexpr (BITS == 2) {          // 32-byte swizzle
    lds_v2(tile + r * 32 + ((((u >> 1) ^ (r >> 2)) & 1) << 4) + (u & 1) * 8, w[0], w[1]);
  } else if constexpr (BITS == 4) {   // 64-byte swizzle
    lds_v4(tile + r * 64 + (((u ^ (r >> 1)) & 3) << 4), w[0], w[1], w[2], w[3]);
  } else if constexpr (BITS == 8) {   // 128-byte swizzle
    lds_v4(tile + r * 128 + (((2 * u) ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
    lds_v4(tile + r * 128 + (((2 * u + 1) ^ (r & 7)) << 4), w[4], w[5], w[6], w[7]);
  } else if constexpr (BITS == 6) {
#pragma unroll
    for (int i = 0; i < 3; ++i) lds_v2(tile + r * 96 + u * 24 + 8 * i, w[2 * i], w[2 * i + 1]);
  } else {                            // 3 and 5 words: an odd unit starts on an odd word
    const uint32_t at = tile + r * (16 * BITS) + u * (4 * BITS);
    if (u & 1) {
      w[0] = lds_u32(at);
#pragma unroll
      for (int i = 1; i < BITS; i += 2) lds_v2(at + 4 * i, w[i], w[i + 1]);
    } else {
#pragma unroll
      for (int i = 0; i + 1 < BITS; i += 2) lds_v2(at + 4 * i, w[i], w[i + 1]);
      w[BITS - 1] = lds_u32(at + 4 * (BITS - 1));
    }
  }
}

// Field e of a BITS-word chunk, not yet masked.
template <int BITS>
__device__ __forceinline__ uint32_t field_raw(const uint32_t (&w)[BITS], int e) {
  const int wi = (e * BITS) >> 5, sh = (e * BITS) & 31;
  return sh + BITS > 32 ? __funnelshift_r(w[wi], w[(wi + 1) % BITS], sh) : (w[wi] >> sh);
}

// s*q+b of 32 consecutive fields in fp32, split into hi + lo numbers of T (16 registers of pairs each, in
// order).  bf16: hi is the value cut off after 8 bits, lo the rounded rest, 2^-17 of the value is lost; f16: both rounded, what
// is lost is 2^-22 of the value from 1/8 up and at most 2^-25 below (against 64 bits the products' errors are those of
// fp32 weights to three digits, for weights of 1e-4 to 1: the rounding of the result is far larger).  f16 numbers end at
// 65504: a larger weight gives inf - inf, which the epilogue finds (repair).
template <int BITS, typename T>
__device__ __forceinline__ void split32(const uint32_t (&w)[BITS], float s, float b, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
  constexpr uint32_t mask = (1u << BITS) - 1u;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 2 * j + h;
      uint32_t f;   // 0x4B0000qq is 2^23 + q exactly
      if constexpr (BITS == 8) f = __byte_perm(w[e >> 2], 0x4B000000u, 0x7540 | (e & 3));
      else f = lop3_and_or(field_raw<BITS>(w, e), mask, 0x4B000000u);
      v[h] = fmaf(__uint_as_float(f) - 8388608.0f, s, b);
    }
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      hi[j] = __byte_perm(__float_as_uint(v[0]), __float_as_uint(v[1]), 0x7632);
      const float l0 = v[0] - __uint_as_float(__float_as_uint(v[0]) & 0xFFFF0000u);
      const float l1 = v[1] - __uint_as_float(__float_as_uint(v[1]) & 0xFFFF0000u);
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo[j]) : "f"(l1), "f"(l0));
    } else {
      asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi[j]) : "f"(v[1]), "f"(v[0]));
      const float2 h2 = __half22float2(*reinterpret_cast<const __half2*>(&hi[j]));
      asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo[j]) : "f"(v[1] - h2.y), "f"(v[0] - h2.x));
    }
  }
}

// Unpacks 32 consecutive BITS-wide fields (BITS words, LSB-first bit stream) of one row into
// 16 bf16x2 registers in natural k order, applying w = s*q + b (one rounding).  s and b are
// the raw bf16 bit patterns.
// Fast form: a field inside a byte, masked in place and read as bf16, is the subnormal (or smallest normal) number
// q * 2^(o - 133), o its lowest bit in the byte: bit 7 is the exponent's lowest bit and continues the subnormal scale
// exactly.  fma.rn.bf16x2 takes subnormal inputs exactly, so one fma with the scale times 2^(133 - o) gives
// round(q * s + b).  A byte permute brings the bytes of fields 2j and 2j+1 into the halves of a register; a field that
// ends in the next byte is first shifted down (a quarter of the 3-bit fields, half of the 5- and 6-bit ones).  1.5 to
// 2 instructions per field (8 bits: 1) where extracting both fields, joining them and subtracting an offset took 3.5.
// It needs the scaled scale to stay finite and normal: biased exponent of s in [1, 121]; other scales (zero, subnormal,
// |s| >= 2^-6 * 2, inf, nan) take the general form.
__device__ __forceinline__ bool scale_has_room(uint32_t s_bits) { return (s_bits & 0x7FFFu) - 0x80u < (122u << 7) - 0x80u; }
template <int BITS>
__device__ __forceinline__ void dequant32_fast(const uint32_t (&w)[BITS], uint32_t s_bits, uint32_t b_bits, uint32_t (&out)[16]) {
  const uint32_t b2 = b_bits * 0x00010001u, s0 = (s_bits + (133u << 7)) * 0x00010001u;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int pl = 2 * j * BITS, ph = pl + BITS;   // first bits of the two fields
    if constexpr (BITS == 8) {
      out[j] = fma_bf16x2(__byte_perm(w[pl >> 5], 0u, (pl & 31) ? 0x4342 : 0x4140), s0, b2);
    } else {
      constexpr uint32_t m = (1u << BITS) - 1u;
      const bool dl = (pl & 7) + BITS <= 8, dh = (ph & 7) + BITS <= 8;   // inside a byte
      const uint32_t ol = dl ? pl & 7 : 0, oh = dh ? ph & 7 : 0;
      const uint32_t bl = dl ? (pl >> 3) & 3 : 0, bh = (dh ? (ph >> 3) & 3 : 0) + 4;
      const uint32_t v = __byte_perm(dl ? w[pl >> 5] : field_raw<BITS>(w, 2 * j), dh ? w[ph >> 5] : field_raw<BITS>(w, 2 * j + 1),
                                     bl * 0x11 + bh * 0x1100);
      out[j] = fma_bf16x2(v & (m << ol | m << (oh + 16)), s0 - (ol * 0x0080u + oh * 0x00800000u), b2);
    }
  }
}
template <int BITS>
__device__ __forceinline__ void dequant32_any(const uint32_t (&w)[BITS], uint32_t s_bits, uint32_t b_bits, uint32_t (&out)[16]) {
  constexpr uint32_t kMagic = 0x43004300u;  // (128.0, 128.0): 0x4300 | q == 128 + q for q < 128
  const uint32_t s2 = s_bits * 0x00010001u, b2 = b_bits * 0x00010001u;
  if constexpr (BITS == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t p[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // p[i] = (q[i], q[i+4]) as bf16 pairs
        const uint32_t t = lop3_and_or(w[j] >> (4 * i), 0x000F000Fu, kMagic);
        p[i] = fma_bf16x2(sub_bf16x2(t, kMagic), s2, b2);
      }
      out[4 * j + 0] = __byte_perm(p[0], p[1], 0x5410);  // (w0, w1)
      out[4 * j + 1] = __byte_perm(p[2], p[3], 0x5410);  // (w2, w3)
      out[4 * j + 2] = __byte_perm(p[0], p[1], 0x7632);  // (w4, w5)
      out[4 * j + 3] = __byte_perm(p[2], p[3], 0x7632);  // (w6, w7)
    }
  } else if constexpr (BITS == 8) {
    // beyond the bf16 integers: through float (0x4B0000qq == 2^23 + q)
    const float sf = __uint_as_float(s_bits << 16), bf = __uint_as_float(b_bits << 16);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int b0 = (j & 1) * 2;
      const float q0 = __uint_as_float(__byte_perm(w[j >> 1], 0x4B000000u, 0x7540 | b0)) - 8388608.0f;
      const float q1 = __uint_as_float(__byte_perm(w[j >> 1], 0x4B000000u, 0x7540 | (b0 + 1))) - 8388608.0f;
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[j]) : "f"(fmaf(q1, sf, bf)), "f"(fmaf(q0, sf, bf)));
    }
  } else {
    constexpr uint32_t mask = (1u << BITS) - 1u;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      uint32_t f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = 2 * j + h, wi = (e * BITS) >> 5, sh = (e * BITS) & 31;
        f[h] = (sh + BITS > 32) ? __funnelshift_r(w[wi], w[(wi + 1) % BITS], sh) : (w[wi] >> sh);
      }
      const uint32_t lo = lop3_and_or(f[0], mask, 0x4300u), hi = lop3_and_or(f[1], mask, 0x4300u);
      const uint32_t t = __byte_perm(lo, hi, 0x5410);
      out[j] = fma_bf16x2(sub_bf16x2(t, kMagic), s2, b2);
    }
  }
}


template <typename T>
__device__ __forceinline__ float bits_to_float(uint32_t v) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float(v << 16);
  else return __half2float(__ushort_as_half((unsigned short)v));
}
// N bytes, of which the first `n` are read and the rest are zeros.
template <int N>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(n) : "memory");
}
__device__ __forceinline__ void st_shared_u16(uint32_t at, unsigned short v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(v) : "memory");
}
// The same for scales or biases that are not aligned to a row's chunk (an expert's slice of a stack of odd size): one stage,
// value by value; a lone value goes where the copied word would have it.  (Out of line: the ordinary loop stays short.)
__device__ __noinline__ void copy_values(uint32_t dst, uint32_t bias_off, const unsigned short* s, const unsigned short* b, int n) {
  for (int e = 0; e < n; ++e) {
    st_shared_u16(dst + 2 * e, __ldg(s + e));
    st_shared_u16(dst + bias_off + 2 * e, __ldg(b + e));
  }
}
__device__ __forceinline__ void st_shared_v4(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// One unit of work of a pair: a tile, or one of the parts of K of a tile.
struct Unit {
  int w_row0;      // transpose: first packed row of this block's half of the tile; else first output column
  int w_row_end;   // transpose: one past the last packed row of this matrix
  int n0;          // first output column of this block's half
  int x_row0;      // first activation row
  int rows, neff;  // valid activation rows, and the same rounded up to what the MMA takes
  int ks0, ks1;    // stages of K
  int parts;       // number of ranges that share the tile; with more than one:
  int slot, slot0; // index of the unit's partial sums, and of those of the tile's first part
  int rtile;       // index of the tile among those left over
};
// Pair j's range of the chunks (spc stages, whole chunks of scales) of the tiles left over.
__device__ __forceinline__ int range_begin(const TcParams& p, int j, int chunks) { return (int)((uint32_t)(j * p.rem * chunks) / (uint32_t)p.cut); }   // (tc_plan keeps it below 2^31)
// Units of the loop `for (u = pair; u < end; u += pairs)`: the pair's whole tiles, then the pieces of its range.
__device__ __forceinline__ int units_end(const TcParams& p, int pair, int pairs) {
  if (p.mtiles) return *p.n_mtiles * p.n_tiles;
  if (pair >= p.cut) return p.full;
  const int chunks = (p.K + kStageK - 1) / kStageK / p.spc, lo = range_begin(p, pair, chunks), hi = range_begin(p, pair + 1, chunks);
  return p.full + (hi > lo ? (hi - 1) / chunks - lo / chunks + 1 : 0) * pairs;
}
__device__ __forceinline__ Unit unit_at(const TcParams& p, int u, int rank) {
  Unit t;
  const int kst = p.K / kStageK + (p.K % kStageK != 0);
  if (p.mtiles == nullptr) {
    int tile = u;
    t.ks0 = 0;
    t.ks1 = kst;
    t.parts = 1;
    if (u >= p.full && p.cut > 0) {
      const int pairs = gridDim.x >> 1, v = u - p.full, i = v / pairs, j = v - i * pairs, chunks = kst / p.spc;
      const int lo = range_begin(p, j, chunks), hi = range_begin(p, j + 1, chunks), r = lo / chunks + i, first = r * chunks;
      t.ks0 = (max(lo, first) - first) * p.spc;
      t.ks1 = (min(hi, first + chunks) - first) * p.spc;
      // the pair whose range holds chunk c is ((c + 1) * cut - 1) / (rem * chunks)
      const uint32_t all = p.rem * chunks;
      const int j0 = (int)((uint32_t)((first + 1) * p.cut - 1) / all), j1 = (int)((uint32_t)((first + chunks) * p.cut - 1) / all);
      t.parts = j1 - j0 + 1;
      t.slot = j + r;           // ranges in order, one more at every tile boundary
      t.slot0 = j0 + r;
      t.rtile = r;
      tile = p.full + r;
    }
    const int tn = p.m_tiles == 1 ? tile : tile / p.m_tiles, tm = tile - tn * p.m_tiles;
    t.n0 = tn * (2 * kTileRows) + rank * kTileRows;
    t.w_row0 = t.n0;
    t.w_row_end = p.N;
    t.x_row0 = tm * p.NT;
    t.rows = min(p.M - t.x_row0, p.NT);
  } else {
    const int g = u / p.n_tiles, tn = u - g * p.n_tiles;
    const MTile mt = p.mtiles[g];
    t.n0 = tn * (2 * kTileRows) + rank * kTileRows;
    t.w_row0 = mt.expert * p.N + t.n0;
    t.w_row_end = mt.expert * p.N + p.N;
    t.x_row0 = mt.row0;
    t.rows = mt.rows;
    t.ks0 = 0;
    t.ks1 = kst;
    t.parts = 1;
  }
  t.neff = (t.rows + 31) & ~31;
  return t;
}

// Epilogue of 32 output columns (one warp): the accumulator comes as mma fragments, is rounded in pairs, transposed
// through shared memory (stmatrix; 64 bytes per token, 16-byte chunks xor-ed with token / 2) and leaves as
// 16-byte stores, 64 contiguous bytes per token.  While an accumulator that has no twin is being read, the tensor
// pipe waits: 64 tokens are staged with one load in flight ahead of the one being rounded, and stored after.
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(uint32_t a, uint32_t b) {
  uint32_t d;
  if constexpr (std::is_same<T, __nv_bfloat16>::value) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(b)), "f"(__uint_as_float(a)));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(b)), "f"(__uint_as_float(a)));
  return d;
}
__device__ __forceinline__ void load_piece(uint32_t tmem, uint32_t (&r)[16]) {   // 32 lanes x 16 columns
  tcgen05_ld_16x16(tmem, r);
  tcgen05_ld_16x16(tmem + (16u << 16), r + 8);
}
// Nonzero where one of a pair of numbers is not finite.
template <typename T>
__device__ __forceinline__ uint32_t odd_pair(uint32_t v) {
  constexpr bool kBf = std::is_same<T, __nv_bfloat16>::value;
  return ((v & (kBf ? 0x7F807F80u : 0x7C007C00u)) + (kBf ? 0x00800080u : 0x04000400u)) & 0x80008000u;   // an exponent of ones carries
}
template <typename T>
__device__ __forceinline__ void stage_piece(uint32_t stg, int lane, const uint32_t (&r)[16]) {
  const uint32_t row = lane & 7, at = stg + row * 64 + ((((uint32_t)lane >> 3) ^ (row >> 1)) << 4);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    stmatrix_x4_trans(at + i * 512, pack_pair<T>(r[4 * i], r[4 * i + 1]), pack_pair<T>(r[4 * i + 2], r[4 * i + 3]),
                      pack_pair<T>(r[8 + 4 * i], r[8 + 4 * i + 1]), pack_pair<T>(r[8 + 4 * i + 2], r[8 + 4 * i + 3]));
}
// 32 tokens straight from the accumulator, for rows of y off 8-byte boundaries (an output head of any size): a lane has a
// column, and the warp stores 64 contiguous bytes per token.  Through the staging tile such rows went out as eight 2-byte
// stores per lane, each instruction in 32 places (4 bits, us: 700
// tokens through [32001, 4096] 201 -> 150, 2048 through [14301, 2048] 167 -> 117).
// Returns nonzero (WATCH) where a result is not finite, as store_chunk does.
template <typename T, bool WATCH>
__device__ __forceinline__ uint32_t store_columns(const TcParams& p, const Unit& t, const uint32_t (&v)[32], int n, int c, int lim) {
  if (n >= p.N) return 0;
  uint32_t odd = 0;
  if constexpr (WATCH) {
#pragma unroll
    for (int j = 0; j < 32; j += 2) odd |= odd_pair<T>(pack_pair<T>(j < lim ? v[j] : 0u, j + 1 < lim ? v[j + 1] : 0u));
  }
  for (int q = 0; q < p.n_out; ++q) {
    T* y = static_cast<T*>(p.y_out[q]) + p.col0 + n;
    if (p.dst_row == nullptr) {
      y += (long long)(t.x_row0 + c) * p.ld;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (j < lim) *y = Elem<T>::from_float(__uint_as_float(v[j]));
        y += p.ld;
      }
    } else {
      const int* row = p.dst_row + t.x_row0 + c;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < lim) y[(long long)row[j] * p.ld] = Elem<T>::from_float(__uint_as_float(v[j]));
    }
  }
  return odd;
}
template <typename T, bool ROWS16, bool WATCH>
__device__ __forceinline__ uint32_t store_chunk(const TcParams& p, const Unit& t, uint32_t stg, int lane, int n0, int c, int lim) {
  const int n = n0 + (lane & 3) * 8;
  const bool whole = n + 8 <= p.N;
  uint32_t odd = 0;
  if (n >= p.N) return odd;
  for (int tok = lane >> 2; tok < lim; tok += 8) {
    uint4 v;
    lds_v4(stg + tok * 64 + (((lane & 3) ^ ((tok >> 1) & 3)) << 4), v.x, v.y, v.z, v.w);
    if constexpr (WATCH) odd |= odd_pair<T>(v.x) | odd_pair<T>(v.y) | odd_pair<T>(v.z) | odd_pair<T>(v.w);
    const int m = t.x_row0 + c + tok;
    const long long at = (long long)(p.dst_row ? p.dst_row[m] : m) * p.ld + p.col0 + n;
    for (int q = 0; q < p.n_out; ++q) {
      T* dst = static_cast<T*>(p.y_out[q]) + at;
      if (ROWS16 && whole) {
        *reinterpret_cast<uint4*>(dst) = v;
      } else if (whole) {
        reinterpret_cast<uint2*>(dst)[0] = make_uint2(v.x, v.y);
        reinterpret_cast<uint2*>(dst)[1] = make_uint2(v.z, v.w);
      } else {
        const T* e = reinterpret_cast<const T*>(&v);
        for (int j = 0; j < 8 && n + j < p.N; ++j) dst[j] = e[j];
      }
    }
  }
  return odd;
}

// A cut tile's fp32 sums, part by part in order, by NW warps of the last block to arrive, which leave them zeroed.  A warp
// takes whole tokens, a lane four columns of each: 16-byte loads, two tokens of four parts at a time.  Returns nonzero (WATCH)
// where a result is not finite.
template <typename T, int NW, bool WATCH>
__device__ __forceinline__ uint32_t sum_parts(const TcParams& p, const Unit& t, int rank, int warp, int lane) {
  uint32_t odd = 0;
  __threadfence();
  const size_t pitch = 2 * (size_t)p.NT * kTileRows / 4;   // from one part to the next
  float4* p0 = reinterpret_cast<float4*>(p.partial + ((size_t)t.slot0 * 2 + rank) * ((size_t)p.NT * kTileRows)) + lane;
  const int n4 = t.n0 + 4 * lane;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int c = warp; c < t.rows; c += 2 * NW) {
    const int n_tok = c + NW < t.rows ? 2 : 1;
    float4* q0 = p0 + (size_t)c * (kTileRows / 4);
    float4 sum[2] = {zero, zero};
    for (int s = 0; s < t.parts; s += 4) {
      float4 v[2][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          v[k][i] = k < n_tok && s + i < t.parts ? __ldcg(q0 + (size_t)(s + i) * pitch + k * (NW * kTileRows / 4)) : zero;
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) { sum[k].x += v[k][i].x; sum[k].y += v[k][i].y; sum[k].z += v[k][i].z; sum[k].w += v[k][i].w; }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k >= n_tok) break;
      for (int s = 0; s < t.parts; ++s) __stcg(q0 + (size_t)s * pitch + k * (NW * kTileRows / 4), zero);
      const uint2 o = make_uint2(pack_pair<T>(__float_as_uint(sum[k].x), __float_as_uint(sum[k].y)),
                                 pack_pair<T>(__float_as_uint(sum[k].z), __float_as_uint(sum[k].w)));
      if constexpr (WATCH) odd |= odd_pair<T>(o.x) | odd_pair<T>(o.y);
      const long long at = (long long)(t.x_row0 + c + k * NW) * p.ld + p.col0 + n4;
      for (int q = 0; q < p.n_out; ++q) {
        T* dst = static_cast<T*>(p.y_out[q]) + at;
        if (n4 + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
          *reinterpret_cast<uint2*>(dst) = o;
        } else {
          const T* e = reinterpret_cast<const T*>(&o);
          for (int i = 0; i < 4 && n4 + i < p.N; ++i) dst[i] = e[i];
        }
      }
    }
  }
  return odd;
}

// The elements of a tile that are not finite, from the weights themselves in fp32, by the epilogue warps.
template <typename T, int BITS, bool TRANSPOSED>
__device__ __forceinline__ void repair(const TcParams& p, int n0, int x_row0, int rows) {
  const int64_t row_words = (TRANSPOSED ? (int64_t)p.K : (int64_t)p.N) * BITS / 32;
  const int group = kTileRows / p.g4;
  for (int i = threadIdx.x - 32 * kFirstEpilogue; i < rows * kTileRows; i += 32 * kEpilogueWarps) {
    const int n = n0 + (i & (kTileRows - 1));
    if (n >= p.N) continue;
    const long long m = x_row0 + i / kTileRows;
    T* y = static_cast<T*>(p.y_out[0]) + m * p.N + n;
    if (fabsf(Elem<T>::to_float(*y)) < INFINITY) continue;
    float sum = 0.0f;
    for (int k = 0; k < p.K && sum == sum; ++k) {
      const int64_t r = TRANSPOSED ? n : k, sc = r * p.row_groups + (TRANSPOSED ? k : n) / group;
      const float w = fmaf((float)stream_get<BITS>(p.wq + r * row_words, TRANSPOSED ? k : n), bits_to_float<T>(p.scales[sc]), bits_to_float<T>(p.biases[sc]));
      sum = fmaf(Elem<T>::to_float(static_cast<const T*>(p.x)[m * p.K + k]), w, sum);
    }
    *y = Elem<T>::from_float(sum);
  }
}

// ROWS16: the rows of y start on 16-byte boundaries (an instantiation of its own: the registers of the other stores cost the
// ordinary products 2 to 4 %).
template <typename T, int BITS, Form F, bool ROWS16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
qmm_tc_kernel(const __grid_constant__ TcMaps maps, const __grid_constant__ TcParams p) {
  using S = Shape<BITS, F>;
  constexpr bool kT = S::kT, kSplit = F != Form::Round;
  constexpr int kSub = S::kSub, kSlotsA = S::kSlotsA;
  constexpr bool kRingFixed = S::kStagesP == S::kFewStagesP;
  const uint32_t nsp = kRingFixed ? S::kStagesP : p.nsp;   // packed stages; where not fixed, a power of two
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // carve-up: [A ring of SplitT] [B ring: nsb stages of two NT/2 * 128-byte sub-tiles] [P ring] [S ring] [barriers]
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t b_sub = (uint32_t)p.NT * 64u;       // NT / 2 rows of 128 bytes (NT is a multiple of 32)
  const uint32_t b_stage = 2u * b_sub;
  unsigned char* ring_b = smem + S::kSmemA;
  unsigned char* ring_p = ring_b + (size_t)p.nsb * b_stage;
  unsigned char* ring_s = ring_p + (size_t)nsp * S::kPStageBytes;   // per chunk: 128 rows of scales, 128 of biases
  unsigned char* staging = ring_s + p.s_slots * 2 * kTileRows * p.cb;    // a tile per epilogue warp
  Barriers* bars = reinterpret_cast<Barriers*>(staging + kEpilogueWarps * S::kStageOut);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int nacc = p.NT <= kAccCols / 2 ? 2 : 1;

  if (threadIdx.x == 32 * 3) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.w) : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x[i]) : "memory");
  }
  if (warp == 0) {   // a lane per barrier of each kind: one thread after another took 0.7 us
    if (lane < (int)nsp) { mbar_init(smem_u32(&bars->full_p[lane]), 1); mbar_init(smem_u32(&bars->empty_p[lane]), S::kPArrivals); }
    if (lane < p.s_slots) {
      mbar_init(smem_u32(&bars->full_s[lane]), 32);
      mbar_init(smem_u32(&bars->empty_s[lane]), p.spc * S::kPArrivals);
    }
    if (lane < p.nsb) mbar_init(smem_u32(&bars->full_b[lane]), 1);
    if (lane < kSlotsA) mbar_init(smem_u32(&bars->full_a[lane]), 2 * kUnpackWarps / S::kSets);
    if (lane < kDoneRing) mbar_init(smem_u32(&bars->done[lane]), 1);
    if (lane < 2) { mbar_init(smem_u32(&bars->acc_full[lane]), 1); mbar_init(smem_u32(&bars->acc_empty[lane]), 2 * kEpilogueWarps); }
    if (lane == 0) {
      bars->abort_flag = 0;
      bars->odd = 0;
      bars->ended = 0;
      bars->help = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
  }
  if (warp == 1) {
    tcgen05_alloc(smem_u32(&bars->tmem_base), kTmemCols);
    tcgen05_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  // Warps 2 and 3 fetch for this block alone: they start at once and meet the other block when they are done.  (33 rows through
  // [4096, 4096], clock marks: first packed stage used 5.1 us after entry, now 4.1 to 5.2; first MMA 7.0 -> 6.0.)
  cluster_arrive();
  if (warp != 2 && warp != 3) cluster_wait();
  tcgen05_fence_after();
  const int total = units_end(p, pair, pairs);
  const uint32_t tmem_base = bars->tmem_base;
  const uint32_t tmem_a = tmem_base + kAccCols;

  if (warp == 0) {
    // ------------------------------------------------------------ x tiles: this block's half of the tokens
    // (The three one-thread roles run at one instruction in ten to twenty cycles beside the unpack warps: their
    // loops hold addresses and ring positions and nothing else.)
    if (elect_one()) {
      const uint32_t full = smem_u32(&bars->full_b[0]), lfull = leader_addr(full), done = smem_u32(&bars->done[0]);
      const uint32_t ring = smem_u32(ring_b), nsb = p.nsb;
      uint32_t sb = 0, it = 0, dst = ring;
      bool ok = true;
      for (int u = pair; ok && u < total; u += pairs) {
        const Unit t = unit_at(p, u, rank);
        const int half = t.neff >> 1, row = t.x_row0 + rank * half;
        const uint32_t bytes = (uint32_t)t.neff * 256u;   // both blocks' halves
        for (int k = t.ks0 * kStageK, k1 = t.ks1 * kStageK; k < k1; k += kStageK, ++it) {
          if (it >= nsb) {   // the stage that used this slot last has been multiplied
            const uint32_t ia = (it - nsb) * kSub + kSub - 1;
            if (!mbar_nap<40>(done + (ia % kDoneRing) * 8, (ia / kDoneRing) & 1u, abort_flag)) { ok = false; break; }
          }
          if (rank == 0) mbar_expect_tx(full + sb * 8, bytes);
          const uint32_t lbar = lfull + sb * 8;
          int r = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int box = 128 >> i;
            if (half & box) {
              tma_load_2d_pair(dst + r * 128, &maps.x[i], k, row + r, lbar);
              tma_load_2d_pair(dst + b_sub + r * 128, &maps.x[i], k + 64, row + r, lbar);
              r += box;
            }
          }
          dst += b_stage;
          if (++sb == nsb) { sb = 0; dst = ring; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader block)
    if (rank == 0 && elect_one()) {
      const uint32_t full_b = smem_u32(&bars->full_b[0]), full_a = smem_u32(&bars->full_a[0]), done = smem_u32(&bars->done[0]);
      const uint64_t desc0 = sw128_desc(smem_u32(ring_b), 16, 1024);
      const uint32_t d_stage = b_stage >> 4, d_sub = b_sub >> 4, nsb = p.nsb;
      const uint64_t desc_a0 = sw128_desc(smem_u32(smem), 8192, 1024);
      uint32_t tcount = 0, ia = 0, sa = 0, pa = 0, sb = 0, pb = 0;
      uint64_t bd0 = desc0;
      bool ok = true;
      for (int u = pair; ok && u < total; u += pairs, ++tcount) {
        const Unit t = unit_at(p, u, 0);
        const uint32_t idesc = make_idesc<T, F>(t.neff);
        const uint32_t ab = nacc == 2 ? (tcount & 1) : 0, an = nacc == 2 ? (tcount >> 1) : tcount;
        const uint32_t acc = tmem_base + ab * (kAccCols / 2);
        if (!mbar_wait_spin(smem_u32(&bars->acc_empty[ab]), (an & 1) ^ 1, abort_flag)) break;
        uint32_t first = 0;
        for (int ks = t.ks0; ok && ks < t.ks1; ++ks) {
          const uint64_t bd1 = bd0 + d_sub;
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            // both looks are under way before either is needed
            const bool ra = mbar_test(full_a + sa * 8, pa), rb = sub > 0 || mbar_test(full_b + sb * 8, pb);
            if (!(ra && rb)) {
              if (!mbar_wait_spin(full_a + sa * 8, pa, abort_flag) || !mbar_wait_spin(full_b + sb * 8, pb, abort_flag)) { ok = false; break; }
            }
            tcgen05_fence_after();
            if constexpr (F == Form::Round) {
              const uint32_t ta = tmem_a + sa * 64;
#pragma unroll
              for (int kk = 0; kk < 8; ++kk) tcgen05_mma_ts(acc, ta + kk * 8, (kk < 4 ? bd0 : bd1) + (kk & 3) * 2, idesc, kk ? 1u : first);
            } else if constexpr (F == Form::Split) {
              const uint32_t ta = tmem_a + sa * 64;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                tcgen05_mma_ts(acc, ta + kk * 8, (sub ? bd1 : bd0) + kk * 2, idesc, kk ? 1u : first);
                tcgen05_mma_ts(acc, ta + 32 + kk * 8, (sub ? bd1 : bd0) + kk * 2, idesc, 1u);
              }
            } else {
              const uint64_t ad = desc_a0 + sa * 2048;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                tcgen05_mma_ss(acc, ad + kk * 128, (sub ? bd1 : bd0) + kk * 2, idesc, kk ? 1u : first);
                tcgen05_mma_ss(acc, ad + 1024 + kk * 128, (sub ? bd1 : bd0) + kk * 2, idesc, 1u);
              }
            }
            first = 1;
            tcgen05_commit_pair(done + (ia % kDoneRing) * 8);
            ++ia;
            if (++sa == (uint32_t)kSlotsA) { sa = 0; pa ^= 1; }
          }
          bd0 += d_stage;
          if (++sb == nsb) { sb = 0; pb ^= 1; bd0 = desc0; }
        }
        if (!ok) break;
        tcgen05_commit_pair(smem_u32(&bars->acc_full[ab]));
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ packed W tiles
    if (elect_one()) {
      const uint32_t full = smem_u32(&bars->full_p[0]), empty = smem_u32(&bars->empty_p[0]), ring = smem_u32(ring_p);
      uint32_t sp = 0, pp = 1, dst = ring;
      bool ok = true;
      for (int u = pair; ok && u < total; u += pairs) {
        const Unit t = unit_at(p, u, rank);
        // transpose: 128 k of 128 rows; else 128 columns of 128 rows (= k)
        int c0 = kT ? (t.n0 / kTileRows) * S::kPRowBytes : t.ks0 * S::kPRowBytes;
        int c1 = kT ? t.ks0 * kStageK : t.w_row0;
        for (int n = t.ks1 - t.ks0; n > 0; --n) {
          if (!mbar_nap<40>(empty + sp * 8, pp, abort_flag)) { ok = false; break; }
          mbar_expect_tx(full + sp * 8, S::kPStageBytes);
          tma_load_2d(dst, &maps.w, c0, c1, full + sp * 8);
          if constexpr (kT) c1 += kStageK; else c0 += S::kPRowBytes;
          dst += S::kPStageBytes;
          if (++sp == nsp) { sp = 0; pp ^= 1; dst = ring; }
        }
      }
    }
    __syncwarp();
    cluster_wait();
  } else if (warp == 3) {
    // ------------------------------------------------------------ scales and biases
    // Asynchronous copies straight into the ring, counted on the chunk's barrier; a lane serves four rows.
    // A copy instruction touches as many cache lines as it has lanes and costs a thousand cycles per eight:
    // a chunk is as many stages as a copy's 16 bytes and the rows' alignment allow.  cp.async moves no
    // less than 4 bytes: where a stage needs one value, the aligned word that holds it is copied.
    uint32_t ss = 0, ps = 0;
    bool ok = true;
    const uint32_t half_chunk = (uint32_t)kTileRows * p.cb;   // bytes of a chunk's scales; the biases follow
    for (int u = pair; ok && u < total; u += pairs) {
      const Unit t = unit_at(p, u, rank);
      for (int ks = t.ks0; ks < t.ks1; ks += p.spc) {
        if (!mbar_nap<100>(smem_u32(&bars->empty_s[ss]), ps ^ 1, abort_flag)) { ok = false; break; }
        const uint32_t dst = smem_u32(ring_s) + ss * 2 * half_chunk + lane * p.cb;
        auto row_at = [&](int i) -> long long {   // rows past the end: results are never stored (transpose), x is zero (no transpose)
          if constexpr (kT) return (long long)min(ks * kStageK + lane + 32 * i, p.K - 1) * p.row_groups + min(t.n0 / kTileRows * p.g4, p.row_groups - p.g4);
          else return (long long)min(t.w_row0 + lane + 32 * i, t.w_row_end - 1) * p.row_groups + ks * p.g4;
        };
        if (p.narrow) {
          for (int i = 0; i < 4; ++i) {
            const long long o = row_at(i);
            copy_values(dst + 32 * i * p.cb + (p.g4 == 1 ? (uint32_t)(o & 1) * 2 : 0), half_chunk, p.scales + o, p.biases + o, p.g4);
          }
          mbar_arrive(smem_u32(&bars->full_s[ss]));
          if (++ss == (uint32_t)p.s_slots) { ss = 0; ps ^= 1; }
          continue;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const long long o = row_at(i);
          const uint32_t d = dst + 32 * i * p.cb;
          if (p.cb == 16) {
            cp_async<16>(d, p.scales + o, 16);
            cp_async<16>(d + half_chunk, p.biases + o, 16);
          } else if (p.cb == 8) {
            cp_async<8>(d, p.scales + o, 8);
            cp_async<8>(d + half_chunk, p.biases + o, 8);
          } else {
            const long long w = o & ~1ll;   // (even already unless the chunk is one value)
            const int n = w + 1 < p.n_scales ? 4 : 2;
            cp_async<4>(d, p.scales + w, n);
            cp_async<4>(d + half_chunk, p.biases + w, n);
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->full_s[ss])) : "memory");
        if (++ss == (uint32_t)p.s_slots) { ss = 0; ps ^= 1; }
      }
    }
    __syncwarp();
    cluster_wait();
  } else if (warp < kFirstEpilogue) {
    // ------------------------------------------------------------ unpack
    // Everything here is counted in instructions: the warps of a scheduler make one instruction about
    // every ten cycles each, and a trip of 450 instructions for 64 fields per thread (150 of them the
    // unpacking) bounded the kernel at 2000 cycles per stage.  So a warp takes a whole slot row per trip
    // (128 or 64 k), ring positions are masks, and addresses are kept as shared-memory words.
    constexpr int kSets = S::kSets, kSetWarps = kUnpackWarps / kSets;
    const int wu = warp - kFirstUnpack;
    const uint32_t set = wu / kSetWarps;   // A slot uses ia = set (mod kSets) are this warp's
    const int quad = warp & 3;             // TMEM lane quadrant this warp may access
    const int half = kT ? (wu >> 2) & 1 : 0;   // kT: which half of the slot's k
    const uint32_t sub = set % kSub;       // which slot of a stage
    const int row = kT ? (int)sub * 64 + half * 32 + lane : quad * 32 + lane;   // packed row of the tile (transpose: TMEM lane)
    const uint32_t t_slot = tmem_a + ((uint32_t)(quad * 32) << 16) + set * 64;   // (transpose) as many slots as sets
    // offset of unit un's value in a chunk row's stage: one value per 1, 2 or 4 units
    const int gsh = p.g4 == 4 ? 0 : (p.g4 == 2 ? 1 : 2);
    const uint32_t s_mask = p.s_slots - 1, s_sh = 31 - __clz(p.s_slots);
    const uint32_t spc_sh = p.spc == 4 ? 2 : (p.spc == 2 ? 1 : 0), half_chunk = (uint32_t)kTileRows * p.cb;
    const bool single = p.spc * p.g4 == 1;   // a chunk is one value: the odd or the even half of the copied word
    const uint32_t s_row = smem_u32(ring_s) + row * p.cb;
    const uint32_t p_base = smem_u32(ring_p), p_sh = nsp == 8 ? 3 : 2;
    const uint32_t bar_a = leader_addr(smem_u32(&bars->full_a[0])), bar_done = smem_u32(&bars->done[0]);
    const uint32_t bar_fp = smem_u32(&bars->full_p[0]), bar_ep = smem_u32(&bars->empty_p[0]);
    const uint32_t bar_fs = smem_u32(&bars->full_s[0]), bar_es = smem_u32(&bars->empty_s[0]);
    uint32_t it0 = 0, c0 = 0;              // stages and chunks of the units before this one
    uint32_t ia = set;
    bool ok = true;
    for (int u = pair; ok && u < total; u += pairs) {
      const Unit t = unit_at(p, u, rank);
      const uint32_t n_st = t.ks1 - t.ks0;
      const uint32_t o_row = kT ? min(t.n0 / kTileRows, p.row_groups - 1) : (uint32_t)min(t.w_row0 + row, t.w_row_end - 1) * p.row_groups + t.ks0;
      for (; ia < (it0 + n_st) * kSub; ia += kSets) {
        const uint32_t it = ia / kSub, ks = it - it0;      // ks counts from the unit's first stage
        const uint32_t c = c0 + (ks >> spc_sh), sp = kRingFixed ? it % S::kStagesP : it & (nsp - 1);
        bool got = mbar_wait_hot(bar_fs + (c & s_mask) * 8, (c >> s_sh) & 1u, abort_flag);
        // Where a ring slot passes from one set to another (its length no multiple of the stages per turn), a set can
        // come to it before the slot's previous stage, another set's, has landed.  The parity asked for is then that of
        // the use before, which reads as complete.  So such rings wait first until the set's own A slot has been multiplied:
        // products run in order, and the slot's previous stage is an earlier one.
        if constexpr (S::kStagesP % (kSets / kSub > 0 ? kSets / kSub : 1) != 0) {
          static_assert(kRingFixed && S::kStagesP > kSlotsA / kSub, "the previous stage of a ring slot is not after that of the A slot");
          const uint32_t prev = ia - kSlotsA;
          got = got && (ia < (uint32_t)kSlotsA || mbar_wait_hot(bar_done + (prev % kDoneRing) * 8, (prev / kDoneRing) & 1u, abort_flag));
        }
        got = got && mbar_wait_hot(bar_fp + sp * 8, (kRingFixed ? it / S::kStagesP : it >> p_sh) & 1u, abort_flag);
        // A wait may run out for some of the lanes only.  They stay (what they unpack is never stored) until the vote below:
        // the votes and tcgen05 instructions from here on need the whole warp.
        const uint32_t tile = p_base + sp * S::kPStageBytes;
        uint32_t at = s_row + (c & s_mask) * 2 * half_chunk + (ks & (p.spc - 1)) * 2 * p.g4;
        if (single) {
          const uint32_t o = kT ? (uint32_t)min((int)((t.ks0 + ks) * kStageK + row), p.K - 1) * p.row_groups + o_row : o_row + ks;
          at += (o & 1) * 2;
        }
        const uint32_t sa = kT ? ia % kSlotsA : set;
        auto slot_free = [&]() {   // the slot's last use has been multiplied
          const uint32_t prev = ia - kSlotsA;
          const bool free = got && (ia < (uint32_t)kSlotsA || mbar_wait_hot(bar_done + (prev % kDoneRing) * 8, (prev / kDoneRing) & 1u, abort_flag));
          return __all_sync(0xFFFFFFFFu, free) != 0;
        };
        if constexpr (F == Form::Round) {
          // One vote and one straight line for the slot's four units: every shared-memory read is under way before it is
          // needed.  With a vote per unit, after which its words and scales were read: 512 tokens through [28672, 8192] at 3 bits 216
          // us, now 209; 57 rows through [4096, 11008] 26.6, now 24.6 (with the shorter set-up and the helpers' sums below).
          // The biases wait for their unit: four registers less (2 bits in groups of 32, 64 rows through [14336, 4096]: 27.4 -> 26.8 us,
          // 57 rows of 4 bits 23.2 -> 23.0).
          uint32_t sv[4], w[2][BITS], vals[16];
#pragma unroll
          for (int un = 0; un < 4; ++un) {
            sv[un] = lds_u16(at + 2 * (un >> gsh));
          }
          load_fields<BITS>(tile, row, 0, w[0]);
          if (__all_sync(0xFFFFFFFFu, scale_has_room(sv[0]) && scale_has_room(sv[1]) && scale_has_room(sv[2]) && scale_has_room(sv[3]))) {
#pragma unroll
            for (int un = 0; un < 4; ++un) {
              if (un < 3) load_fields<BITS>(tile, row, un + 1, w[(un + 1) & 1]);
              dequant32_fast<BITS>(w[un & 1], sv[un], lds_u16(at + 2 * (un >> gsh) + half_chunk), vals);
              if (un == 0) {
                if (!slot_free()) { ok = false; break; }
                tcgen05_fence_after();
              }
              tcgen05_st_x16(t_slot + un * 16, vals);
            }
          } else if (slot_free()) {
            tcgen05_fence_after();
#pragma unroll
            for (int un = 0; un < 4; ++un) {
              load_fields<BITS>(tile, row, un, w[0]);
              dequant32_any<BITS>(w[0], sv[un], lds_u16(at + 2 * (un >> gsh) + half_chunk), vals);
              tcgen05_st_x16(t_slot + un * 16, vals);
            }
          } else {
            ok = false;
          }
        } else if constexpr (F == Form::Split) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t w[BITS], hi[16], lo[16];
            const int un = 2 * (int)sub + h;
            load_fields<BITS>(tile, row, un, w);
            const uint32_t v = at + 2 * (un >> gsh);
            split32<BITS, T>(w, bits_to_float<T>(lds_u16(v)), bits_to_float<T>(lds_u16(v + half_chunk)), hi, lo);
            if (h == 0) {
              if (!slot_free()) { ok = false; break; }
              tcgen05_fence_after();
            }
            tcgen05_st_x16(t_slot + h * 16, hi);
            tcgen05_st_x16(t_slot + 32 + h * 16, lo);
          }
        } else {
          uint32_t w[BITS], hi[16], lo[16];
          load_fields<BITS>(tile, row, quad, w);
          const uint32_t v = at + 2 * (quad >> gsh);
          split32<BITS, T>(w, bits_to_float<T>(lds_u16(v)), bits_to_float<T>(lds_u16(v + half_chunk)), hi, lo);
          if (!slot_free()) { ok = false; break; }
          // M-major tile: 128 bytes (64 columns) per k, 16-byte chunks xor-ed with k mod 8
          const int k = half * 32 + lane;
          const uint32_t a0 = smem_u32(smem) + sa * 32768 + (quad >> 1) * 8192 + k * 128;
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            const uint32_t d = a0 + (((((quad & 1) << 2) + c4) ^ (k & 7)) << 4);
            st_shared_v4(d, hi[4 * c4], hi[4 * c4 + 1], hi[4 * c4 + 2], hi[4 * c4 + 3]);
            st_shared_v4(d + 16384, lo[4 * c4], lo[4 * c4 + 1], lo[4 * c4 + 2], lo[4 * c4 + 3]);
          }
        }
        if (!ok) break;
        // Publish the slot; the packed stage and the scales are released only here, after the stores that
        // consume the unpacked registers: the shared-memory reads above have then returned for every lane.
        if constexpr (kT) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        } else {
          tcgen05_wait_st();
          tcgen05_fence_before();
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cluster(bar_a + sa * 8);
          mbar_arrive(bar_ep + sp * 8);
          mbar_arrive(bar_es + (c & s_mask) * 8);
        }
      }
      it0 += n_st;
      c0 += n_st >> spc_sh;
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quad = warp & 3;
    const int chalf = (warp - kFirstEpilogue) >> 2;  // which half of the token columns
    const uint32_t stg = smem_u32(staging) + (warp - kFirstEpilogue) * S::kStageOut;
    const uint32_t lane_field = (uint32_t)(quad * 32) << 16;
    uint32_t tcount = 0;
    for (int u = pair; u < total; u += pairs, ++tcount) {
      const Unit t = unit_at(p, u, rank);
      const uint32_t ab = nacc == 2 ? (tcount & 1) : 0, an = nacc == 2 ? (tcount >> 1) : tcount;
      // One warp looks, the others are held by a hardware barrier.  All go by what it found: the abort flag may be
      // raised between two warps' looks at it, and a warp that left alone would keep the others at the next barrier.
      // (Two words: the one of two tiles ago has been read by all who have passed the last tile's barrier.)
      if (warp == kFirstEpilogue) {
        const bool landed = __all_sync(0xFFFFFFFFu, mbar_nap<100>(smem_u32(&bars->acc_full[ab]), an & 1, abort_flag));
        if (lane == 0) bars->landed[tcount & 1] = landed;
        __syncwarp();
      }
      asm volatile("bar.sync 3, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
      if (!bars->landed[tcount & 1]) break;
      tcgen05_fence_after();
      const int n = t.n0 + quad * 32 + lane;
      const int c_begin = chalf * (t.neff >> 1), c_end = c_begin + (t.neff >> 1);
      const uint32_t acc = tmem_base + ab * (kAccCols / 2) + lane_field;
      // after the last load the accumulator is free for another tile's MMAs
      auto release = [&]() {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_addr(smem_u32(&bars->acc_empty[ab])));
      };
      if (t.parts == 1 && (ROWS16 || p.y_align == 8)) {
        uint32_t r[2][16];
        load_piece(acc + c_begin, r[0]);
        for (int c0 = c_begin; c0 < c_end; c0 += S::kOutTok) {
#pragma unroll
          for (int i = 0; i < S::kOutTok / 16; ++i) {
            const int c = c0 + 16 * i;
            if (c < c_end) {                             // (halves are whole 16-column pieces)
              tcgen05_wait_ld16(r[i & 1]);
              if (c + 16 < c_end) load_piece(acc + c + 16, r[(i + 1) & 1]);
              else release();
              stage_piece<T>(stg + i * 1024, lane, r[i & 1]);
            }
          }
          __syncwarp();
          if (store_chunk<T, ROWS16, kSplit>(p, t, stg, lane, t.n0 + quad * 32, c0, min(min(t.rows, c_end) - c0, S::kOutTok))) bars->odd = 1;
          __syncwarp();   // the staging tile may be written again
        }
      } else {
        float* part = p.partial + ((size_t)t.slot * 2 + rank) * ((size_t)p.NT * kTileRows) + quad * 32 + lane;
        for (int c = c_begin; c < c_end; c += 32) {
          uint32_t v[32];
          tcgen05_ld_x32(acc + c, v);
          tcgen05_wait_ld();
          if (c + 32 >= c_end) release();
          const int lim = min(t.rows, c_end) - c;  // valid columns of this chunk
          if (!ROWS16 && t.parts == 1) {
            if (store_columns<T, kSplit>(p, t, v, n, c, lim)) bars->odd = 1;
            __syncwarp();   // the next load needs the whole warp
            continue;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < lim) __stcg(part + (size_t)(c + j) * kTileRows, __uint_as_float(v[j]));
        }
      }
      if (t.parts > 1) {
        // The last of the tile's pairs to arrive (per block of the pair: each has its own 128 columns) adds the parts.
        __threadfence();
        asm volatile("bar.sync 2, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
        if (warp == kFirstEpilogue && lane == 0) {
          uint32_t* ctr = p.counters + t.rtile * 2 + rank;
          const bool last = atomicAdd(ctr, 1u) == (uint32_t)t.parts - 1;
          if (last) *ctr = 0;
          bars->last = last;
        }
        asm volatile("bar.sync 2, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
        if (bars->last) {
          if (kSplit && warp == kFirstEpilogue && lane == 0) bars->ended |= 1u << ((u - p.full) / pairs & 31);
          if (!kSplit && u + pairs >= total) {
            if (warp == kFirstEpilogue && lane == 0) bars->help = 1;   // below, with the unpack warps
          } else if (sum_parts<T, kEpilogueWarps, kSplit>(p, t, rank, warp - kFirstEpilogue, lane)) {
            bars->odd = 1;
          }
        }
        asm volatile("bar.sync 2, %0;" ::"n"(kEpilogueWarps * 32) : "memory");   // `last` may be written again
      }
    }
  }
  if constexpr (!kSplit) {
    if (warp >= kFirstUnpack) {
      // A pair's last unit, where it is part of a cut tile and this block the last of the tile's, is added up by the unpack warps
      // too, which have nothing left to do.  (The split forms' loops have no registers for it: 1531 f16 tokens 275 -> 279 us.)
      constexpr int kAll = kUnpackWarps + kEpilogueWarps;
      __syncwarp();
      asm volatile("bar.sync 4, %0;" ::"n"(kAll * 32) : "memory");
      if (bars->help) {
        const int u = pair + (total - 1 - pair) / pairs * pairs;
        sum_parts<T, kAll, false>(p, unit_at(p, u, rank), rank, warp - kFirstUnpack, lane);
      }
    }
  } else {
    if (warp >= kFirstEpilogue) {
      __syncwarp();
      asm volatile("bar.sync 3, %0;" ::"n"(kEpilogueWarps * 32) : "memory");   // every result and every `odd` is there
      if (bars->odd != 0) {
        for (int u = pair; u < total; u += pairs) {
          const Unit t = unit_at(p, u, rank);
          if (t.parts == 1 || (bars->ended >> ((u - p.full) / pairs & 31) & 1)) repair<T, BITS, !kT>(p, t.n0, t.x_row0, t.rows);
        }
      }
    }
  }

  // ---- teardown: both blocks meet, then the tensor memory is returned
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicMax(&p.status[0], 3u);
  if (threadIdx.x == 0) peer_signal_tail(p.sig);   // every store of the block precedes the barrier above
  __syncwarp();
  cluster_sync();
  if (warp == 1) {
    tcgen05_fence_after();
    tcgen05_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------- host side
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
                    qres == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<EncodeFn>(sym) : nullptr;
  }();
  return fn;
}

int sm_pairs() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 74;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 2) n = 148;
    cached[dev] = n / 2;
  }
  return cached[dev];
}

Form form_of(int dtype, bool transpose) {
  return !transpose ? Form::SplitT : (dtype == B200Q_BF16 ? Form::Round : Form::Split);
}

template <int BITS, Form F>
size_t fixed_smem(int cb, int slots, bool few) {
  using S = Shape<BITS, F>;
  return 1024 + S::kSmemA + (size_t)(few ? S::kFewStagesP : S::kStagesP) * S::kPStageBytes + (size_t)slots * 2 * kTileRows * cb + kEpilogueWarps * S::kStageOut +
         sizeof(Barriers) + 64;
}
size_t fixed_smem(int bits, Form f, int cb, int slots, bool few) {
  size_t n = 0;
  B200Q_DISPATCH_BITS(bits, BITS, {
    n = f == Form::Round ? fixed_smem<BITS, Form::Round>(cb, slots, few)
                         : (f == Form::Split ? fixed_smem<BITS, Form::Split>(cb, slots, few) : fixed_smem<BITS, Form::SplitT>(cb, slots, few));
  });
  return n;
}

// Token width of a tile and the number of pairs that share the tiles left over from whole waves: the choice with the
// least estimated time, in cycles.  A stage takes the longer of its MMAs (4 cycles per token, 8 when split) and of its
// unpacking; a tile adds the exposed part of its epilogue; the last part of a cut tile to arrive reads and zeroes
// `parts` times its fp32 sums, and all of them pass through L2 three times (1531 f16 tokens through [14336, 4096], 40
// tiles left over: 273 us with a whole last wave, 289 us cut; 512 tokens through [28672, 8192], 2 left over: 234 / 217).
struct TcPlan {
  int nt, m_tiles, n_tiles, full, rem, cut;
};
TcPlan tc_plan(int64_t M, int64_t N, int64_t K, Form f) {
  TcPlan best{};
  double best_t = 1e300;
  const int pairs = sm_pairs();
  const int kst = (int)((K + kStageK - 1) / kStageK);
  const int n_tiles = (int)((N + 2 * kTileRows - 1) / (2 * kTileRows));
  const int cap = (int)(M >= 256 ? 256 : (M + 31) / 32 * 32);
  for (int nt = cap; nt >= 32; nt -= 32) {
    const int64_t m_tiles = (M + nt - 1) / nt;
    const int64_t tiles = m_tiles * n_tiles;
    const double stage = f == Form::Round ? (4.0 * nt > 800 ? 4.0 * nt : 800.0) : (8.0 * nt > 1300 ? 8.0 * nt : 1300.0);
    const double exposed = nt <= kAccCols / 2 ? 1000.0 : 1000.0 + 10.0 * nt, tile = kst * stage + exposed;
    const int64_t waves = tiles / pairs;
    const int rem = (int)(tiles - waves * pairs);
    // s parts per tile, on rem * s pairs; or, where that leaves pairs idle, an equal range for every pair
    for (int s = 1; s <= 16 && (s == 1 || (s * 4 <= kst && (long long)pairs * pairs * (kst + 1) < INT32_MAX)); ++s) {
      const bool all = (long long)rem * s > pairs;
      const int cut = all ? pairs : rem * s;
      double last = 0.0;
      if (rem > 0 && s == 1) last = tile;
      if (rem > 0 && s > 1) {
        const double share = (double)rem * kst / cut, parts = all ? (double)(int)(kst / share) + 2.0 : (double)s;
        last = (double)(int)(share + 0.999) * stage + (all ? 2.0 : 1.0) * exposed + 4000.0 + parts * (24.0 * nt + 200.0) + 1.2 * nt * cut;
      }
      const double t = waves * tile + last;
      if (t < best_t) {
        best_t = t;
        best = TcPlan{nt, (int)m_tiles, n_tiles, (int)(s == 1 ? tiles : tiles - rem), s == 1 ? 0 : rem, s == 1 ? 0 : cut};
      }
      if (all || rem == 0) break;
    }
  }
  return best;
}

size_t counter_bytes(const TcPlan& pl) { return ((size_t)pl.rem * 2 * 4 + 255) / 256 * 256; }
size_t split_bytes(const TcPlan& pl) {
  if (pl.cut == 0) return 0;
  return counter_bytes(pl) + (size_t)(pl.cut + pl.rem) * 2 * pl.nt * kTileRows * 4;
}

// x maps (boxes of 128, 64, 32 and 16 rows of 64 k) and the map of the packed matrix.
int encode_maps(TcMaps& m, const char* tag, const void* x, int64_t x_rows, int64_t K, int dtype, const void* wq,
                int64_t w_rows, int64_t w_row_bytes, int bits) {
  EncodeFn enc = encode_fn();
  if (!enc) return fail(B200Q_ERR_CUDA, "[%s] cuTensorMapEncodeTiled is not available", tag);
  if (int rc = bind_context()) return rc;
  const cuuint32_t estr[2] = {1, 1};
  for (int i = 0; i < 4; ++i) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)x_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)(128 >> i)};
    CUresult r = enc(&m.x[i], dtype == B200Q_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                     const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(B200Q_ERR_CUDA, "[%s] tensor map for x failed (%d)", tag, (int)r);
  }
  const cuuint64_t dims[2] = {(cuuint64_t)w_row_bytes, (cuuint64_t)w_rows};
  const cuuint64_t strides[1] = {(cuuint64_t)w_row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(16 * bits), (cuuint32_t)kTileRows};
  const CUtensorMapSwizzle sw = bits == 2 ? CU_TENSOR_MAP_SWIZZLE_32B : (bits == 4 ? CU_TENSOR_MAP_SWIZZLE_64B
                                : (bits == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE));
  CUresult r = enc(&m.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(wq), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(B200Q_ERR_CUDA, "[%s] tensor map for w failed (%d)", tag, (int)r);
  return B200Q_OK;
}

// Once per kernel, device and thread.
int allow_smem(const void* kernel) {
  constexpr int kMost = 64;   // instantiations: 48
  static thread_local const void* done[64][kMost];
  static thread_local int count[64];
  int dev = 0;
  B200Q_CUDA_OK(cudaGetDevice(&dev));
  const bool known = dev >= 0 && dev < 64;
  for (int i = 0; known && i < count[dev]; ++i)
    if (done[dev][i] == kernel) return B200Q_OK;
  B200Q_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
  if (known && count[dev] < kMost) done[dev][count[dev]++] = kernel;
  return B200Q_OK;
}

template <typename T, int BITS, Form F>
int launch_one(unsigned grid, size_t smem, cudaStream_t st, const TcMaps& maps, const TcParams& p) {
  // A plain launch: programmatic stream serialization would hide about 2 us of set-up.  It was taken back after a launch
  // that failed once, while a ring of packed stages could still be read before its stage had landed (see the unpack warps); it
  // has not been tried again since.
  auto go = [&](auto kernel) -> int {
    if (int rc = allow_smem((const void*)kernel)) return rc;
    kernel<<<grid, kThreads, smem, st>>>(maps, p);
    B200Q_LAUNCH_OK("qmm_tc_kernel");
    return B200Q_OK;
  };
  return p.y_align == 16 ? go(qmm_tc_kernel<T, BITS, F, true>) : go(qmm_tc_kernel<T, BITS, F, false>);
}

int row_alignment(const TcParams& p) {
  uintptr_t at = (uintptr_t)p.ld * 2 | (uintptr_t)p.col0 * 2;
  for (int q = 0; q < p.n_out; ++q) at |= reinterpret_cast<uintptr_t>(p.y_out[q]);
  return (at & 15) == 0 ? 16 : ((at & 7) == 0 ? 8 : 2);
}

// Completes the parameters that depend on the shape of the kernel and launches it for `units` units of work.
int launch_tc(int dtype, int bits, int group, Form f, long long units, cudaStream_t st, const TcMaps& maps, TcParams& p) {
  p.y_align = row_alignment(p);
  p.g4 = kTileRows / group;
  p.spc = 1;
  if (f != Form::SplitT)
    while (p.spc < 4 && p.spc * p.g4 < 8 && p.row_groups % (2 * p.spc * p.g4) == 0 &&
           ((reinterpret_cast<uintptr_t>(p.scales) | reinterpret_cast<uintptr_t>(p.biases)) % (4 * p.spc * p.g4)) == 0)
      p.spc *= 2;
  p.cb = p.spc * p.g4 * 2 < 4 ? 4 : p.spc * p.g4 * 2;
  p.narrow = (reinterpret_cast<uintptr_t>(p.scales) | reinterpret_cast<uintptr_t>(p.biases)) % p.cb != 0;   // (only with chunks of one stage)
  p.s_slots = p.spc == 4 ? 2 : 4;
  const size_t stage = (size_t)p.NT * 128;
  const bool few = fixed_smem(bits, f, p.cb, p.s_slots, false) + 3 * stage > kSmemMax;   // three stages of x come first
  p.nsp = few ? 4 : 8;
  const size_t fixed = fixed_smem(bits, f, p.cb, p.s_slots, few);
  long long nsb = (long long)((kSmemMax - fixed) / stage);
  p.nsb = (int)(nsb > kMaxStagesB ? kMaxStagesB : nsb);
  size_t smem = fixed + p.nsb * stage;
  // What is left holds more chunks of scales.
  const size_t chunk = 2 * kTileRows * (size_t)p.cb;
  while (2 * p.s_slots <= kMaxSlotsS && smem + p.s_slots * chunk <= kSmemMax) {
    smem += p.s_slots * chunk;
    p.s_slots *= 2;
  }
  // More than half of an SM's shared memory: guarantees one block per SM, so the 512-column
  // tensor-memory allocation never has to wait for a co-resident block of this kernel.
  if (smem < 120 * 1024) smem = 120 * 1024;
  const long long pairs = sm_pairs();
  const unsigned grid = 2u * (unsigned)(units < pairs ? units : pairs);
  int rc = fail(B200Q_ERR_UNSUPPORTED, "[quantized_matmul] unsupported bits %d", bits);
  B200Q_DISPATCH_BITS(bits, BITS, {
    if (f == Form::Round) rc = launch_one<__nv_bfloat16, BITS, Form::Round>(grid, smem, st, maps, p);
    else if (f == Form::Split) rc = launch_one<__half, BITS, Form::Split>(grid, smem, st, maps, p);
    else if (dtype == B200Q_BF16) rc = launch_one<__nv_bfloat16, BITS, Form::SplitT>(grid, smem, st, maps, p);
    else rc = launch_one<__half, BITS, Form::SplitT>(grid, smem, st, maps, p);
  });
  return rc;
}

void set_outputs(TcParams& p, const PeerOut& peers, void* y, int64_t ld) {
  if (peers.n > 0) {
    p.n_out = peers.n; p.ld = peers.ld; p.col0 = peers.col0;
    for (int q = 0; q < peers.n; ++q) p.y_out[q] = peers.y[q];
    p.sig = peers.sig;
  } else {
    p.n_out = 1; p.ld = ld; p.col0 = 0; p.y_out[0] = y;
  }
}

}  // namespace

// bf16 or f16, one matrix.  Transposed: whole stages of 128 k.  Not transposed: whole blocks of 128
// columns (a tile row of the packed matrix) and a row pitch of x that TMA takes.
bool qmm_tc_supported(const QmmArgs& a) {
  if ((a.dtype != B200Q_BF16 && a.dtype != B200Q_F16) || a.w_batched || a.batch != 1) return false;
  if (a.M < 1 || a.N < 1 || a.K < 1 || a.M > (1 << 30) || a.N > (1 << 30)) return false;
  if ((a.transpose ? a.K : a.N) % kStageK != 0 || a.K % 8 != 0) return false;
  // TMA: 16-byte aligned bases and row pitches
  return !((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.wq)) & 15);
}

size_t qmm_tc_workspace_bytes(const QmmArgs& a) {
  return split_bytes(tc_plan(a.M, a.N, a.K, form_of(a.dtype, a.transpose))) + kStatusBytes;
}

int qmm_tc(const QmmArgs& a, cudaStream_t st) {
  if (!a.ws || a.ws_bytes < kStatusBytes)
    return fail(B200Q_ERR_WORKSPACE, "[quantized_matmul] workspace of %zu bytes required, %zu given",
                (size_t)kStatusBytes, a.ws_bytes);
  const Form f = form_of(a.dtype, a.transpose);
  TcPlan pl = tc_plan(a.M, a.N, a.K, f);
  // a caller's smaller workspace, or one that the 16-byte accesses to the partial sums do not fit: no shared tiles
  if (a.ws_bytes < split_bytes(pl) + kStatusBytes || (reinterpret_cast<uintptr_t>(a.ws) & 15)) {
    pl.full += pl.rem;
    pl.rem = pl.cut = 0;
  }
  const int64_t qaxis = a.transpose ? a.K : a.N;
  TcMaps maps;
  if (int rc = encode_maps(maps, "quantized_matmul", a.x, a.M, a.K, a.dtype, a.wq, a.transpose ? a.N : a.K,
                           qaxis * a.bits / 8, a.bits))
    return rc;
  TcParams p{};
  p.scales = (const unsigned short*)a.scales;
  p.biases = (const unsigned short*)a.biases;
  p.x = a.x;
  p.wq = a.wq;
  set_outputs(p, a.peers, a.y, a.N);
  p.status = reinterpret_cast<uint32_t*>(static_cast<char*>(a.ws) + a.ws_bytes - kStatusBytes);
  p.M = (int)a.M; p.N = (int)a.N; p.K = (int)a.K;
  p.NT = pl.nt; p.m_tiles = pl.m_tiles; p.n_tiles = pl.n_tiles;
  p.full = pl.full; p.rem = pl.rem; p.cut = pl.cut;
  p.counters = static_cast<uint32_t*>(a.ws);
  p.partial = reinterpret_cast<float*>(static_cast<char*>(a.ws) + counter_bytes(pl));
  p.row_groups = (int)(qaxis / a.group);
  p.n_scales = (a.transpose ? a.N : a.K) * p.row_groups;
  return launch_tc(a.dtype, a.bits, a.group, f, (long long)pl.full + pl.cut, st, maps, p);
}

int qmm_tc_grouped(const GroupedArgs& a, cudaStream_t st) {
  TcMaps maps;
  if (int rc = encode_maps(maps, "gather_qmm", a.x_sorted, a.n_rows, a.K, B200Q_BF16, a.wq, a.E * a.N, a.K * a.bits / 8, a.bits))
    return rc;
  TcParams p{};
  p.mtiles = static_cast<const MTile*>(a.mtiles);
  p.n_mtiles = a.n_mtiles;
  p.dst_row = a.dst_row;
  p.scales = (const unsigned short*)a.scales;
  p.biases = (const unsigned short*)a.biases;
  set_outputs(p, a.peers, a.y, a.N);
  p.ld = a.N; p.col0 = 0;
  p.status = a.status;
  p.M = (int)a.n_rows; p.N = (int)a.N; p.K = (int)a.K;
  p.NT = a.nt; p.m_tiles = 0;
  p.n_tiles = (int)((a.N + 2 * kTileRows - 1) / (2 * kTileRows));
  p.row_groups = (int)(a.K / a.group);
  p.n_scales = a.E * a.N * p.row_groups;
  // an upper bound of the units; the kernel reads the exact count
  return launch_tc(B200Q_BF16, a.bits, a.group, Form::Round, (long long)p.n_tiles * a.max_mtiles, st, maps, p);
}

}  // namespace b200q
