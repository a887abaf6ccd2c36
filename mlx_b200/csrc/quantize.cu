// Affine group-wise quantize / dequantize kernels (HBM-bound element-wise work).
//
// quantize reproduces, bit for bit, the float arithmetic of the reference CPU
// implementation quantize<T,U> (mlx/backend/cpu/quantized.cpp:1148-1211): three IEEE
// divisions, rint (round half to even), clamp to [0, 2^bits-1], scale/bias rounded to
// T with round-to-nearest-even.  dequantize reproduces the op-composed reference
// (mlx/ops.cpp:5320-5323): multiply then add, each rounded to T.
//
// Both are bound by HBM only if a value costs about ten instructions; how they get there stands at the kernels.
#include <type_traits>

#include "common.cuh"

namespace b200q {
namespace {

template <typename T>
__device__ __forceinline__ void store8(T* __restrict__ p, const float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint4 raw;
    T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = Elem<T>::from_float(v[i]);
    *reinterpret_cast<uint4*>(p) = raw;
  }
}

// ---------------------------------------------------------------------------- quantize
// A warp takes kIter * 512 consecutive values: a lane loads 16 of every 512 (two 128-bit loads of a 16-bit type,
// coalesced), so a group of g values lies in g/16 neighbouring lanes.  Minima and maxima are found by
// shuffles; then every lane computes scale and bias of ONE group (the three IEEE divisions, which in a thread per
// eight values cost more than everything else) and hands them back by shuffles.
//
// q = rint((w - bias) / scale) without a division per value: fma(w - bias, r, 1.5 * 2^23) rounds the product to
// an integer (half to even) in the low mantissa bits.  It is done twice, with r a few units in the last
// place below and above 1 / scale: where both agree, the correctly rounded quotient rounds to the same
// integer; the others are divided as the reference does.  That is no rare case: for 16-bit weights w - bias is a
// multiple of a coarse unit, and about one value in 250 lies exactly half way between two fields.
// No lower clamp is needed: w - bias has the sign of scale, and where bias is 0 every |w / scale| is at most 1/2.
// The fields are packed by multiply-adds on the bit patterns: sum_i u_i 2^(i bits) mod 2^32 is the packed word plus a
// constant.  About 12 instructions per value, none on the quarter-rate conversion unit (which rint and
// the float-to-int conversion used).
// 28672 x 8192 bf16, groups of 64 (device time): to 4 bits 321 -> 136 us (4.4 TB/s), to 8 bits 401 -> 152; f32 99.
// Up to 2^22 values a warp takes one row: there the blocks are few and it is one warp's chain that takes the time (four
// rows / one, us: 256 x 1024 bf16 to 4 bits 3.7 / 2.5, f32 to 8 bits 4.3 / 2.6; 1024 x 1024 3.9 / 3.0; 2048 x 2048 6.2 /
// 6.0; 4096 x 4096 13.5 / 16.3).  Groups of 32 have two rows per warp and keep them (64 x 1024 2.5 / 2.4, 2048 x 2048 5.1 / 5.6).
constexpr int64_t kSmall = 1 << 22;
template <int GROUP, bool SMALL>
struct QuantShape {
  static constexpr int kIter = GROUP == 32 ? 2 : (SMALL ? 1 : 4);   // 512-value rows per warp: at most one group per lane
  static constexpr int kLanes = GROUP / 16;                 // lanes per group
  static constexpr int kPerIter = 512 / GROUP;              // groups per row
};

constexpr float kMagic = 12582912.0f;                       // 1.5 * 2^23
constexpr uint32_t kMagicBits = 0x4B400000u;

// sum of u[i] * 2^(i * BITS) over N values, without the magic numbers' share
template <int BITS, int N>
__device__ __forceinline__ uint32_t pack_fields(const float* u) {
  uint32_t acc = __float_as_uint(u[N - 1]), c = kMagicBits;
#pragma unroll
  for (int i = N - 2; i >= 0; --i) {
    acc = acc * (1u << BITS) + __float_as_uint(u[i]);
    c = c * (1u << BITS) + kMagicBits;
  }
  acc -= c;
  return acc;
}

// Fields whose bit is set in `which` (field 0: bit 15), computed with the division of the reference and put into
// the packed words o.  Out of line: inlined divisions push the loop out of the instruction cache.
template <typename T, int BITS>
__device__ __noinline__ uint4 exact_fields(const T* __restrict__ w, float s, float b, uint32_t which, uint4 o) {
  constexpr float n_bins = (float)((1 << BITS) - 1);
  constexpr unsigned long long kMask = (1ull << BITS) - 1ull;
  unsigned long long lo = (unsigned long long)o.y << 32 | o.x, hi = (unsigned long long)o.w << 32 | o.z;
  while (which) {
    const int i = __clz((int)which) - 16;
    which &= ~(0x8000u >> i);
    float q = rintf(__fdiv_rn(__fsub_rn(Elem<T>::to_float(w[i]), b), s));
    q = (q < 0.0f) ? 0.0f : q;
    q = (n_bins < q) ? n_bins : q;
    const unsigned long long f = (uint32_t)q;
    const int at = i * BITS;
    if (at < 64) lo = (lo & ~(kMask << at)) | f << at;
    if (at >= 64) hi = (hi & ~(kMask << (at - 64))) | f << (at - 64);
    else if (at + BITS > 64) hi = (hi & ~(kMask >> (64 - at))) | f >> (64 - at);
  }
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

template <typename T>
struct Pack16 {   // 16 values in the form they are loaded in
  T v[16];
};
template <typename T>
__device__ __forceinline__ void load16(const T* p, Pack16<T>& d) {
  const uint4* s = reinterpret_cast<const uint4*>(p);
  uint4* o = reinterpret_cast<uint4*>(d.v);
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i) o[i] = __ldg(s + i);
}
template <typename T>
__device__ __forceinline__ void minmax16(const Pack16<T>& d, float& lo, float& hi) {
  if constexpr (sizeof(T) == 4) {
    lo = hi = d.v[0];
#pragma unroll
    for (int i = 1; i < 16; ++i) { lo = fminf(lo, d.v[i]); hi = fmaxf(hi, d.v[i]); }
  } else {
    using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
    const T2* p = reinterpret_cast<const T2*>(d.v);
    T2 l = p[0], h = p[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) { l = __hmin2(l, p[i]); h = __hmax2(h, p[i]); }
    lo = fminf(Elem<T>::to_float(l.x), Elem<T>::to_float(l.y));
    hi = fmaxf(Elem<T>::to_float(h.x), Elem<T>::to_float(h.y));
  }
}

template <typename T, int BITS, int GROUP, bool SMALL>
__global__ void __launch_bounds__(256)
quantize_kernel(const T* __restrict__ w, uint32_t* __restrict__ wq, T* __restrict__ scales,
                T* __restrict__ biases, int64_t n) {
  using Q = QuantShape<GROUP, SMALL>;
  constexpr int IT = Q::kIter;
  const int lane = threadIdx.x & 31;
  const int64_t base = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (IT * 512);
  if (base >= n) return;

  Pack16<T> v[IT];
  float lo[IT], hi[IT];
#pragma unroll
  for (int k = 0; k < IT; ++k) {
    const int64_t at = base + k * 512 + lane * 16;
    if (at < n) {
      load16(w + at, v[k]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[k].v[i] = Elem<T>::from_float(0.0f);
    }
  }
#pragma unroll
  for (int k = 0; k < IT; ++k) {
    minmax16(v[k], lo[k], hi[k]);
#pragma unroll
    for (int off = 1; off < Q::kLanes; off <<= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], off));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], off));
    }
  }
  // lane j takes group j of the warp's values: group j % kPerIter of row j / kPerIter
  float w_min = 0.0f, w_max = 0.0f;
#pragma unroll
  for (int k = 0; k < IT; ++k) {
    const int src = (lane % Q::kPerIter) * Q::kLanes;
    const float l = __shfl_sync(0xffffffffu, lo[k], src), h = __shfl_sync(0xffffffffu, hi[k], src);
    if (lane / Q::kPerIter == k) { w_min = l; w_max = h; }
  }
  // The reference's comparisons pass over NaN and start from (inf, -inf); a minimum is NaN only where all of the group is.
  if (w_min != w_min) { w_min = INFINITY; w_max = -INFINITY; }
  constexpr float n_bins = (float)((1 << BITS) - 1);
  const float eps = 1e-7f;
  const bool mask = fabsf(w_min) > fabsf(w_max);
  float scale = __fdiv_rn(__fsub_rn(w_max, w_min), n_bins);
  scale = (scale < eps) ? eps : scale;
  scale = mask ? scale : -scale;
  const float edge = mask ? w_min : w_max;
  const float q0 = rintf(__fdiv_rn(edge, scale));
  float bias = 0.0f;
  if (q0 != 0.0f) {
    scale = __fdiv_rn(edge, q0);
    bias = edge;
  }
  const float inv = __frcp_rn(scale);
  {
    const int64_t g = base / GROUP + lane;
    if (lane < IT * Q::kPerIter && g * GROUP < n) {
      scales[g] = Elem<T>::from_float(scale);
      biases[g] = Elem<T>::from_float(bias);
    }
  }

#pragma unroll
  for (int k = 0; k < IT; ++k) {
    const int src = k * Q::kPerIter + lane / Q::kLanes;
    const float s = __shfl_sync(0xffffffffu, scale, src), b = __shfl_sync(0xffffffffu, bias, src);
    const float r = __shfl_sync(0xffffffffu, inv, src);
    const float r0 = r * (1.0f - 0x1p-21f), r1 = r * (1.0f + 0x1p-21f);
    float u[16];
    float differ = 0.0f;   // 16 bits, value 0 in the highest: both results are integers k or k + 1
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float d = __fsub_rn(Elem<T>::to_float(v[k].v[i]), b);
      const float t = __fmaf_rn(d, r0, kMagic);
      differ = __fmaf_rn(differ, 2.0f, __fsub_rn(__fmaf_rn(d, r1, kMagic), t));
      u[i] = fminf(t, kMagic + n_bins);
    }
    const int64_t at = base + k * 512 + lane * 16;
    uint32_t o[4] = {0, 0, 0, 0};   // 16 * BITS bits per lane: whole words, or with 3 and 5 bits half a word more
    if constexpr (BITS == 2) {
      o[0] = pack_fields<2, 16>(u);
    } else if constexpr (BITS == 4) {
      o[0] = pack_fields<4, 8>(u); o[1] = pack_fields<4, 8>(u + 8);
    } else if constexpr (BITS == 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = pack_fields<8, 4>(u + 4 * i);
    } else if constexpr (BITS == 3) {
      const uint32_t a = pack_fields<3, 8>(u), c = pack_fields<3, 8>(u + 8);   // 24 bits each
      o[0] = a | c << 24; o[1] = c >> 8;
    } else if constexpr (BITS == 6) {
      const uint32_t a = pack_fields<6, 4>(u), c = pack_fields<6, 4>(u + 4), d = pack_fields<6, 4>(u + 8), e = pack_fields<6, 4>(u + 12);
      o[0] = a | c << 24; o[1] = c >> 8 | d << 16; o[2] = d >> 16 | e << 8;
    } else {
      const uint32_t a = pack_fields<5, 4>(u), c = pack_fields<5, 4>(u + 4), d = pack_fields<5, 4>(u + 8), e = pack_fields<5, 4>(u + 12);   // 20 bits each
      o[0] = a | c << 20; o[1] = c >> 12 | d << 8 | e << 28; o[2] = e >> 4;
    }
    // (The comparison means nothing where 1 / scale or a product is not an ordinary number: all sixteen then.)
    const bool plain = fabsf(s) < 1e30f && fabsf(r) < 1e30f;
    if ((differ != 0.0f || !plain) && at < n) {
      const uint32_t which = plain && differ > 0.0f && differ < 65536.0f ? (uint32_t)differ : 0xFFFFu;
      const uint4 e = exact_fields<T, BITS>(w + at, s, b, which, make_uint4(o[0], o[1], o[2], o[3]));
      o[0] = e.x; o[1] = e.y; o[2] = e.z; o[3] = e.w;
    }
    if constexpr (BITS == 3 || BITS == 5) {
      // two lanes share a word: the even lane stores it and the words before it, the odd lane the words after it
      constexpr int F = BITS / 2;                            // whole words of a lane
      uint32_t* out = wq + (at / 32) * BITS;
      const uint32_t next = __shfl_down_sync(0xffffffffu, o[0], 1);
      if (at < n) {
        if ((lane & 1) == 0) {
#pragma unroll
          for (int i = 0; i < F; ++i) out[i] = o[i];
          out[F] = (o[F] & 0xFFFFu) | next << 16;
        } else {
#pragma unroll
          for (int i = 0; i < F; ++i) out[F + 1 + i] = o[i] >> 16 | o[i + 1] << 16;
        }
      }
    } else if (at < n) {
      uint32_t* out = wq + at * BITS / 32;
      if constexpr (BITS == 2) {
        out[0] = o[0];
      } else if constexpr (BITS == 4) {   // wq may be only 4-byte aligned
        if ((reinterpret_cast<uintptr_t>(wq) & 7) == 0) *reinterpret_cast<uint2*>(out) = make_uint2(o[0], o[1]);
        else { out[0] = o[0]; out[1] = o[1]; }
      } else if constexpr (BITS == 8) {
        if ((reinterpret_cast<uintptr_t>(wq) & 15) == 0) *reinterpret_cast<uint4*>(out) = make_uint4(o[0], o[1], o[2], o[3]);
        else { out[0] = o[0]; out[1] = o[1]; out[2] = o[2]; out[3] = o[3]; }
      } else {
        out[0] = o[0]; out[1] = o[1]; out[2] = o[2];
      }
    }
  }
}

// ---------------------------------------------------------------------------- dequantize
// The 8 fields of chunk c: they start at byte c*BITS, at byte offset 0..3 of a word, and for every supported
// width end within 64 bits from there.
template <int BITS>
__device__ __forceinline__ uint2 chunk_bits(const uint32_t* __restrict__ wq, int64_t c, int64_t n_words) {
  if constexpr (BITS == 4) return make_uint2(__ldg(wq + c), 0u);
  const int64_t byte = c * BITS, w0 = byte >> 2;
  const int sh = (int)(byte & 3) * 8;
  const uint32_t a = __ldg(wq + w0);
  const uint32_t b = (w0 + 1 < n_words) ? __ldg(wq + w0 + 1) : 0u;
  if constexpr (BITS == 8) return make_uint2(a, b);
  return make_uint2(__funnelshift_r(a, b, sh), b >> sh);
}

// Values of a chunk: round_T(round_T(q * s) + b), multiply and add being separate operations of type T in the
// reference.  16-bit types in packed pairs: q comes out of the bit pattern 128 + q (bf16) or 1024 + q (f16) exactly;
// mul.rn and add.rn on pairs round as the fp32 operation followed by the conversion does (the fp32 product is
// exact, and so is every fp32 sum that could land between two values of T).
template <typename T, int BITS>
__device__ __forceinline__ void store_chunk(T* __restrict__ dst, uint2 bits, T s_t, T b_t) {
  if constexpr (sizeof(T) == 4) {
    const uint64_t v64 = (uint64_t)bits.y << 32 | bits.x;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __fadd_rn(__fmul_rn((float)(uint32_t)((v64 >> (i * BITS)) & ((1u << BITS) - 1u)), s_t), b_t);
    store8(dst, v);
  } else {
    constexpr bool kBf = std::is_same<T, __nv_bfloat16>::value;
    using T2 = typename std::conditional<kBf, __nv_bfloat162, __half2>::type;
    constexpr uint32_t kMask = (1u << BITS) - 1u;
    constexpr uint32_t kOff = kBf ? 0x43004300u : 0x64006400u;   // (128, 128) or (1024, 1024)
    T2 s2, b2;
    s2.x = s2.y = s_t;
    b2.x = b2.y = b_t;
    uint32_t q[4];   // fields (2i, 2i+1)
    if constexpr (kBf && BITS == 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t w = i < 2 ? bits.x : bits.y;
        const float f0 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 | (2 * i & 3))) - 8388608.0f;
        const float f1 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 | ((2 * i + 1) & 3))) - 8388608.0f;
        const __nv_bfloat162 t = __floats2bfloat162_rn(f0, f1);
        q[i] = *reinterpret_cast<const uint32_t*>(&t);
      }
    } else {
      uint32_t m[4];
      if constexpr (BITS == 4 || BITS == 2) {   // masks over both halves: fields (i, i + 4)
        const uint32_t w = BITS == 4 ? bits.x : __byte_perm(bits.x, 0u, 0x4140);
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = ((w >> (BITS * i)) & (kMask * 0x00010001u)) | kOff;
        q[0] = __byte_perm(m[0], m[1], 0x5410); q[1] = __byte_perm(m[2], m[3], 0x5410);
        q[2] = __byte_perm(m[0], m[1], 0x7632); q[3] = __byte_perm(m[2], m[3], 0x7632);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t f[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int at = (2 * i + h) * BITS;
            f[h] = ((at >= 32 ? bits.y >> (at - 32) : (at + BITS > 32 ? __funnelshift_r(bits.x, bits.y, at) : bits.x >> at)) & kMask);
          }
          q[i] = (f[0] | f[1] << 16) | kOff;
        }
      }
      T2 off;
      *reinterpret_cast<uint32_t*>(&off) = kOff;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const T2 t = __hsub2(*reinterpret_cast<const T2*>(&q[i]), off);
        q[i] = *reinterpret_cast<const uint32_t*>(&t);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const T2 t = __hadd2_rn(__hmul2_rn(*reinterpret_cast<const T2*>(&q[i]), s2), b2);   // (_rn: never contracted to one fma)
      q[i] = *reinterpret_cast<const uint32_t*>(&t);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(q[0], q[1], q[2], q[3]);
  }
}

// CHUNKS chunks of 8 values per thread, a block apart: four keep enough loads in flight for HBM.  28672 x 8192 bf16,
// groups of 64: from 4 bits 134 -> 99 us (6.1 TB/s), from 3 bits 138 -> 111.  One up to 2^22 values (f32: 2^23), where one
// thread's chain takes the time (four / one, us: 256 x 1024 f16 from 3 bits 2.2 / 1.5, f32 3.0 / 1.8; 2048 x 2048 4.0 / 3.2;
// 2048 x 4096 f16 5.7 / 5.5, from 4 bits 5.0 / 5.6, f32 12.7 / 11.6).
constexpr int kDequantChunks = 4;

template <typename T, int BITS, int CHUNKS>
__global__ void __launch_bounds__(256)
dequantize_kernel(const uint32_t* __restrict__ wq, const T* __restrict__ scales,
                  const T* __restrict__ biases, T* __restrict__ out, int64_t n_chunks,
                  int group_shift /* log2(group/8) */, int64_t n_words) {
  const int64_t c0 = (int64_t)blockIdx.x * (256 * CHUNKS) + threadIdx.x;
  uint2 bits[CHUNKS];
  T s[CHUNKS], b[CHUNKS];
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int64_t c = c0 + 256 * i;
    if (c < n_chunks) {
      bits[i] = chunk_bits<BITS>(wq, c, n_words);
      s[i] = scales[c >> group_shift];
      b[i] = biases[c >> group_shift];
    }
  }
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int64_t c = c0 + 256 * i;
    if (c < n_chunks) store_chunk<T, BITS>(out + c * 8, bits[i], s[i], b[i]);
  }
}

template <typename T>
int launch_quantize(const T* w, int64_t n_elems, int group, int bits, uint32_t* wq, T* s, T* b,
                    cudaStream_t st) {
  if (n_elems == 0) return B200Q_OK;
  bool done = false;
  B200Q_DISPATCH_BITS(bits, BITS, {
    auto go = [&](auto gtag, auto small) {
      constexpr int G = decltype(gtag)::value;
      constexpr int64_t per_block = 8 * QuantShape<G, small>::kIter * 512;
      quantize_kernel<T, BITS, G, small><<<(unsigned)((n_elems + per_block - 1) / per_block), 256, 0, st>>>(w, wq, s, b, n_elems);
    };
    auto pick = [&](auto small) {
      if (group == 64) go(std::integral_constant<int, 64>{}, small);
      else go(std::integral_constant<int, 128>{}, small);
    };
    if (group == 32) go(std::integral_constant<int, 32>{}, std::false_type{});
    else if (n_elems <= kSmall) pick(std::true_type{});
    else pick(std::false_type{});
    done = true;
  });
  if (!done) return fail(B200Q_ERR_INVALID_ARGUMENT, "[quantize] unsupported bits %d", bits);
  B200Q_LAUNCH_OK("quantize_kernel");
  return B200Q_OK;
}

template <typename T>
int launch_dequantize(const uint32_t* wq, const T* s, const T* b, int64_t n_elems, int group,
                      int bits, T* out, cudaStream_t st) {
  const int64_t n_chunks = n_elems / 8;
  if (n_chunks == 0) return B200Q_OK;
  const bool small = n_elems <= (sizeof(T) == 4 ? 2 : 1) * kSmall;
  const int64_t per_block = 256 * (small ? 1 : kDequantChunks);
  const unsigned grid = (unsigned)((n_chunks + per_block - 1) / per_block);
  const int gshift = group == 32 ? 2 : (group == 64 ? 3 : 4);
  const int64_t n_words = n_elems * bits / 32;
  bool done = false;
  B200Q_DISPATCH_BITS(bits, BITS, {
    if (small) dequantize_kernel<T, BITS, 1><<<grid, 256, 0, st>>>(wq, s, b, out, n_chunks, gshift, n_words);
    else dequantize_kernel<T, BITS, kDequantChunks><<<grid, 256, 0, st>>>(wq, s, b, out, n_chunks, gshift, n_words);
    done = true;
  });
  if (!done) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize] unsupported bits %d", bits);
  B200Q_LAUNCH_OK("dequantize_kernel");
  return B200Q_OK;
}

// Rows of the packed matrix chosen by `ids` (an embedding look-up): out[i, :] = dequantize(row ids[i]).
// An id outside [0, rows) gives a row of zeros; nothing is read for it.
template <typename T, int BITS>
__global__ void __launch_bounds__(256)
dequantize_rows_kernel(const uint32_t* __restrict__ wq, const T* __restrict__ scales,
                       const T* __restrict__ biases, const uint32_t* __restrict__ ids, T* __restrict__ out,
                       int64_t rows, int chunks_per_row, int group_shift, int64_t n_words) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= chunks_per_row) return;
  const int64_t i = blockIdx.y;
  const uint32_t id = __ldg(ids + i);
  T* dst = out + (i * chunks_per_row + c) * 8;
  if ((int64_t)id >= rows) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
    store8(dst, v);
    return;
  }
  const int64_t cg = (int64_t)id * chunks_per_row + c;  // chunk index in the whole matrix
  const int64_t g = cg >> group_shift;
  store_chunk<T, BITS>(dst, chunk_bits<BITS>(wq, cg, n_words), scales[g], biases[g]);
}

template <typename T>
int launch_dequantize_rows(const uint32_t* wq, const T* s, const T* b, const uint32_t* ids, int64_t n_ids,
                           int64_t rows, int64_t K, int group, int bits, T* out, cudaStream_t st) {
  const int cpr = (int)(K / 8);
  const int gshift = group == 32 ? 2 : (group == 64 ? 3 : 4);
  const int64_t n_words = rows * K * bits / 32;
  bool done = false;
  for (int64_t i0 = 0; i0 < n_ids; i0 += 65535) {   // gridDim.y limit
    const unsigned ny = (unsigned)((n_ids - i0) < 65535 ? (n_ids - i0) : 65535);
    dim3 grid((unsigned)((cpr + 255) / 256), ny);
    B200Q_DISPATCH_BITS(bits, BITS, {
      dequantize_rows_kernel<T, BITS><<<grid, 256, 0, st>>>(wq, s, b, ids + i0, out + i0 * K, rows, cpr, gshift, n_words);
      done = true;
    });
    if (!done) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize_rows] unsupported bits %d", bits);
    B200Q_LAUNCH_OK("dequantize_rows_kernel");
  }
  return B200Q_OK;
}

int check_quant_args(const char* tag, int dtype, int64_t rows, int64_t K, int group, int bits) {
  if (dtype != B200Q_F32 && dtype != B200Q_F16 && dtype != B200Q_BF16)
    return fail(B200Q_ERR_INVALID_ARGUMENT, "[%s] Only real floating types are supported (dtype code %d).", tag, dtype);
  if (!valid_group(group))
    return fail(B200Q_ERR_INVALID_ARGUMENT,
                "[%s] The requested group size %d is not supported. The supported group sizes are 32, 64, and 128.", tag, group);
  if (!valid_bits(bits))
    return fail(B200Q_ERR_INVALID_ARGUMENT,
                "[%s] The requested number of bits %d is not supported. The supported bits are 2, 3, 4, 5, 6 and 8.", tag, bits);
  if (rows < 0 || K < 0)
    return fail(B200Q_ERR_INVALID_ARGUMENT, "[%s] negative shape (%lld, %lld).", tag, (long long)rows, (long long)K);
  if (K % group != 0)
    return fail(B200Q_ERR_INVALID_ARGUMENT,
                "[%s] The last dimension of the matrix needs to be divisible by the quantization group size %d. "
                "However the provided matrix has shape (%lld, %lld)", tag, group, (long long)rows, (long long)K);
  return B200Q_OK;
}

}  // namespace
}  // namespace b200q

using namespace b200q;

extern "C" int b200q_quantize(const void* w, int dtype, int64_t rows, int64_t K, int group_size,
                              int bits, uint32_t* wq, void* scales, void* biases, void* stream) {
  if (int rc = check_quant_args("quantize", dtype, rows, K, group_size, bits)) return rc;
  const int64_t n = rows * K;
  if (n == 0) return B200Q_OK;
  if (!w || !wq || !scales || !biases) return fail(B200Q_ERR_INVALID_ARGUMENT, "[quantize] null pointer");
  if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(wq) & 3))
    return fail(B200Q_ERR_INVALID_ARGUMENT, "[quantize] w must be 16-byte aligned and wq 4-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_F32:
      return launch_quantize<float>((const float*)w, n, group_size, bits, wq, (float*)scales, (float*)biases, st);
    case B200Q_F16:
      return launch_quantize<__half>((const __half*)w, n, group_size, bits, wq, (__half*)scales, (__half*)biases, st);
    default:
      return launch_quantize<__nv_bfloat16>((const __nv_bfloat16*)w, n, group_size, bits, wq,
                                            (__nv_bfloat16*)scales, (__nv_bfloat16*)biases, st);
  }
}

extern "C" int b200q_dequantize(const uint32_t* wq, const void* scales, const void* biases, int dtype,
                                int64_t rows, int64_t K, int group_size, int bits, void* out,
                                void* stream) {
  if (int rc = check_quant_args("dequantize", dtype, rows, K, group_size, bits)) return rc;
  const int64_t n = rows * K;
  if (n == 0) return B200Q_OK;
  if (!wq || !scales || !biases || !out) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize] null pointer");
  if ((reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(wq) & 3))
    return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize] out must be 16-byte aligned and wq 4-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_F32:
      return launch_dequantize<float>(wq, (const float*)scales, (const float*)biases, n, group_size, bits, (float*)out, st);
    case B200Q_F16:
      return launch_dequantize<__half>(wq, (const __half*)scales, (const __half*)biases, n, group_size, bits, (__half*)out, st);
    default:
      return launch_dequantize<__nv_bfloat16>(wq, (const __nv_bfloat16*)scales, (const __nv_bfloat16*)biases, n,
                                              group_size, bits, (__nv_bfloat16*)out, st);
  }
}

extern "C" int b200q_dequantize_rows(const uint32_t* wq, const void* scales, const void* biases, const uint32_t* ids,
                                     int64_t n_ids, int dtype, int64_t rows, int64_t K, int group_size, int bits,
                                     void* out, void* stream) {
  if (int rc = check_quant_args("dequantize_rows", dtype, rows, K, group_size, bits)) return rc;
  if (n_ids < 0) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize_rows] negative number of ids (%lld).", (long long)n_ids);
  if (K / 8 > INT32_MAX) return fail(B200Q_ERR_UNSUPPORTED, "[dequantize_rows] row too long.");
  if (n_ids == 0 || K == 0) return B200Q_OK;
  if (!out || !ids) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize_rows] null pointer");
  if (rows > 0 && (!wq || !scales || !biases)) return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize_rows] null pointer");
  if ((reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(wq) & 3))
    return fail(B200Q_ERR_INVALID_ARGUMENT, "[dequantize_rows] out must be 16-byte aligned and wq 4-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_F32:
      return launch_dequantize_rows<float>(wq, (const float*)scales, (const float*)biases, ids, n_ids, rows, K, group_size,
                                           bits, (float*)out, st);
    case B200Q_F16:
      return launch_dequantize_rows<__half>(wq, (const __half*)scales, (const __half*)biases, ids, n_ids, rows, K,
                                            group_size, bits, (__half*)out, st);
    default:
      return launch_dequantize_rows<__nv_bfloat16>(wq, (const __nv_bfloat16*)scales, (const __nv_bfloat16*)biases, ids,
                                                   n_ids, rows, K, group_size, bits, (__nv_bfloat16*)out, st);
  }
}
