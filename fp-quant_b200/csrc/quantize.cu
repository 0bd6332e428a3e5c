// Fused block-Hadamard rotation + micro-scaled FP4 quantisation (MXFP4 / NVFP4) for sm_100a.
//
// One thread owns 32 contiguous elements of a row (64 B of bf16 = two 128-bit loads, one
// 256-bit load on sm_100).  Butterfly stages with pair distance <= 16 run in registers, the
// stages for distance 32 and 64 exchange registers with the neighbouring lanes by warp
// shuffle.  All rotation arithmetic is IEEE fp32 add/sub/mul in a fixed order (distances
// 1,2,4,..,g/2, then one multiply by fl32(1/sqrt(g))) so that a CPU can reproduce it bit
// for bit.  The scale chain and the division that precedes E2M1 rounding reproduce the
// fp32 operation sequence of the reference Quantizer (src/quantization/quantizer.py:107-168,
// src/quantization/quant_ops.py:57-94 of IST-DASLab/FP-Quant).
//
// The kernel is HBM-bound: 2 B read + 0.5 B codes + 1/g B scale per element.

#include "common.cuh"

namespace fpq {
namespace {

// MODE_ROTATE_MASK: the input is multiplied by a packed 0/1 mask on its way into the rotation (the backward of a
// clipping quantiser: mask the gradient, then rotate it back).
enum Mode { MODE_CODES = 0, MODE_DEQUANT = 1, MODE_ROTATE = 2, MODE_ABSMAX = 3, MODE_ROTATE_MASK = 4 };

struct QuantParams {
  const void* x;
  int64_t n_chunks;     // rows * cols / 32
  uint32_t chunks_per_row;
  uint64_t row_magic;   // ceil(2^64 / chunks_per_row) (0 when chunks_per_row == 1): chunk -> row by one multiply
  uint8_t* codes;       // [rows, cols/2]
  uint8_t* sbytes;      // scale bytes
  float* sf32;          // fp32 scales, row-major
  int32_t* nan_flag;    // set when one of them is NaN
  void* y;              // dequantised / rotated output
  const float* gs;      // NVFP4 tensor scale
  uint32_t* absmax_bits;
  uint8_t* mask;        // QuEST clip mask: one bit per element (codes) or one byte per element (dequantised output)
  const uint32_t* mask_in;   // MODE_ROTATE_MASK: one word per chunk, bit i = element i counts
  uint32_t sf_tiles_per_row_block;  // ceil((cols/g)/4)
  uint32_t rows, pad_rows;          // swizzled scale layout: rows of the tensor and rows up to the next multiple of 128
  int layout;
  int out_bf16;
  int ste;
};

typedef unsigned long long u64;

__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(u64 p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// 32 contiguous elements of a row as they lie in memory: sixteen 32-bit words of bf16 pairs, or
// sixteen 64-bit words of fp32 pairs (element 2j in the low half of word j).
template <bool IN_BF16> struct RawChunk;
template <> struct RawChunk<true> { uint32_t w[16]; };
template <> struct RawChunk<false> { u64 w[16]; };

__device__ __forceinline__ void load_raw(const void* base, int64_t chunk, bool active, RawChunk<true>& r) {
  if (active) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(base) + chunk * 16;
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]),
                   "=r"(r.w[6]), "=r"(r.w[7])
                 : "l"(p));
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[8]), "=r"(r.w[9]), "=r"(r.w[10]), "=r"(r.w[11]), "=r"(r.w[12]), "=r"(r.w[13]),
                   "=r"(r.w[14]), "=r"(r.w[15])
                 : "l"(p + 8));
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) r.w[j] = 0;
  }
}
__device__ __forceinline__ void load_raw(const void* base, int64_t chunk, bool active, RawChunk<false>& r) {
  if (active) {
    const u64* p = reinterpret_cast<const u64*>(base) + chunk * 16;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      asm volatile("ld.global.nc.L1::no_allocate.v4.b64 {%0,%1,%2,%3}, [%4];"
                   : "=l"(r.w[4 * q]), "=l"(r.w[4 * q + 1]), "=l"(r.w[4 * q + 2]), "=l"(r.w[4 * q + 3])
                   : "l"(p + 4 * q));
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) r.w[j] = 0ull;
  }
}

#ifndef FPQ_Q_UNPACK
#define FPQ_Q_UNPACK 0      // 1: bf16 -> fp32 with cvt instead of shift / mask (measured: see the profile notes)
#endif
#ifndef FPQ_Q_MAX3
#define FPQ_Q_MAX3 1
#endif

// Raw words -> fp32 pairs.  With STAGE1 the first butterfly stage (distance 1: the two elements
// of a pair become their sum and difference) is applied on the way.
template <bool STAGE1>
__device__ __forceinline__ void unpack_chunk(const RawChunk<true>& r, u64 (&P)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
#if FPQ_Q_UNPACK == 1
    uint16_t l16, h16;
    float a, b;
    asm("mov.b32 {%0, %1}, %2;" : "=h"(l16), "=h"(h16) : "r"(r.w[j]));
    asm("cvt.f32.bf16 %0, %1;" : "=f"(a) : "h"(l16));
    asm("cvt.f32.bf16 %0, %1;" : "=f"(b) : "h"(h16));
#else
    const float a = __uint_as_float(r.w[j] << 16), b = __uint_as_float(r.w[j] & 0xffff0000u);
#endif
    P[j] = STAGE1 ? pack2(__fadd_rn(a, b), __fsub_rn(a, b)) : pack2(a, b);
  }
}
template <bool STAGE1>
__device__ __forceinline__ void unpack_chunk(const RawChunk<false>& r, u64 (&P)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (STAGE1) {
      float a, b;
      unpack2(r.w[j], a, b);
      P[j] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
    } else {
      P[j] = r.w[j];
    }
  }
}

// The first butterfly stage on pairs that unpack_chunk<false> left as they were.
__device__ __forceinline__ void stage1_chunk(u64 (&P)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float a, b;
    unpack2(P[j], a, b);
    P[j] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
  }
}

// P *= the chunk's mask bits as 0.0 / 1.0.  A product and no selection: what is not finite stays visible under a
// zero bit (inf * 0 = NaN), as in the unfused elementwise multiply.
__device__ __forceinline__ void mask_chunk(u64 (&P)[16], uint32_t bits) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float lo = __uint_as_float((bits >> (2 * j)) & 1u ? 0x3f800000u : 0u);
    const float hi = __uint_as_float((bits >> (2 * j + 1)) & 1u ? 0x3f800000u : 0u);
    P[j] = mul2(P[j], pack2(lo, hi));
  }
}

// Butterfly stages with pair distance 1..min(GH,32)/2 inside the thread, then the
// cross-lane stages for distance 32 (GH >= 64) and 64 (GH == 128), then * 1/sqrt(GH).
template <int GH>
__device__ __forceinline__ constexpr float hadamard_scale() {
  return GH == 16 ? 0.25f : GH == 32 ? 0.17677669529663687f : GH == 64 ? 0.125f : GH == 128 ? 0.08838834764831845f : 1.0f;
}

template <int GH, bool SCALE = true>
__device__ __forceinline__ void rotate_chunk(u64 (&P)[16], int lane) {
  // distance 1 (inside each packed pair) was applied by unpack_chunk<true>
  // distances 2, 4, 8, 16 <-> pair index distance 1, 2, 4, 8
#pragma unroll
  for (int d = 1; d < 16; d <<= 1) {
    if (GH != 0 && 2 * d < (GH < 32 ? GH : 32)) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if ((j & d) == 0) {
          u64 a = P[j], b = P[j + d];
          P[j] = add2(a, b);
          P[j + d] = sub2(a, b);
        }
      }
    }
  }
  if (GH >= 64) {
#pragma unroll
    for (int bit = 1; bit < GH / 32; bit <<= 1) {
      const float sgn = (lane & bit) ? -1.0f : 1.0f;
      const u64 S = pack2(sgn, sgn);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        u64 other = __shfl_xor_sync(0xffffffffu, P[j], bit);
        P[j] = fma2(S, P[j], other);  // bit clear: own + other, bit set: other - own
      }
    }
  }
  if (SCALE && GH != 0) {
    const float c = hadamard_scale<GH>();
    const u64 C = pack2(c, c);
#pragma unroll
    for (int j = 0; j < 16; ++j) P[j] = mul2(P[j], C);
  }
}

__device__ __forceinline__ u64 mul2_rz(u64 a, u64 b) {
  u64 r;
  asm("mul.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// MXFP4 shortcut.  With s = fl(4/3) * 2^(e-2) the E2M1 code of fl(fl(t*c) / s) -- t the unscaled
// butterfly output, c = 1/sqrt(g) -- equals the code of ONE rounded product t * (m * 2^(2-e)):
//   c a power of two (g = 16, 64, or no rotation): m = 0.75 * c, product rounded toward zero;
//   g = 32, 128:                                   m = fl(c / fl(4/3)), product rounded to nearest.
// Both were checked against the two-step form on every fp32 input within 20000 ulps of each of the
// seven rounding boundaries (and on random inputs); away from the boundaries the two values differ
// by a few ulps at most, which cannot change the code.
template <int GH>
__device__ __forceinline__ u64 mx_code_multiplier(int e) {
  constexpr bool POW2 = GH == 0 || GH == 16 || GH == 64;
  constexpr uint32_t mbits = GH == 0 ? 0x3f400000u : GH == 16 ? 0x3e400000u : GH == 64 ? 0x3dc00000u
                           : GH == 32 ? 0x3e07c3b6u : 0x3d87c3b6u;
  (void)POW2;
  const float m = __uint_as_float(mbits + ((uint32_t)(2 - e) << 23));   // exact scaling by 2^(2-e)
  return pack2(m, m);
}

__device__ __forceinline__ float absmax_pairs(const u64* P, int n) {
  float m = 0.0f;
#pragma unroll
  for (int j = 0; j < n; ++j) {
    float a, b;
    unpack2(P[j], a, b);
#if FPQ_Q_MAX3
    asm("max.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(a)), "f"(fabsf(b)));
#else
    m = fmaxf(m, fmaxf(fabsf(a), fabsf(b)));
#endif
  }
  return m;
}

// floor(fl32(log2(m))) as torch's fp32 log2 yields it: the exponent field, plus one when m is
// so close below a power of two that the correctly rounded fp32 logarithm is that integer.
__device__ __forceinline__ int mx_exponent(float m /* >= 2^-126, finite */) {
  uint32_t b = __float_as_uint(m);
  int e = (int)(b >> 23) - 127;
  if ((b & 0x7fffffu) >= 0x7fff00u) {
    float l = (float)log2((double)m);
    e = (int)floorf(l);
  }
  return max(-127, min(127, e));
}

// MXFP4 scale of one 32-element group: returns the divisor s and the stored byte.
// The reference computes e = floor(log2(m)) with m = fl(6 * fl(fl(2a) / 12)), which lies within
// two ulps of a.  When a's mantissa is at least four ulps away from both ends of its binade (and
// from the 0x7fff00 threshold of the logarithm's rounding artefact) m has a's exponent, so the
// division chain is only evaluated for the rare group maxima near a power of two.
__device__ __forceinline__ float mx_scale(float a, uint32_t& byte, int& e) {
  const uint32_t bits = __float_as_uint(a);
  const uint32_t mant = bits & 0x7fffffu, ex = bits >> 23;   // a >= 0
  if (mant - 4u <= 0x7ffef7u && ex - 8u <= 239u) {           // mant in [4, 0x7ffefb], ex in [8, 247]
    e = (int)ex - 127;
    byte = ex;
    return __uint_as_float(((ex - 2u) << 23) | 0x2aaaabu);
  }
  float s0 = __fdiv_rn(__fmul_rn(2.0f, a), 12.0f);
  float m = fmaxf(__fmul_rn(6.0f, s0), 1.17549435e-38f);
  e = mx_exponent(m);
  byte = (uint32_t)(e + 127);
  float s;
  if (e >= -124) {
    // fl(2^(e-2) / 0.75) = 2^(e-2) * fl(4/3): exponent field e-2+127, mantissa of fl(4/3)
    s = __uint_as_float(((uint32_t)(e + 125) << 23) | 0x2aaaabu);
  } else {
    s = __fdiv_rn(ldexpf(1.0f, e - 2), 0.75f);  // subnormal power of two
    if (s == 0.0f) s = 1.0f;
  }
  return s;
}

// Third value of the FMT template parameter (not part of the C ABI's format numbers): MXFP4 codes and
// E8M0 scale bytes with the QuEST scale rule instead of the group maximum.
constexpr int FMT_MXQUEST = 2;

// QuEST scale of one 32-element group (inference_lib/src/fp_quant/module/triton/mxfp4.py:51-59):
// std = sqrt(mean(x^2) - mean(x)^2), scale = fl(fl(c * std) + 1e-8) with c = fl32(2.92247856 / 6)
// (pseudoquant_linear_fns.py:20), divisor 2^floor(log2(scale)), stored byte = that exponent + 127.
// The sums run over the sixteen register pairs in order, even and odd elements separately (one packed
// add per pair), then even + odd; squares are rounded products (no fused multiply-add), so a CPU
// reproduces every bit.  A variance that rounds below zero counts as zero.  scale >= 1e-8 is a normal
// number, so the exponent field is floor(log2(scale)) exactly.
__device__ __forceinline__ float quest_scale(const u64* P, uint32_t& byte) {
  u64 acc = P[0], acc2 = mul2(P[0], P[0]);
#pragma unroll
  for (int j = 1; j < 16; ++j) {
    acc = add2(acc, P[j]);
    acc2 = add2(acc2, mul2(P[j], P[j]));
  }
  float a0, a1, q0, q1;
  unpack2(acc, a0, a1);
  unpack2(acc2, q0, q1);
  const float mean = __fmul_rn(__fadd_rn(a0, a1), 0.03125f);
  const float mean_sq = __fmul_rn(__fadd_rn(q0, q1), 0.03125f);
  const float var = fmaxf(__fsub_rn(mean_sq, __fmul_rn(mean, mean)), 0.0f);
  const float scale = __fadd_rn(__fmul_rn(0.48707976f, __fsqrt_rn(var)), 1e-8f);
  byte = (__float_as_uint(scale) >> 23) & 0xffu;
  return __uint_as_float(byte << 23);
}

// NVFP4 scale of one 16-element group.
__device__ __forceinline__ float nv_scale(float a, float gs, float rgs, uint32_t& byte) {
  // s0 = fl(fl(2a) / 12) = fl(a / 3) / 2.  With r = fl(1/3), q = fl(a r), e = a - 3 q (exact, fused) the
  // value fl(q + e r) is the correctly rounded a / 3 for every fp32 mantissa (checked exhaustively on the
  // CPU); halving is exact while nothing underflows, so the general division is kept for the extremes.
  float s0;
  if (a > 7.8886e-31f /* 2^-100 */ && a < 1.3292e36f /* 2^120 */) {
    const float r = 0.333333343f;             // 0x3eaaaaab
    float q = __fmul_rn(a, r);
    const float e = __fmaf_rn(-3.0f, q, a);
    q = __fmaf_rn(e, r, q);
    s0 = 0.5f * q;
  } else {
    s0 = __fdiv_rn(__fmul_rn(2.0f, a), 12.0f);
  }
  float t = fminf(fmaxf(__fmul_rn(s0, gs), -448.0f), 448.0f);
  uint16_t u2;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(u2) : "f"(0.0f), "f"(t));
  uint32_t u = u2 & 0xffu;
  // decode the (non-negative) E4M3 byte exactly: (8+m) * 2^(e-10), or m * 2^-9 when e == 0
  uint32_t ex = u >> 3, ma = u & 7u;
  float uf = ex == 0 ? (float)ma * 0.001953125f : __uint_as_float(((ex + 120u) << 23) | (ma << 20));
  float s = __fmul_rn(uf, rgs);
  byte = u;
  return s == 0.0f ? 1.0f : s;
}

// Correctly rounded y / s for the pairs P[0..n): reciprocal once per group, then the classic
// multiply + two fused residual corrections, two elements per instruction.  Falls back to
// per-element IEEE division when s is so small or large that the reciprocal or a residual
// could leave the normal range.
__device__ __forceinline__ void divide_pairs(u64* P, int n, float s) {
  const float as = fabsf(s);
  if (as > 7.8886e-31f /* 2^-100 */ && as < 1.2676e30f /* 2^100 */) {
    const float r = __frcp_rn(s);
    const u64 R = pack2(r, r), NS = pack2(-s, -s);
#pragma unroll
    for (int j = 0; j < n; ++j) {
      u64 y = P[j];
      u64 q = mul2(y, R);
      u64 e = fma2(q, NS, y);
      q = fma2(e, R, q);
      e = fma2(q, NS, y);
      P[j] = fma2(e, R, q);
    }
  } else {
#pragma unroll
    for (int j = 0; j < n; ++j) {
      float a, b;
      unpack2(P[j], a, b);
      P[j] = pack2(__fdiv_rn(a, s), __fdiv_rn(b, s));
    }
  }
}

// Eight quotients (4 pairs) -> one word of eight 4-bit codes, element 0 in the lowest nibble.
#ifndef FPQ_Q_PACKMOV
#define FPQ_Q_PACKMOV 1
#endif
__device__ __forceinline__ uint32_t codes_word(const u64* P) {
  uint32_t w = 0;
#if FPQ_Q_PACKMOV
  float a0, b0, a1, b1, a2, b2, a3, b3;
  unpack2(P[0], a0, b0);
  unpack2(P[1], a1, b1);
  unpack2(P[2], a2, b2);
  unpack2(P[3], a3, b3);
  asm("{ .reg .b8 t0, t1, t2, t3;\n"
      "  cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n"
      "  cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n"
      "  cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n"
      "  cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n"
      "  mov.b32 %0, {t0, t1, t2, t3}; }"
      : "=r"(w)
      : "f"(a0), "f"(b0), "f"(a1), "f"(b1), "f"(a2), "f"(b2), "f"(a3), "f"(b3));
#else
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    unpack2(P[j], a, b);
    uint32_t byte;
    asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u32.u8 %0, t; }"
        : "=r"(byte)
        : "f"(b), "f"(a));
    w |= byte << (8 * j);
  }
#endif
  return patch_zero_codes(w);
}

__device__ __forceinline__ size_t swizzled_offset(uint32_t row, uint32_t sfc, uint32_t tiles_per_row_block) {
  return ((size_t)(row >> 7) * tiles_per_row_block + (sfc >> 2)) * 512u + (row & 31u) * 16u +
         ((row >> 5) & 3u) * 4u + (sfc & 3u);
}

// chunk index -> (row, chunk in row).  One 64 x 64 -> high 64 multiply: with M = ceil(2^64 / d)
// the quotient floor(c * M / 2^64) is exact whenever c * (M d - 2^64) < 2^64, which holds for
// c, d < 2^32.  Larger chunk counts take the division.
__device__ __forceinline__ void chunk_row(const QuantParams& p, int64_t c, uint32_t& row, uint32_t& cir) {
  if (p.chunks_per_row == 1) {
    row = (uint32_t)c;
    cir = 0;
  } else if (p.row_magic) {
    row = (uint32_t)__umul64hi((u64)c, p.row_magic);
    cir = (uint32_t)c - row * p.chunks_per_row;
  } else {
    row = (uint32_t)(c / p.chunks_per_row);
    cir = (uint32_t)(c - (int64_t)row * p.chunks_per_row);
  }
}

// Where a caller wants the chunk's codes and scale byte instead of having them stored.
struct ChunkOut {
  uint32_t cw[4];
  uint32_t sb;
};

// Everything that happens to one chunk of 32 elements after its load.
template <int GH, int FMT, bool IN_BF16, int MODE>
__device__ __forceinline__ void process_chunk(const QuantParams& p, const RawChunk<IN_BF16>& raw, int64_t c,
                                              bool active, int lane, float gs, float rgs, float& running_max,
                                              uint32_t mask_bits = 0, ChunkOut* keep = nullptr) {
    u64 P[16];
    if (MODE == MODE_ROTATE_MASK) {
      unpack_chunk<false>(raw, P);
      mask_chunk(P, mask_bits);
      if (GH != 0) stage1_chunk(P);
    } else {
      unpack_chunk<GH != 0>(raw, P);
    }
    // MXFP4 codes take the unscaled butterfly output (the 1/sqrt(g) factor is folded into the
    // code multiplier); every other mode works on the scaled rotation.
    constexpr bool MX_FAST = MODE == MODE_CODES && FMT == FPQ_FMT_MXFP4;
    // NVFP4 codes with a rotation whose 1/sqrt(g) is a power of two (g = 16, 64): the factor c goes into the
    // divisor instead, t / (s / c) = (t c) / s exactly, which saves the sixteen scaling multiplies.
    constexpr bool NV_FOLD = MODE == MODE_CODES && FMT == FPQ_FMT_NVFP4 && (GH == 16 || GH == 64);
    rotate_chunk<GH, !(MX_FAST || NV_FOLD)>(P, lane);

    if (MODE == MODE_ABSMAX) {
      running_max = fmaxf(running_max, absmax_pairs(P, 16));
      return;
    }
    if (MODE == MODE_ROTATE || MODE == MODE_ROTATE_MASK) {
      if (active) {
        if (p.out_bf16) {
          uint4* o = reinterpret_cast<uint4*>(p.y) + c * 4;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float a, b;
              unpack2(P[4 * q + j], a, b);
              __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
              w[j] = *reinterpret_cast<uint32_t*>(&h);
            }
            o[q] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        } else {
          ulonglong2* o = reinterpret_cast<ulonglong2*>(p.y) + c * 8;
#pragma unroll
          for (int q = 0; q < 8; ++q) o[q] = make_ulonglong2(P[2 * q], P[2 * q + 1]);
        }
      }
      return;
    }

    // ---- scales
    constexpr int NG = FMT == FPQ_FMT_NVFP4 ? 2 : 1;  // groups per thread
    constexpr int PG = 16 / NG;                       // pairs per group
    float s[NG];
    float amax_g[NG];
    uint32_t sb[NG];
    int mx_e = 0;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      if (FMT == FMT_MXQUEST) break;
      float a = absmax_pairs(P + g * PG, PG);
      if ((MX_FAST || NV_FOLD) && GH != 0) a = __fmul_rn(a, hadamard_scale<GH>());   // max |t*c| = fl(c * max |t|)
      if (NV_FOLD) amax_g[g] = a;
      s[g] = FMT == FPQ_FMT_NVFP4 ? nv_scale(a, gs, rgs, sb[g]) : mx_scale(a, sb[g], mx_e);
    }
    if (FMT == FMT_MXQUEST) s[0] = quest_scale(P, sb[0]);
    if (MODE == MODE_CODES && keep) keep->sb = sb[0];
    if (MODE == MODE_CODES && active && !keep) {
      if (p.sbytes) {
        size_t off = (size_t)c * NG;
        if (p.layout == FPQ_SCALES_SWIZZLED) {
          uint32_t row, cir;
          chunk_row(p, c, row, cir);
          off = swizzled_offset(row, cir * NG, p.sf_tiles_per_row_block);
        }
        if (NG == 2)
          *reinterpret_cast<uint16_t*>(p.sbytes + off) = (uint16_t)(sb[0] | (sb[NG - 1] << 8));
        else
          p.sbytes[off] = (uint8_t)sb[0];
      }
      if (p.sf32) {
        if (NG == 2)
          *reinterpret_cast<float2*>(p.sf32 + c * 2) = make_float2(s[0], s[NG - 1]);
        else
          p.sf32[c] = s[0];
        if (p.nan_flag && (s[0] != s[0] || s[NG - 1] != s[NG - 1])) *p.nan_flag = 1;
      }
    }
    if (MODE == MODE_CODES && !keep && p.codes == nullptr) return;

    // ---- keep the rotated values when the straight-through form needs them
    u64 Y[MODE == MODE_DEQUANT ? 16 : 1];
    if (MODE == MODE_DEQUANT) {
#pragma unroll
      for (int j = 0; j < 16; ++j) Y[j] = P[j];
    }

    if (MX_FAST) {
      if (mx_e >= -120 && mx_e <= 120) {
        const u64 MK = mx_code_multiplier<GH>(mx_e);
        constexpr bool RZ = GH == 0 || GH == 16 || GH == 64;
#pragma unroll
        for (int j = 0; j < 16; ++j) P[j] = RZ ? mul2_rz(P[j], MK) : mul2(P[j], MK);
      } else {   // extreme exponents: scale, then divide exactly
        if (GH != 0) {
          const float cc = hadamard_scale<GH>();
          const u64 C = pack2(cc, cc);
#pragma unroll
          for (int j = 0; j < 16; ++j) P[j] = mul2(P[j], C);
        }
        divide_pairs(P, 16, s[0]);
      }
    } else if (NV_FOLD) {
      constexpr float c = GH == 16 ? 0.25f : 0.125f;
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const float sf = s[g] * (1.0f / c);
        // Exact while nothing leaves the normal range: then t c is exact for every element that can get a
        // non-zero code (an element whose t c is subnormal is > 2^20 below the group's scale).
        if (amax_g[g] > 7.8886e-31f /* 2^-100 */ && sf < 1.2676e30f /* 2^100 */) {
          divide_pairs(P + g * PG, PG, sf);
        } else {
          const u64 C = pack2(c, c);
#pragma unroll
          for (int j = 0; j < PG; ++j) P[g * PG + j] = mul2(P[g * PG + j], C);
          divide_pairs(P + g * PG, PG, s[g]);
        }
      }
    } else if (FMT == FMT_MXQUEST && sb[0] < 254u) {
      // the divisor is a power of two with a normal reciprocal: one multiply rounds the same exact quotient
      // (with the mask below: 8192 x 17408 in 67 us instead of 88)
      const float r = __uint_as_float((254u - sb[0]) << 23);
      const u64 R = pack2(r, r);
#pragma unroll
      for (int j = 0; j < 16; ++j) P[j] = mul2(P[j], R);
    } else {
#pragma unroll
      for (int g = 0; g < NG; ++g) divide_pairs(P + g * PG, PG, s[g]);
    }

    if (FMT == FMT_MXQUEST && p.mask != nullptr) {
      // bit i set = element i lies inside the grid's range (|x / 2^e| < 6, triton/mxfp4.py:105-110)
      // = the sign of |x / 2^e| - 6 (a subtraction never rounds across zero; a NaN comes out positive), shifted in
      // from the last element to the first
      uint32_t inside = 0;
#pragma unroll
      for (int j = 15; j >= 0; --j) {
        float a, b;
        unpack2(P[j], a, b);
        inside = __funnelshift_l(__float_as_uint(__fadd_rn(fabsf(b), -6.0f)), inside, 1);
        inside = __funnelshift_l(__float_as_uint(__fadd_rn(fabsf(a), -6.0f)), inside, 1);
      }
      if (active) {
        if (MODE == MODE_CODES) {
          reinterpret_cast<uint32_t*>(p.mask)[c] = inside;            // bit i of byte b = element 8 b + i
        } else {
          uint4* o = reinterpret_cast<uint4*>(p.mask) + c * 2;        // one bool byte per element
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t nib = (inside >> (16 * h + 4 * q)) & 15u;
              w[q] = (nib & 1u) | ((nib & 2u) << 7) | ((nib & 4u) << 14) | ((nib & 8u) << 21);
            }
            o[h] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }

    uint32_t cw[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) cw[q] = codes_word(P + 4 * q);

    if (MODE == MODE_CODES && keep) {
#pragma unroll
      for (int q = 0; q < 4; ++q) keep->cw[q] = cw[q];
    } else if (MODE == MODE_CODES) {
      if (active) reinterpret_cast<uint4*>(p.codes)[c] = make_uint4(cw[0], cw[1], cw[2], cw[3]);
    } else {  // MODE_DEQUANT
      float out[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float sc = s[(i * NG) / 32];
        float v = __fmul_rn(e2m1_value((cw[i / 8] >> (4 * (i % 8))) & 15u), sc);
        if (p.ste) {
          float a, b;
          unpack2(Y[i / 2], a, b);
          const float x = (i & 1) ? b : a;
          v = __fadd_rn(x, __fsub_rn(v, x));
        }
        out[i] = v;
      }
      if (active) {
        if (p.out_bf16) {
          uint4* o = reinterpret_cast<uint4*>(p.y) + c * 4;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              __nv_bfloat162 h = __floats2bfloat162_rn(out[8 * q + 2 * j], out[8 * q + 2 * j + 1]);
              w[j] = *reinterpret_cast<uint32_t*>(&h);
            }
            o[q] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        } else {
          float4* o = reinterpret_cast<float4*>(p.y) + c * 8;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            o[q] = make_float4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
        }
      }
    }
}

#ifndef FPQ_Q_PREFETCH
#define FPQ_Q_PREFETCH 1
#endif
#ifndef FPQ_Q_MINBLOCKS
#define FPQ_Q_MINBLOCKS 3
#endif

// A warp walks the chunks 32 at a time with a grid-wide stride.  For bf16 input the next chunk's
// sixteen words are loaded into a second register set before the current chunk is processed, so
// every thread keeps two 64-byte requests in flight.
template <bool IN_BF16, int MODE>
struct Prefetches { static constexpr bool value = FPQ_Q_PREFETCH && IN_BF16 && MODE != MODE_DEQUANT; };

template <int GH, int FMT, bool IN_BF16, int MODE>
__global__ void __launch_bounds__(256, Prefetches<IN_BF16, MODE>::value ? FPQ_Q_MINBLOCKS : 1) quant_kernel(const QuantParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t stride = (((int64_t)gridDim.x * blockDim.x) >> 5) * 32;
  launch_dependents();         // the next kernel may set itself up while this one runs
  grid_dependency_wait();      // the input (and the global scale) may come from the previous kernel
  float gs = 0.0f, rgs = 0.0f;
  if (FMT == FPQ_FMT_NVFP4 && (MODE == MODE_CODES || MODE == MODE_DEQUANT)) {
    gs = *p.gs;
    rgs = gs == 0.0f ? 0.0f : __frcp_rn(gs);
  }
  float running_max = 0.0f;

  int64_t cb = warp * 32;
  if (Prefetches<IN_BF16, MODE>::value) {
    RawChunk<IN_BF16> r0, r1;
    uint32_t m0 = 0, m1 = 0;                 // the chunk's mask word travels with it
    auto load_mask = [&](int64_t c, uint32_t& m) {
      if (MODE == MODE_ROTATE_MASK) m = c < p.n_chunks ? p.mask_in[c] : 0u;
    };
    if (cb < p.n_chunks) load_raw(p.x, cb + lane, cb + lane < p.n_chunks, r0);
    load_mask(cb + lane, m0);
    while (cb < p.n_chunks) {
      int64_t nx = cb + stride + lane;
      load_raw(p.x, nx, nx < p.n_chunks, r1);
      load_mask(nx, m1);
      process_chunk<GH, FMT, IN_BF16, MODE>(p, r0, cb + lane, cb + lane < p.n_chunks, lane, gs, rgs, running_max, m0);
      cb += stride;
      if (cb >= p.n_chunks) break;
      nx = cb + stride + lane;
      load_raw(p.x, nx, nx < p.n_chunks, r0);
      load_mask(nx, m0);
      process_chunk<GH, FMT, IN_BF16, MODE>(p, r1, cb + lane, cb + lane < p.n_chunks, lane, gs, rgs, running_max, m1);
      cb += stride;
    }
  } else {
    for (; cb < p.n_chunks; cb += stride) {
      const int64_t c = cb + lane;
      RawChunk<IN_BF16> r;
      load_raw(p.x, c, c < p.n_chunks, r);
      process_chunk<GH, FMT, IN_BF16, MODE>(p, r, c, c < p.n_chunks, lane, gs, rgs, running_max);
    }
  }

  if (MODE == MODE_CODES && p.pad_rows != 0) {
    // swizzled scale bytes of the rows between the tensor's last row and the end of its 128-row block: zero
    // (the GEMM's TMA loads whole 512-byte tiles, and a defined value keeps its pad rows finite)
    const int64_t n_words = (int64_t)p.pad_rows * p.sf_tiles_per_row_block;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
      const uint32_t r = p.rows + (uint32_t)(w / p.sf_tiles_per_row_block);
      const uint32_t kb = (uint32_t)(w % p.sf_tiles_per_row_block);
      *reinterpret_cast<uint32_t*>(p.sbytes + swizzled_offset(r, kb * 4u, p.sf_tiles_per_row_block)) = 0u;
    }
  }

  if (MODE == MODE_ABSMAX) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      running_max = fmaxf(running_max, __shfl_xor_sync(0xffffffffu, running_max, o));
    if (lane == 0) atomicMax(p.absmax_bits, __float_as_uint(running_max));
  }
}

// ---------------------------------------------------------------------------------------------------
// SiLU(gate) * up fused in front of the rotate + quantise pass: the input of an MLP's down-projection
// (src/utils/llama_utils.py:62-70 of IST-DASLab/FP-Quant computes `act_fn(gate) * up`, rotates it and
// quantises it in three passes over memory).  The activation keeps the reference's rounding points: it is
// what torch computes for bf16 tensors, silu in fp32 rounded to bf16, then the product rounded to bf16;
// from there on the chunk goes through process_chunk like any bf16 input.
__device__ __forceinline__ uint32_t silu_mul_word(uint32_t g2, uint32_t u2) {
  const float g0 = __uint_as_float(g2 << 16), g1 = __uint_as_float(g2 & 0xffff0000u);
  const float u0 = __uint_as_float(u2 << 16), u1 = __uint_as_float(u2 & 0xffff0000u);
  // x / (1 + exp(-x)) with the library exponential and an IEEE division, as torch evaluates silu
  const float s0 = __bfloat162float(__float2bfloat16_rn(__fdiv_rn(g0, __fadd_rn(1.0f, expf(-g0)))));
  const float s1 = __bfloat162float(__float2bfloat16_rn(__fdiv_rn(g1, __fadd_rn(1.0f, expf(-g1)))));
  const __nv_bfloat162 h = __floats2bfloat162_rn(__fmul_rn(s0, u0), __fmul_rn(s1, u1));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// The same for the sixteen words of a chunk whose gates all lie in [-80, 80], two elements per instruction:
//   t = 2^(-g log2 e): log2 e = C1 + C2 with C1 of 16 bits, so that g C1 is exact (g has 8 bits); what is
//   left is 2^(-g C2) = 1 - g C2 ln 2 (within 2^-23 at |g| = 80, less below) and the error of ex2.approx;
//   g / (1 + t) by reciprocal and one fused residual correction (Markstein, IBM J. Res. Dev. 34, 1990).
// t is raised by 2^-25: silu(2^-7) lies 5e-6 of a bf16 unit below a rounding tie, where fp32 has to land on the tie as
// the library's does (every raise from 2^-26 to 2^-23 agrees on all inputs, none at all misses this one).
// silu is a function of 16 input bits here: the rounded result equals the library exponential with the IEEE division on
// every one of them, which a test checks for all gates up to 80.  5.5 instructions an element instead of about 25: the kernel, bound by
// instruction issue before, takes 137 us instead of 215 for 8192 x 17408 (MXFP4, rotation 32; 4.7 TB/s of 6.5).
__device__ __forceinline__ void silu_mul_chunk(const RawChunk<true>& g, const RawChunk<true>& u, RawChunk<true>& h) {
  const u64 NC1 = pack2(-1.44268798828125f, -1.44268798828125f);            // -(log2 e rounded to 16 bits)
  const u64 NC2 = pack2(-4.8884952e-06f, -4.8884952e-06f);                  // -(log2 e - C1) ln 2
  const u64 EPS = pack2(2.9802322e-08f, 2.9802322e-08f);                    // 2^-25, see above
  const u64 ONE = pack2(1.0f, 1.0f), NEG = pack2(-1.0f, -1.0f);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const u64 G = pack2(__uint_as_float(g.w[j] << 16), __uint_as_float(g.w[j] & 0xffff0000u));
    const u64 U = pack2(__uint_as_float(u.w[j] << 16), __uint_as_float(u.w[j] & 0xffff0000u));
    float z0, z1, d0, d1, r0, r1, q0, q1;
    unpack2(mul2(G, NC1), z0, z1);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(z0));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(z1));
    u64 T = pack2(z0, z1);
    T = fma2(T, fma2(G, NC2, EPS), T);
    const u64 D = add2(T, ONE);
    unpack2(D, d0, d1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
    const u64 R = pack2(r0, r1);
    u64 Q = mul2(G, R);
    Q = fma2(fma2(mul2(D, NEG), Q, G), R, Q);
    unpack2(Q, q0, q1);
    const __nv_bfloat162 s2 = __floats2bfloat162_rn(q0, q1);
    const uint32_t sw = *reinterpret_cast<const uint32_t*>(&s2);
    unpack2(mul2(pack2(__uint_as_float(sw << 16), __uint_as_float(sw & 0xffff0000u)), U), q0, q1);
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(q0, q1);
    h.w[j] = *reinterpret_cast<const uint32_t*>(&h2);
  }
}

// Largest |gate| of the chunk at most 80 and no NaN among them.
__device__ __forceinline__ bool silu_range_ok(const RawChunk<true>& g) {
  uint32_t m = g.w[0] & 0x7fff7fffu;
#pragma unroll
  for (int j = 1; j < 16; ++j) asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(g.w[j] & 0x7fff7fffu));
  return (m & 0xffffu) <= 0x42a0u && (m >> 16) <= 0x42a0u;        // 0x42a0 = 80; NaN patterns lie above
}

constexpr int SILU_THREADS = 128, SILU_BLOCKS = 5;      // 96 registers: two chunks of loads, one of results, no spills

template <int GH, int FMT>
__global__ void __launch_bounds__(SILU_THREADS, SILU_BLOCKS) quant_silu_mul_kernel(const QuantParams p, const void* up) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t stride = (((int64_t)gridDim.x * blockDim.x) >> 5) * 32;
  launch_dependents();
  grid_dependency_wait();
  float gs = 0.0f, rgs = 0.0f;
  if (FMT == FPQ_FMT_NVFP4) {
    gs = *p.gs;
    rgs = gs == 0.0f ? 0.0f : __frcp_rn(gs);
  }
  float unused_max = 0.0f;
  int64_t cb = warp * 32;
  RawChunk<true> g, u;
  if (cb < p.n_chunks) {
    load_raw(p.x, cb + lane, cb + lane < p.n_chunks, g);
    load_raw(up, cb + lane, cb + lane < p.n_chunks, u);
  }
  while (cb < p.n_chunks) {
    RawChunk<true> h;
    if (silu_range_ok(g)) {
      silu_mul_chunk(g, u, h);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) h.w[j] = silu_mul_word(g.w[j], u.w[j]);
    }
    const int64_t nx = cb + stride + lane;          // the next chunk's loads fly while this one is quantised
    load_raw(p.x, nx, nx < p.n_chunks, g);
    load_raw(up, nx, nx < p.n_chunks, u);
    process_chunk<GH, FMT, true, MODE_CODES>(p, h, cb + lane, cb + lane < p.n_chunks, lane, gs, rgs, unused_max);
    cb += stride;
  }
  if (p.pad_rows != 0) {
    const int64_t n_words = (int64_t)p.pad_rows * p.sf_tiles_per_row_block;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
      const uint32_t r = p.rows + (uint32_t)(w / p.sf_tiles_per_row_block);
      const uint32_t kb = (uint32_t)(w % p.sf_tiles_per_row_block);
      *reinterpret_cast<uint32_t*>(p.sbytes + swizzled_offset(r, kb * 4u, p.sf_tiles_per_row_block)) = 0u;
    }
  }
}

template <int GH, int FMT>
int launch_silu_mul(const QuantParams& params, const void* up, cudaStream_t stream) {
  QuantParams p = params;
  p.row_magic = (p.chunks_per_row >= 2 && p.n_chunks < (1ll << 32)) ? ~0ull / p.chunks_per_row + 1 : 0;
  const int64_t blocks_needed = ceil_div64(p.n_chunks, SILU_THREADS);
  int64_t blocks = (int64_t)sm_count() * SILU_BLOCKS;          // persistent: the resident blocks of every SM
  if (blocks > blocks_needed) blocks = blocks_needed;
  if (blocks < 1) blocks = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(SILU_THREADS, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_dependent_launch() ? 1 : 0;
  FPQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, quant_silu_mul_kernel<GH, FMT>, p, up));
  return FPQ_OK;
}

// ---------------------------------------------------------------------------------------------------
// Quantise the TRANSPOSE of a matrix: x [t_rows, n] row-major -> MXFP4 of x^T [n, t_pad], rotated and scaled along the
// t axis (groups of 32 consecutive rows of x), without materialising x^T.  Two sources:
//   bf16: the upstream gradient, an operand of the weight-gradient GEMM of the quantised backward pass
//         (backward_t_bf16, inference_lib/src/fp_quant/module/qutlass_ops.py:218-245 of IST-DASLab/FP-Quant);
//   MXFP4: codes and scale bytes of the forward, dequantised, divided by *alpha and rounded to bf16 on the way
//         (backward_qt_bf16, qutlass_ops.py:248-274), so that the bf16 transpose never goes through memory.
// A warp takes a 32 x 32 tile of x, turns it round through shared memory as words of two consecutive t, and every
// lane then owns one output chunk: 32 consecutive t of one column of x, i.e. exactly the chunk process_chunk
// expects.  The next tile's loads fly meanwhile.  A warp takes runs of four tiles along t: the codes of two tiles leave
// as one 32-byte store per output row and the scale bytes of a run as one word (single 16-byte and 1-byte stores to
// 32 different rows cost more than the arithmetic).  Rows of x beyond t_rows read as zero (t_pad may exceed t_rows).
// The rotation must stay inside a chunk: group 0, 16 or 32.
// Bound by issue and by the latency of its scattered loads; 8192 x 17408: 82 us from bf16 (4.4 TB/s; 127 us without
// prefetch and with 16-byte stores), 119 us from MXFP4 (199 us as two kernels with the bf16 transpose between them).
struct TransposeIn {
  int64_t t_rows, n;
  const uint8_t* scales;       // MXFP4 source: E8M0 bytes of the codes (in QuantParams::x), [t_rows, n / 32]
  const float* alpha;
  int scale_layout;
};

// Column `col` of a tile: sixteen words of consecutive t pairs, 16-byte aligned.  Twenty words a column and eight more
// every eight columns make both the word stores and the 128-bit loads below free of bank conflicts.
__device__ __forceinline__ int tq_word(int col) { return col * 20 + 8 * (col >> 3); }
constexpr int TQ_WORDS = 32 * 20 + 32;
constexpr int TQ_THREADS = 128, TQ_BLOCKS = 5;      // 96 registers
constexpr int TQ_RUN = 4;      // tiles along t that a warp takes together

template <bool FP4IN> struct TransposeRaw;
template <> struct TransposeRaw<false> { uint4 v[4]; };                          // eight columns of rows 2k, 2k+1, 2k+16, 2k+17
template <> struct TransposeRaw<true> { uint2 c[2]; int e[2]; };                 // sixteen codes of rows 2k, 2k+1
constexpr int TQ_DEAD = -100000;                                                  // "exponent" of a row beyond t_rows

__device__ __forceinline__ void load_tile(const QuantParams& p, const TransposeIn& in, int64_t t0, int64_t j0, int lane,
                                          TransposeRaw<false>& r) {
  const int64_t col = j0 + (lane & 3) * 8;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t row = t0 + (lane >> 2) * 2 + (q & 1) + 16 * (q >> 1);
    r.v[q] = make_uint4(0u, 0u, 0u, 0u);
    if (row < in.t_rows && col < in.n)
      r.v[q] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.x) + row * in.n + col));
  }
}
__device__ __forceinline__ void load_tile(const QuantParams& p, const TransposeIn& in, int64_t t0, int64_t j0, int lane,
                                          TransposeRaw<true>& r) {
  const int64_t sf_cols = in.n / 32, ct = j0 / 32;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t row = t0 + (lane >> 1) * 2 + h;
    r.c[h] = make_uint2(0u, 0u);
    r.e[h] = TQ_DEAD;
    if (row < in.t_rows) {
      r.c[h] = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(p.x) + (row * in.n + j0) / 2 + (lane & 1) * 8));
      const size_t off = in.scale_layout == FPQ_SCALES_SWIZZLED
                             ? swizzled_offset((uint32_t)row, (uint32_t)ct, (uint32_t)((sf_cols + 3) / 4))
                             : (size_t)(row * sf_cols + ct);
      r.e[h] = (int)__ldg(in.scales + off) - 127;
    }
  }
}

// bf16 of (E2M1 magnitude / alpha), magnitudes 2 i and 2 i + 1 in a word.
struct QuotientTable {
  uint32_t w[4];
  float alpha;
  bool usable;
};
__device__ __forceinline__ void make_quotients(const float* alpha, QuotientTable& t) {
  t.alpha = *alpha;
  t.usable = t.alpha > 9.5367e-7f && t.alpha < 1.048576e6f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(__fdiv_rn(e2m1_magnitude(2 * i), t.alpha),
                                                   __fdiv_rn(e2m1_magnitude(2 * i + 1), t.alpha));
    t.w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}

// The row's bf16 values of the eight magnitudes, low bytes and high bytes (once more with the sign; the zero stays +0).
// fl((m 2^e) / a) = fl(m / a) 2^e while nothing leaves the normal range: e is added to the exponent fields.
struct RowTable {
  uint32_t lo_a, lo_b, hi_a, hi_b, nhi_a, nhi_b;
};
__device__ __forceinline__ void make_row_table(const QuotientTable& t, int e, RowTable& r) {
  uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
  if (e != TQ_DEAD) {
    const uint32_t add = (uint32_t)(e * 0x00800080);        // both halves stay positive: no borrow between them
    w0 = t.w[0] + (uint32_t)(e * 0x00800000);               // magnitude 0 stays 0
    w1 = t.w[1] + add;
    w2 = t.w[2] + add;
    w3 = t.w[3] + add;
  }
  r.lo_a = __byte_perm(w0, w1, 0x6420); r.hi_a = __byte_perm(w0, w1, 0x7531);
  r.lo_b = __byte_perm(w2, w3, 0x6420); r.hi_b = __byte_perm(w2, w3, 0x7531);
  r.nhi_a = (r.hi_a | 0x80808080u) & 0xffffff00u;
  r.nhi_b = r.hi_b | 0x80808080u;
}
// Four codes -> four bf16 values in two words.
__device__ __forceinline__ void row_lookup(const RowTable& r, uint32_t x, uint32_t& w01, uint32_t& w23) {
  const uint32_t sel = x & 0x7777u;
  const uint32_t lo4 = __byte_perm(r.lo_a, r.lo_b, sel);
  const uint32_t hi4 = __byte_perm(__byte_perm(r.hi_a, r.hi_b, sel), __byte_perm(r.nhi_a, r.nhi_b, sel),
                                   ((x & 0x8888u) >> 1) | 0x3210u);
  w01 = __byte_perm(lo4, hi4, 0x5140);
  w23 = __byte_perm(lo4, hi4, 0x7362);
}
__device__ __forceinline__ uint32_t slow_quotient(uint32_t code, int e, float alpha) {
  const float v = e == TQ_DEAD ? 0.0f : __fdiv_rn(scalbnf(e2m1_value(code), e), alpha);
  const __nv_bfloat16 h = __float2bfloat16_rn(v + 0.0f);
  return *reinterpret_cast<const uint16_t*>(&h);
}

__device__ __forceinline__ void store_tile(const TransposeRaw<false>& r, const QuotientTable&, int lane, uint32_t* tile) {
  const int piece = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t a[4] = {r.v[2 * h].x, r.v[2 * h].y, r.v[2 * h].z, r.v[2 * h].w};
    const uint32_t b[4] = {r.v[2 * h + 1].x, r.v[2 * h + 1].y, r.v[2 * h + 1].z, r.v[2 * h + 1].w};
    uint32_t* dst = tile + tq_word(piece * 8) + (lane >> 2) + 8 * h;
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[20 * j] = __byte_perm(a[j / 2], b[j / 2], (j & 1) ? 0x7632 : 0x5410);
  }
}
__device__ __forceinline__ void store_tile(const TransposeRaw<true>& r, const QuotientTable& t, int lane, uint32_t* tile) {
  const int half = lane & 1, k = lane >> 1;
  const bool fast0 = r.e[0] == TQ_DEAD || (r.e[0] > -100 && r.e[0] < 100);
  const bool fast1 = r.e[1] == TQ_DEAD || (r.e[1] > -100 && r.e[1] < 100);
  if (t.usable && fast0 && fast1) {
    RowTable ta, tb;
    make_row_table(t, r.e[0], ta);
    make_row_table(t, r.e[1], tb);
#pragma unroll
    for (int q = 0; q < 4; ++q) {                            // columns 16 half + 4 q ... + 3
      const uint32_t wa = q < 2 ? r.c[0].x : r.c[0].y, wb = q < 2 ? r.c[1].x : r.c[1].y;
      uint32_t a01, a23, b01, b23;
      row_lookup(ta, (q & 1) ? wa >> 16 : wa, a01, a23);
      row_lookup(tb, (q & 1) ? wb >> 16 : wb, b01, b23);
      uint32_t* dst = tile + tq_word(16 * half + 4 * q) + k;
      dst[0] = __byte_perm(a01, b01, 0x5410);
      dst[20] = __byte_perm(a01, b01, 0x7632);
      dst[40] = __byte_perm(a23, b23, 0x5410);
      dst[60] = __byte_perm(a23, b23, 0x7632);
    }
  } else {
    u64 ca = (u64)r.c[0].x | ((u64)r.c[0].y << 32), cb = (u64)r.c[1].x | ((u64)r.c[1].y << 32);
#pragma unroll 1
    for (int j = 0; j < 16; ++j, ca >>= 4, cb >>= 4)
      tile[tq_word(16 * half + j) + k] = slow_quotient((uint32_t)ca & 15u, r.e[0], t.alpha) |
                                         (slow_quotient((uint32_t)cb & 15u, r.e[1], t.alpha) << 16);
  }
}

template <int GH, bool FP4IN>
__global__ void __launch_bounds__(TQ_THREADS, TQ_BLOCKS) quant_transposed_kernel(const QuantParams p, const TransposeIn in) {
  static_assert(GH == 0 || GH == 16 || GH == 32, "the rotation group must fit one 32-element chunk");
  __shared__ __align__(16) uint32_t tiles[TQ_THREADS / 32][TQ_WORDS];
  const int lane = threadIdx.x & 31;
  uint32_t* tile = tiles[threadIdx.x >> 5];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  launch_dependents();
  grid_dependency_wait();
  QuotientTable quot{};
  if (FP4IN) make_quotients(in.alpha, quot);
  const int64_t col_tiles = (in.n + 31) / 32;
  const int t_tiles = (int)p.chunks_per_row, runs = (t_tiles + TQ_RUN - 1) / TQ_RUN;
  float unused_max = 0.0f;
  // run index = t_run * col_tiles + column tile: neighbouring warps read neighbouring pieces of the same rows
  int64_t run = warp, ct = 0;
  int tt = 0, t_end = 0;
  auto start_run = [&]() {
    const int64_t tr = run / col_tiles;
    ct = run - tr * col_tiles;
    tt = (int)tr * TQ_RUN;
    t_end = min(tt + TQ_RUN, t_tiles);
  };
  const int64_t n_runs = col_tiles * runs;
  const bool pair_stores = t_tiles % 2 == 0 && ((uintptr_t)p.codes & 31) == 0;
  uint4 before = make_uint4(0u, 0u, 0u, 0u);     // codes of the previous tile of the run
  uint32_t scale_word = 0;
  TransposeRaw<FP4IN> raw;
  if (run < n_runs) {
    start_run();
    load_tile(p, in, (int64_t)tt * 32, ct * 32, lane, raw);
  }
  while (run < n_runs) {
    __syncwarp();                               // every lane has read the previous tile
    store_tile(raw, quot, lane, tile);
    const int64_t out_row = ct * 32 + lane;
    const int chunk = tt, sub = chunk % TQ_RUN;
    const bool run_ends = ++tt == t_end;
    if (run_ends) {
      run += n_warps;
      if (run < n_runs) start_run();
    }
    if (run < n_runs) load_tile(p, in, (int64_t)tt * 32, ct * 32, lane, raw);
    __syncwarp();
    RawChunk<true> c;
    const uint4* src = reinterpret_cast<const uint4*>(tile + tq_word(lane));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 w = src[q];
      c.w[4 * q] = w.x; c.w[4 * q + 1] = w.y; c.w[4 * q + 2] = w.z; c.w[4 * q + 3] = w.w;
    }
    ChunkOut out;
    process_chunk<GH, FPQ_FMT_MXFP4, true, MODE_CODES>(p, c, 0, true, lane, 0.0f, 0.0f, unused_max, 0, &out);
    scale_word = sub == 0 ? out.sb : scale_word | (out.sb << (8 * sub));
    if (out_row < in.n) {
      uint4* dst = reinterpret_cast<uint4*>(p.codes) + out_row * t_tiles + chunk;
      const uint4 now = make_uint4(out.cw[0], out.cw[1], out.cw[2], out.cw[3]);
      if (sub & 1) {
        if (pair_stores) {
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst - 1), "r"(before.x), "r"(before.y),
                       "r"(before.z), "r"(before.w), "r"(now.x), "r"(now.y), "r"(now.z), "r"(now.w) : "memory");
        } else {
          dst[-1] = before;
          dst[0] = now;
        }
      } else if (run_ends) {
        dst[0] = now;
      }
      before = now;
      if (run_ends) {
        const int first = chunk - sub;
        if (p.layout == FPQ_SCALES_SWIZZLED) {      // a run is one word of the layout; what lies beyond t_pad is zero
          *reinterpret_cast<uint32_t*>(p.sbytes + swizzled_offset((uint32_t)out_row, (uint32_t)first, p.sf_tiles_per_row_block)) =
              scale_word;
        } else {
          uint8_t* sp = p.sbytes + out_row * t_tiles + first;
          for (int i = 0; i <= sub; ++i) sp[i] = (uint8_t)(scale_word >> (8 * i));
        }
      }
    }
  }
  if (p.pad_rows != 0) {
    const int64_t n_words = (int64_t)p.pad_rows * p.sf_tiles_per_row_block;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
      const uint32_t r = p.rows + (uint32_t)(w / p.sf_tiles_per_row_block);
      const uint32_t kb = (uint32_t)(w % p.sf_tiles_per_row_block);
      *reinterpret_cast<uint32_t*>(p.sbytes + swizzled_offset(r, kb * 4u, p.sf_tiles_per_row_block)) = 0u;
    }
  }
}

template <int GH, bool FP4IN>
int launch_transposed_one(const QuantParams& p, const TransposeIn& in, cudaStream_t stream) {
  const int64_t runs = ((in.n + 31) / 32) * (int64_t)((p.chunks_per_row + TQ_RUN - 1) / TQ_RUN);
  int64_t blocks = (int64_t)sm_count() * TQ_BLOCKS;          // persistent: the resident blocks of every SM
  if (blocks > ceil_div64(runs, TQ_THREADS / 32)) blocks = ceil_div64(runs, TQ_THREADS / 32);
  if (blocks < 1) blocks = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(TQ_THREADS, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_dependent_launch() ? 1 : 0;
  FPQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, quant_transposed_kernel<GH, FP4IN>, p, in));
  return FPQ_OK;
}

// x (bf16) or codes with `scales` and `alpha` (MXFP4): [t_rows, n] -> codes [n, t_pad/2] and scale bytes.
template <bool FP4IN>
int launch_transposed(const void* x, const uint8_t* scales, int in_layout, const float* alpha, int64_t t_rows, int64_t n,
                      int64_t t_pad, int hadamard_group, uint8_t* codes, uint8_t* scale_bytes, int scale_layout,
                      cudaStream_t stream) {
  QuantParams p{};
  p.x = x;
  p.n_chunks = n * t_pad / 32;
  p.chunks_per_row = (uint32_t)(t_pad / 32);
  p.codes = codes;
  p.sbytes = scale_bytes;
  p.sf_tiles_per_row_block = (uint32_t)ceil_div64(t_pad / 32, 4);
  p.layout = scale_layout;
  if (scale_layout == FPQ_SCALES_SWIZZLED) {
    p.rows = (uint32_t)n;
    p.pad_rows = (uint32_t)(ceil_div64(n, 128) * 128 - n);
  }
  TransposeIn in{t_rows, n, scales, alpha, in_layout};
  switch (hadamard_group) {
    case 0: return launch_transposed_one<0, FP4IN>(p, in, stream);
    case 16: return launch_transposed_one<16, FP4IN>(p, in, stream);
    default: return launch_transposed_one<32, FP4IN>(p, in, stream);
  }
}

template <int FMT>
int launch_silu_mul_gh(int gh, const QuantParams& p, const void* up, cudaStream_t stream) {
  switch (gh) {
    case 0: return launch_silu_mul<0, FMT>(p, up, stream);
    case 16: return launch_silu_mul<16, FMT>(p, up, stream);
    case 32: return launch_silu_mul<32, FMT>(p, up, stream);
    case 64: return launch_silu_mul<64, FMT>(p, up, stream);
    case 128: return launch_silu_mul<128, FMT>(p, up, stream);
  }
  set_error("hadamard_group must be 0, 16, 32, 64 or 128 (got %d)", gh);
  return FPQ_ERR_INVALID_ARGUMENT;
}

template <int GH, int FMT, bool IN_BF16, int MODE>
int launch_one(const QuantParams& params, cudaStream_t stream) {
  QuantParams p = params;
  p.row_magic = (p.chunks_per_row >= 2 && p.n_chunks < (1ll << 32)) ? ~0ull / p.chunks_per_row + 1 : 0;
  // persistent grid: exactly the number of blocks that are resident at once
  static int resident[64] = {};
  int dev = 0;
  FPQ_CHECK_CUDA(cudaGetDevice(&dev));
  int per_sm = dev < 64 ? resident[dev] : 0;
  if (per_sm == 0) {
    FPQ_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, quant_kernel<GH, FMT, IN_BF16, MODE>, 256, 0));
    if (per_sm < 1) per_sm = 1;
    if (dev < 64) resident[dev] = per_sm;
  }
  const int64_t warps_needed = ceil_div64(p.n_chunks, 32);
  const int64_t blocks_needed = ceil_div64(warps_needed, 8);
  int64_t blocks = (int64_t)sm_count() * per_sm;
  if (blocks > blocks_needed) blocks = blocks_needed;
  if (blocks < 1) blocks = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // Early launch is for short calls, where setting up counts.  Codes of an input that fills the chip more than once are
  // launched in order: next to the tail of the previous layer's GEMM the early blocks can cost more than they save.
  // Passes in a row, in order against early: 3001 x 5120 x 17408 146.7 us against 149.5, 11127 x 1664 x 1648 40.0 against
  // 40.6; 8192 x 12288 x 4096 223.2 against 221.6, 814 x 15808 x 12880 104.8 against 103.3; 0 on average over nine shapes.
  const bool early = MODE != MODE_CODES || blocks_needed <= (int64_t)sm_count() * per_sm;
  cfg.numAttrs = early && use_dependent_launch() ? 1 : 0;
  FPQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, quant_kernel<GH, FMT, IN_BF16, MODE>, p));
  return FPQ_OK;
}

template <int FMT, bool IN_BF16, int MODE>
int launch_gh(int gh, const QuantParams& p, cudaStream_t stream) {
  switch (gh) {
    case 0: return launch_one<0, FMT, IN_BF16, MODE>(p, stream);
    case 16: return launch_one<16, FMT, IN_BF16, MODE>(p, stream);
    case 32: return launch_one<32, FMT, IN_BF16, MODE>(p, stream);
    case 64: return launch_one<64, FMT, IN_BF16, MODE>(p, stream);
    case 128: return launch_one<128, FMT, IN_BF16, MODE>(p, stream);
  }
  set_error("hadamard_group must be 0, 16, 32, 64 or 128 (got %d)", gh);
  return FPQ_ERR_INVALID_ARGUMENT;
}

template <int MODE>
int launch_mode(int gh, int fmt, int dtype, const QuantParams& p, cudaStream_t stream) {
  if constexpr (MODE == MODE_ROTATE || MODE == MODE_ABSMAX) {
    return dtype == FPQ_DT_BF16 ? launch_gh<FPQ_FMT_MXFP4, true, MODE>(gh, p, stream)
                                : launch_gh<FPQ_FMT_MXFP4, false, MODE>(gh, p, stream);
  } else {
    if (fmt == FMT_MXQUEST)
      return dtype == FPQ_DT_BF16 ? launch_gh<FMT_MXQUEST, true, MODE>(gh, p, stream)
                                  : launch_gh<FMT_MXQUEST, false, MODE>(gh, p, stream);
    if (fmt == FPQ_FMT_MXFP4)
      return dtype == FPQ_DT_BF16 ? launch_gh<FPQ_FMT_MXFP4, true, MODE>(gh, p, stream)
                                  : launch_gh<FPQ_FMT_MXFP4, false, MODE>(gh, p, stream);
    return dtype == FPQ_DT_BF16 ? launch_gh<FPQ_FMT_NVFP4, true, MODE>(gh, p, stream)
                                : launch_gh<FPQ_FMT_NVFP4, false, MODE>(gh, p, stream);
  }
}

int check_common(const void* x, int dtype, int64_t rows, int64_t cols, int gh) {
  FPQ_CHECK_ARG(x != nullptr, "x is NULL");
  FPQ_CHECK_ARG(dtype == FPQ_DT_BF16 || dtype == FPQ_DT_F32, "dtype must be FPQ_DT_BF16 or FPQ_DT_F32");
  FPQ_CHECK_ARG(rows >= 0 && cols > 0, "bad shape [%lld, %lld]", (long long)rows, (long long)cols);
  FPQ_CHECK_ARG(cols % 32 == 0, "cols (%lld) must be a multiple of 32", (long long)cols);
  FPQ_CHECK_ARG(gh == 0 || gh == 16 || gh == 32 || gh == 64 || gh == 128,
                "hadamard_group must be 0, 16, 32, 64 or 128 (got %d)", gh);
  FPQ_CHECK_ARG(gh == 0 || cols % gh == 0, "cols (%lld) must be a multiple of the hadamard group %d",
                (long long)cols, gh);
  FPQ_CHECK_ARG(((uintptr_t)x & 31) == 0, "x must be 32-byte aligned");
  FPQ_CHECK_ARG(rows * cols / 32 < (int64_t)1 << 40, "tensor too large");
  return FPQ_OK;
}

// ------------------------------------------------------------------ auxiliary kernels
__global__ void global_scale_update_kernel(const uint32_t* absmax_bits, float* gs, int32_t* status) {
  float a = __uint_as_float(*absmax_bits);
  if (a == 0.0f) {
    if (status) *status = 1;
    return;
  }
  float cur = __fmul_rn(2688.0f, __fdiv_rn(1.0f, a));
  const float now = fminf(*gs, cur);
  *gs = now;
  if (status) *status = isfinite(now) ? 0 : 1;
}

// Eight consecutive elements of a tensor as fp32 and back.
template <bool BF16>
__device__ __forceinline__ void load8(const void* x, int64_t w, float (&v)[8]) {
  if (BF16) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(x) + w);
    const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(r[j] << 16);
      v[2 * j + 1] = __uint_as_float(r[j] & 0xffff0000u);
    }
  } else {
    const float4 a = __ldg(reinterpret_cast<const float4*>(x) + 2 * w), b = __ldg(reinterpret_cast<const float4*>(x) + 2 * w + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}
template <bool BF16>
__device__ __forceinline__ void store8(void* out, int64_t w, const float (&o)[8]) {
  if (BF16) {
    uint32_t r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
      r[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    reinterpret_cast<uint4*>(out)[w] = make_uint4(r[0], r[1], r[2], r[3]);
  } else {
    reinterpret_cast<float4*>(out)[2 * w] = make_float4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<float4*>(out)[2 * w + 1] = make_float4(o[4], o[5], o[6], o[7]);
  }
}
// Eight quotients -> a word of codes, as e2m1_code gives them: a NaN counts as zero.
__device__ __forceinline__ uint32_t codes_of8(const float (&q)[8]) {
  u64 P[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    P[j] = pack2(q[2 * j] == q[2 * j] ? q[2 * j] : 0.0f, q[2 * j + 1] == q[2 * j + 1] ? q[2 * j + 1] : 0.0f);
  return codes_word(P);
}
// The grid values of a word of codes (code 8, the zero, is -0 as e2m1_value has it).
__device__ __forceinline__ void values_of8(uint32_t word, float (&v)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t h2;
    asm("{ .reg .b8 t; .reg .b16 u; cvt.u16.u32 u, %1; cvt.u8.u16 t, u; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(h2) : "r"((word >> (8 * j)) & 0xffu));
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h2));
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}

// One thread per eight consecutive elements (one word of codes).  SHARED: the eight share a scale (the group is a
// multiple of eight), which sits at element / group whatever the row.  HBM-bound: 4 B in and 4 B out per fp32 element;
// 4096 x 4096 in 21 us instead of 42 with a general division, seven comparisons and a 64-bit division per element.
template <bool IN_BF16, bool SHARED>
__global__ void __launch_bounds__(256) apply_scales_kernel(const void* x, int64_t n_words, uint32_t cols,
                                                           const float* scales, uint32_t group, int out_kind,
                                                           void* out) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
       w += (int64_t)gridDim.x * blockDim.x) {
    float v[8], q[8], s[8];
    load8<IN_BF16>(x, w, v);
    if (SHARED) {
      const uint32_t per = group >> 3;
      const float s0 = __ldg(scales + (n_words < (1ll << 32) ? (int64_t)((uint32_t)w / per) : w / per));
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = s0;
      float m = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(v[j]));
      const float as = fabsf(s0);
      // multiply by the reciprocal and correct twice: the IEEE quotient while neither it nor the residuals leave the
      // normal range (a quotient that underflows is a zero code either way)
      if (m < 1.1529215e18f /* 2^60 */ && as > 8.6736174e-19f /* 2^-60 */ && as < 1.1529215e18f) {
        u64 P[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) P[j] = pack2(v[2 * j], v[2 * j + 1]);
        divide_pairs(P, 4, s0);
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(P[j], q[2 * j], q[2 * j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = __fdiv_rn(v[j], s0);
      }
    } else {
      const int64_t e0 = w * 8;
      const int64_t row = e0 / cols;
      const uint32_t col = (uint32_t)(e0 - row * cols);
      const float* srow = scales + row * (cols / group);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s[j] = srow[(col + j) / group];
        q[j] = __fdiv_rn(v[j], s[j]);
      }
    }
    const uint32_t word = codes_of8(q);
    if (out_kind == FPQ_OUT_CODES) {
      reinterpret_cast<uint32_t*>(out)[w] = word;
      continue;
    }
    float o[8];
    values_of8(word, o);
    if (out_kind != FPQ_OUT_GRID) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = __fmul_rn(o[j], s[j]);
        o[j] = out_kind == FPQ_OUT_DEQUANT_STE ? __fadd_rn(v[j], __fsub_rn(d, v[j])) : d;
      }
    }
    store8<IN_BF16>(out, w, o);
  }
}

// q * (the scale of its group), one rounding to the tensors' type; eight elements a thread, one scale for all of them.
template <bool BF16>
__global__ void __launch_bounds__(256) multiply_scales_kernel(const void* q, int64_t n_words, const void* scales, uint32_t per,
                                                              void* out) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
       w += (int64_t)gridDim.x * blockDim.x) {
    float v[8];
    load8<BF16>(q, w, v);
    const int64_t i = n_words < (1ll << 32) ? (int64_t)((uint32_t)w / per) : w / per;
    const float s = BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(scales)[i])
                         : __ldg(reinterpret_cast<const float*>(scales) + i);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(v[j], s);
    store8<BF16>(out, w, v);
  }
}

template <bool IN_BF16>
__global__ void __launch_bounds__(256) pack_grid_kernel(const void* q, int64_t n_words, uint32_t* packed) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
       w += (int64_t)gridDim.x * blockDim.x) {
    float v[8];
    load8<IN_BF16>(q, w, v);
    packed[w] = codes_of8(v);
  }
}

__global__ void __launch_bounds__(256) swizzle_scales_kernel(const uint8_t* __restrict__ src, uint32_t rows,
                                                             uint32_t sf_cols, uint32_t rows_pad,
                                                             uint32_t tiles_per_row_block,
                                                             uint32_t* __restrict__ dst) {
  // one thread per destination word (4 scale bytes of one row inside one tile)
  const int64_t n_words = (int64_t)rows_pad * tiles_per_row_block;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
       w += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t tile = (uint32_t)(w >> 7), in_tile = (uint32_t)(w & 127);
    const uint32_t rb = tile / tiles_per_row_block, kb = tile - rb * tiles_per_row_block;
    const uint32_t row = rb * 128 + (in_tile & 3u) * 32 + (in_tile >> 2);
    uint32_t word = 0;
    if (row < rows) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t c = kb * 4 + j;
        if (c < sf_cols) word |= (uint32_t)src[(size_t)row * sf_cols + c] << (8 * j);
      }
    }
    dst[w] = word;
  }
}

__global__ void __launch_bounds__(128) rotate_dense_kernel(const void* x, int in_bf16, void* y, int out_bf16,
                                                           int64_t n_groups, int g, const float* matrix) {
  // one warp per group; the g x g matrix lives in shared memory
  extern __shared__ float sm[];
  float* M = sm;                  // g * g
  float* xs = sm + g * g;         // 4 warps * g
  for (int i = threadIdx.x; i < g * g; i += blockDim.x) M[i] = matrix[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float* xw = xs + wid * g;
  for (int64_t grp = (int64_t)blockIdx.x * 4 + wid; grp < n_groups; grp += (int64_t)gridDim.x * 4) {
    for (int i = lane; i < g; i += 32)
      xw[i] = in_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[grp * g + i])
                      : reinterpret_cast<const float*>(x)[grp * g + i];
    __syncwarp();
    for (int j = lane; j < g; j += 32) {
      float acc = 0.0f;
      for (int k = 0; k < g; ++k) acc = __fadd_rn(acc, __fmul_rn(xw[k], M[k * g + j]));
      if (out_bf16) reinterpret_cast<__nv_bfloat16*>(y)[grp * g + j] = __float2bfloat16_rn(acc);
      else reinterpret_cast<float*>(y)[grp * g + j] = acc;
    }
    __syncwarp();
  }
}

int grid_for(int64_t work_items, int threads);

// ------------------------------------------------------------------ MSE observer
// One thread per scale group.  Candidates fl(f_i * s0), f_i = 1 - i * max_shrink / iters evaluated in double
// and rounded to fp32 as the reference's Python float is by the tensor multiply; error
// sum_j |x_j - grid(fl(x_j / s)) * s| ^ norm; the first strictly smaller error wins; the winner then goes
// through the scale-precision chain (src/quantization/quantizer.py:117-134, :143-165).  The candidates are
// not rounded to E4M3 / E8M0 during the search.
template <int G, bool NV, bool IN_BF16>
__global__ void __launch_bounds__(128) mse_scales_kernel(const void* __restrict__ x, int64_t n_groups,
                                                         const float* __restrict__ gs_ptr, int iters, double max_shrink,
                                                         float norm, float* __restrict__ scales_out) {
  float gs = 0.0f, rgs = 0.0f;
  if (NV) {
    gs = *gs_ptr;
    rgs = gs == 0.0f ? 0.0f : __fdiv_rn(1.0f, gs);
  }
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += (int64_t)gridDim.x * blockDim.x) {
    float v[G];
    if (IN_BF16) {
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + g * G);
#pragma unroll
      for (int q = 0; q < G / 8; ++q) {
        const uint4 raw = src[q];
        const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[8 * q + 2 * j] = __uint_as_float(r[j] << 16);
          v[8 * q + 2 * j + 1] = __uint_as_float(r[j] & 0xffff0000u);
        }
      }
    } else {
      const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + g * G);
#pragma unroll
      for (int q = 0; q < G / 4; ++q) {
        const float4 t = src[q];
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
      }
    }
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < G; ++j) a = fmaxf(a, fabsf(v[j]));
    const float s0 = __fdiv_rn(__fmul_rn(2.0f, a), 12.0f);
    float best = s0, best_err = __int_as_float(0x7f800000);
    if (s0 != 0.0f) {                         // an all-zero group divides 0 by 0: no candidate is ever "better"
      for (int i = 0; i < iters; ++i) {
        const float f = (float)(1.0 - (double)i * max_shrink / (double)iters);
        const float s = __fmul_rn(f, s0);
        float err = 0.0f;
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const float gv = e2m1_value(e2m1_code(__fdiv_rn(v[j], s)));
          const float d = fabsf(__fsub_rn(v[j], __fmul_rn(gv, s)));
          err = __fadd_rn(err, powf(d, norm));
        }
        if (err < best_err) {
          best_err = err;
          best = s;
        }
      }
    }
    uint32_t byte;
    float out;
    if (NV) {
      float t = fminf(fmaxf(__fmul_rn(best, gs), -448.0f), 448.0f);
      uint16_t u2;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(u2) : "f"(0.0f), "f"(t));
      const uint32_t u = u2 & 0xffu, ex = u >> 3, ma = u & 7u;
      const float uf = ex == 0 ? (float)ma * 0.001953125f : __uint_as_float(((ex + 120u) << 23) | (ma << 20));
      out = __fmul_rn(uf, rgs);
      byte = u;
    } else {
      const float m = fmaxf(__fmul_rn(6.0f, best), 1.17549435e-38f);
      const int e = mx_exponent(m);
      out = e >= -124 ? __uint_as_float(((uint32_t)(e + 125) << 23) | 0x2aaaabu) : __fdiv_rn(ldexpf(1.0f, e - 2), 0.75f);
      byte = (uint32_t)(e + 127);
    }
    (void)byte;
    scales_out[g] = out == 0.0f ? 1.0f : out;
  }
}

template <int G, bool NV>
int launch_mse(const void* x, int dtype, int64_t n_groups, const float* gs, int iters, double max_shrink, float norm,
               float* out, cudaStream_t st) {
  const int grid = grid_for(n_groups, 128);
  if (dtype == FPQ_DT_BF16)
    mse_scales_kernel<G, NV, true><<<grid, 128, 0, st>>>(x, n_groups, gs, iters, max_shrink, norm, out);
  else
    mse_scales_kernel<G, NV, false><<<grid, 128, 0, st>>>(x, n_groups, gs, iters, max_shrink, norm, out);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

int grid_for(int64_t work_items, int threads) {
  int64_t b = ceil_div64(work_items, threads);
  int64_t cap = (int64_t)sm_count() * 16;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace
}  // namespace fpq

using namespace fpq;

extern "C" int fpq_rotate_hadamard(const void* x, int dtype_in, void* y, int dtype_out, int64_t rows,
                                   int64_t cols, int group, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype_in, rows, cols, group)) return rc;
  FPQ_CHECK_ARG(group != 0, "group must be 16, 32, 64 or 128");
  FPQ_CHECK_ARG(y != nullptr && ((uintptr_t)y & 15) == 0, "y must be non-NULL and 16-byte aligned");
  FPQ_CHECK_ARG(dtype_out == FPQ_DT_BF16 || dtype_out == FPQ_DT_F32, "bad dtype_out");
  FPQ_CHECK_ARG(x != y || dtype_in == dtype_out, "in-place rotation needs equal dtypes");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.y = y;
  p.out_bf16 = dtype_out == FPQ_DT_BF16;
  return launch_mode<MODE_ROTATE>(group, 0, dtype_in, p, (cudaStream_t)stream);
}

// Backward of rotate + clip: y = rotate(x .* mask) in one pass over the gradient.  HBM-bound: 2 B + 1/8 B read and 2 B
// written per element.  The mask word rides along with its chunk's two loads.  Unpacking the mask into a bf16 tensor and
// multiplying first took six elementwise passes: 300 us of a 8192 x 4096 gradient and 445 us of a 12288 x 4096 one, which
// made a QuEST training step of that layer 1.49 ms; with this kernel it is 0.94 ms.
extern "C" int fpq_rotate_hadamard_masked(const void* x_bf16, const uint8_t* mask, void* y_bf16, int64_t rows,
                                          int64_t cols, int group, fpq_stream_t stream) {
  if (int rc = check_common(x_bf16, FPQ_DT_BF16, rows, cols, group)) return rc;
  FPQ_CHECK_ARG(mask != nullptr && ((uintptr_t)mask & 3) == 0, "mask must be non-NULL and 4-byte aligned");
  FPQ_CHECK_ARG(y_bf16 != nullptr && ((uintptr_t)y_bf16 & 15) == 0, "y must be non-NULL and 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x_bf16;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.y = y_bf16;
  p.mask_in = reinterpret_cast<const uint32_t*>(mask);
  p.out_bf16 = 1;
  return launch_gh<FPQ_FMT_MXFP4, true, MODE_ROTATE_MASK>(group, p, (cudaStream_t)stream);
}

extern "C" int fpq_rotate_dense(const void* x, int dtype_in, void* y, int dtype_out, int64_t rows,
                                int64_t cols, int group, const float* matrix, fpq_stream_t stream) {
  FPQ_CHECK_ARG(x && y && matrix, "NULL pointer");
  FPQ_CHECK_ARG(group == 16 || group == 32 || group == 64 || group == 128, "group must be 16, 32, 64 or 128");
  FPQ_CHECK_ARG(rows >= 0 && cols > 0 && cols % group == 0, "cols must be a multiple of group");
  FPQ_CHECK_ARG(x != y, "fpq_rotate_dense cannot run in place");
  if (rows == 0) return FPQ_OK;
  const int64_t n_groups = rows * cols / group;
  const size_t smem = (size_t)(group * group + 4 * group) * sizeof(float);
  FPQ_CHECK_CUDA(cudaFuncSetAttribute(rotate_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  rotate_dense_kernel<<<grid_for(n_groups, 4), 128, smem, (cudaStream_t)stream>>>(
      x, dtype_in == FPQ_DT_BF16, y, dtype_out == FPQ_DT_BF16, n_groups, group, matrix);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_absmax(const void* x, int dtype, int64_t rows, int64_t cols, int hadamard_group,
                          uint32_t* absmax_bits, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(absmax_bits != nullptr, "absmax_bits is NULL");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.absmax_bits = absmax_bits;
  return launch_mode<MODE_ABSMAX>(hadamard_group, 0, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_global_scale_update(const uint32_t* absmax_bits, float* global_scale, int32_t* status,
                                       fpq_stream_t stream) {
  FPQ_CHECK_ARG(absmax_bits && global_scale, "NULL pointer");
  global_scale_update_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(absmax_bits, global_scale, status);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_quantize(const void* x, int dtype, int64_t rows, int64_t cols, int hadamard_group,
                            int format, const float* global_scale, uint8_t* codes, uint8_t* scale_bytes,
                            int scale_layout, float* scales_f32, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(format == FPQ_FMT_MXFP4 || format == FPQ_FMT_NVFP4, "format must be FPQ_FMT_MXFP4 or FPQ_FMT_NVFP4");
  FPQ_CHECK_ARG(format != FPQ_FMT_NVFP4 || global_scale != nullptr, "NVFP4 needs a global_scale pointer");
  FPQ_CHECK_ARG(scale_layout == FPQ_SCALES_ROWMAJOR || scale_layout == FPQ_SCALES_SWIZZLED, "bad scale_layout");
  FPQ_CHECK_ARG(codes || scale_bytes || scales_f32, "no output requested");
  FPQ_CHECK_ARG(((uintptr_t)codes & 15) == 0 && ((uintptr_t)scale_bytes & 15) == 0 && ((uintptr_t)scales_f32 & 15) == 0,
                "outputs must be 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  const int g = format == FPQ_FMT_NVFP4 ? 16 : 32;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.codes = codes;
  p.sbytes = scale_bytes;
  p.sf32 = scales_f32;
  p.gs = global_scale;
  p.sf_tiles_per_row_block = (uint32_t)ceil_div64(cols / g, 4);
  p.layout = scale_layout;
  if (scale_bytes && scale_layout == FPQ_SCALES_SWIZZLED) {
    FPQ_CHECK_ARG(rows < ((int64_t)1 << 31), "too many rows for the swizzled scale layout");
    p.rows = (uint32_t)rows;
    p.pad_rows = (uint32_t)(ceil_div64(rows, 128) * 128 - rows);
  }
  return launch_mode<MODE_CODES>(hadamard_group, format, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_quantize_silu_mul(const void* gate_bf16, const void* up_bf16, int64_t rows, int64_t cols,
                                     int hadamard_group, int format, const float* global_scale, uint8_t* codes,
                                     uint8_t* scale_bytes, int scale_layout, fpq_stream_t stream) {
  if (int rc = check_common(gate_bf16, FPQ_DT_BF16, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(up_bf16 != nullptr && ((uintptr_t)up_bf16 & 31) == 0, "up must be non-NULL and 32-byte aligned");
  FPQ_CHECK_ARG(format == FPQ_FMT_MXFP4 || format == FPQ_FMT_NVFP4, "format must be FPQ_FMT_MXFP4 or FPQ_FMT_NVFP4");
  FPQ_CHECK_ARG(format != FPQ_FMT_NVFP4 || global_scale != nullptr, "NVFP4 needs a global_scale pointer");
  FPQ_CHECK_ARG(scale_layout == FPQ_SCALES_ROWMAJOR || scale_layout == FPQ_SCALES_SWIZZLED, "bad scale_layout");
  FPQ_CHECK_ARG(codes != nullptr && scale_bytes != nullptr, "codes and scale_bytes are required");
  FPQ_CHECK_ARG(((uintptr_t)codes & 15) == 0 && ((uintptr_t)scale_bytes & 15) == 0, "outputs must be 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  const int g = format == FPQ_FMT_NVFP4 ? 16 : 32;
  QuantParams p{};
  p.x = gate_bf16;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.codes = codes;
  p.sbytes = scale_bytes;
  p.gs = global_scale;
  p.sf_tiles_per_row_block = (uint32_t)ceil_div64(cols / g, 4);
  p.layout = scale_layout;
  if (scale_layout == FPQ_SCALES_SWIZZLED) {
    FPQ_CHECK_ARG(rows < ((int64_t)1 << 31), "too many rows for the swizzled scale layout");
    p.rows = (uint32_t)rows;
    p.pad_rows = (uint32_t)(ceil_div64(rows, 128) * 128 - rows);
  }
  return format == FPQ_FMT_NVFP4 ? launch_silu_mul_gh<FPQ_FMT_NVFP4>(hadamard_group, p, up_bf16, (cudaStream_t)stream)
                                 : launch_silu_mul_gh<FPQ_FMT_MXFP4>(hadamard_group, p, up_bf16, (cudaStream_t)stream);
}

extern "C" int fpq_quantize_transposed(const void* x_bf16, int64_t t_rows, int64_t n, int64_t t_pad, int hadamard_group,
                                       uint8_t* codes, uint8_t* scale_bytes, int scale_layout, fpq_stream_t stream) {
  FPQ_CHECK_ARG(x_bf16 && codes && scale_bytes, "NULL pointer");
  FPQ_CHECK_ARG(t_rows > 0 && n > 0 && n % 8 == 0, "n (%lld) must be a positive multiple of 8", (long long)n);
  FPQ_CHECK_ARG(t_pad >= t_rows && t_pad % 32 == 0, "t_pad (%lld) must be a multiple of 32 not below t_rows", (long long)t_pad);
  FPQ_CHECK_ARG(hadamard_group == 0 || hadamard_group == 16 || hadamard_group == 32,
                "the rotation group of the transposing quantiser must be 0, 16 or 32 (got %d)", hadamard_group);
  FPQ_CHECK_ARG(scale_layout == FPQ_SCALES_ROWMAJOR || scale_layout == FPQ_SCALES_SWIZZLED, "bad scale_layout");
  FPQ_CHECK_ARG(((uintptr_t)x_bf16 & 15) == 0 && ((uintptr_t)codes & 15) == 0 && ((uintptr_t)scale_bytes & 15) == 0,
                "pointers must be 16-byte aligned");
  FPQ_CHECK_ARG(n < ((int64_t)1 << 31) && t_pad < ((int64_t)1 << 31), "shape too large");
  return launch_transposed<false>(x_bf16, nullptr, 0, nullptr, t_rows, n, t_pad, hadamard_group, codes, scale_bytes,
                                  scale_layout, (cudaStream_t)stream);
}

extern "C" int fpq_mxfp4_requantize_transposed(const uint8_t* codes_in, const uint8_t* scales_in, int scale_layout_in,
                                               const float* alpha, int64_t t_rows, int64_t n, int64_t t_pad,
                                               int hadamard_group, uint8_t* codes, uint8_t* scale_bytes, int scale_layout,
                                               fpq_stream_t stream) {
  FPQ_CHECK_ARG(codes_in && scales_in && alpha && codes && scale_bytes, "NULL pointer");
  FPQ_CHECK_ARG(t_rows > 0 && n > 0 && n % 32 == 0, "n (%lld) must be a positive multiple of 32", (long long)n);
  FPQ_CHECK_ARG(t_pad >= t_rows && t_pad % 32 == 0, "t_pad (%lld) must be a multiple of 32 not below t_rows", (long long)t_pad);
  FPQ_CHECK_ARG(hadamard_group == 0 || hadamard_group == 16 || hadamard_group == 32,
                "the rotation group of the transposing quantiser must be 0, 16 or 32 (got %d)", hadamard_group);
  for (int layout : {scale_layout_in, scale_layout})
    FPQ_CHECK_ARG(layout == FPQ_SCALES_ROWMAJOR || layout == FPQ_SCALES_SWIZZLED, "bad scale layout");
  FPQ_CHECK_ARG(((uintptr_t)codes_in & 15) == 0 && ((uintptr_t)codes & 15) == 0 && ((uintptr_t)scale_bytes & 15) == 0,
                "pointers must be 16-byte aligned");
  FPQ_CHECK_ARG(n < ((int64_t)1 << 31) && t_pad < ((int64_t)1 << 31), "shape too large");
  return launch_transposed<true>(codes_in, scales_in, scale_layout_in, alpha, t_rows, n, t_pad, hadamard_group, codes,
                                 scale_bytes, scale_layout, (cudaStream_t)stream);
}

extern "C" int fpq_fake_quantize(const void* x, int dtype, int64_t rows, int64_t cols, int hadamard_group,
                                 int format, const float* global_scale, void* y, int ste, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(format == FPQ_FMT_MXFP4 || format == FPQ_FMT_NVFP4, "format must be FPQ_FMT_MXFP4 or FPQ_FMT_NVFP4");
  FPQ_CHECK_ARG(format != FPQ_FMT_NVFP4 || global_scale != nullptr, "NVFP4 needs a global_scale pointer");
  FPQ_CHECK_ARG(y != nullptr && ((uintptr_t)y & 15) == 0, "y must be non-NULL and 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.y = y;
  p.gs = global_scale;
  p.out_bf16 = dtype == FPQ_DT_BF16;
  p.ste = ste;
  return launch_mode<MODE_DEQUANT>(hadamard_group, format, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_quantize_quest(const void* x, int dtype, int64_t rows, int64_t cols, int hadamard_group,
                                  uint8_t* codes, uint8_t* scale_bytes, int scale_layout, uint8_t* clip_mask,
                                  fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(scale_layout == FPQ_SCALES_ROWMAJOR || scale_layout == FPQ_SCALES_SWIZZLED, "bad scale_layout");
  FPQ_CHECK_ARG(codes != nullptr, "codes is NULL");
  FPQ_CHECK_ARG(((uintptr_t)codes & 15) == 0 && ((uintptr_t)scale_bytes & 15) == 0 && ((uintptr_t)clip_mask & 3) == 0,
                "codes and scale_bytes must be 16-byte aligned, clip_mask 4-byte aligned");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.codes = codes;
  p.sbytes = scale_bytes;
  p.mask = clip_mask;
  p.sf_tiles_per_row_block = (uint32_t)ceil_div64(cols / 32, 4);
  p.layout = scale_layout;
  if (scale_bytes && scale_layout == FPQ_SCALES_SWIZZLED) {
    FPQ_CHECK_ARG(rows < ((int64_t)1 << 31), "too many rows for the swizzled scale layout");
    p.rows = (uint32_t)rows;
    p.pad_rows = (uint32_t)(ceil_div64(rows, 128) * 128 - rows);
  }
  return launch_mode<MODE_CODES>(hadamard_group, FMT_MXQUEST, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_fake_quantize_quest(const void* x, int dtype, int64_t rows, int64_t cols, int hadamard_group,
                                       void* y, uint8_t* clip_mask, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, hadamard_group)) return rc;
  FPQ_CHECK_ARG(y != nullptr && ((uintptr_t)y & 15) == 0, "y must be non-NULL and 16-byte aligned");
  FPQ_CHECK_ARG(((uintptr_t)clip_mask & 15) == 0, "clip_mask must be 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.y = y;
  p.mask = clip_mask;
  p.out_bf16 = dtype == FPQ_DT_BF16;
  return launch_mode<MODE_DEQUANT>(hadamard_group, FMT_MXQUEST, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_apply_scales(const void* x, int dtype, int64_t rows, int64_t cols, const float* scales,
                                int group, int out_kind, void* out, fpq_stream_t stream) {
  FPQ_CHECK_ARG(x && scales && out, "NULL pointer");
  FPQ_CHECK_ARG(dtype == FPQ_DT_BF16 || dtype == FPQ_DT_F32, "bad dtype");
  FPQ_CHECK_ARG(rows >= 0 && cols > 0 && group > 0 && cols % group == 0 && cols % 8 == 0,
                "group (%d) must divide cols (%lld) and cols must be a multiple of 8", group, (long long)cols);
  FPQ_CHECK_ARG(out_kind >= FPQ_OUT_CODES && out_kind <= FPQ_OUT_DEQUANT_STE, "bad out_kind");
  FPQ_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)out & 15) == 0, "x and out must be 16-byte aligned");
  FPQ_CHECK_ARG(cols < ((int64_t)1 << 31), "cols too large");
  if (rows == 0) return FPQ_OK;
  const int64_t n_words = rows * cols / 8;
  const int grid = grid_for(n_words, 256);
  const bool shared = group % 8 == 0;
  auto kernel = dtype == FPQ_DT_BF16 ? (shared ? apply_scales_kernel<true, true> : apply_scales_kernel<true, false>)
                                     : (shared ? apply_scales_kernel<false, true> : apply_scales_kernel<false, false>);
  kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(x, n_words, (uint32_t)cols, scales, (uint32_t)group, out_kind, out);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_multiply_scales(const void* q, int dtype, int64_t n, const void* scales, int group, void* out,
                                   fpq_stream_t stream) {
  FPQ_CHECK_ARG(q && scales && out, "NULL pointer");
  FPQ_CHECK_ARG(dtype == FPQ_DT_BF16 || dtype == FPQ_DT_F32, "bad dtype");
  FPQ_CHECK_ARG(n >= 0 && group > 0 && group % 8 == 0 && n % group == 0, "the group (%d) must be a multiple of 8 that divides n", group);
  FPQ_CHECK_ARG(((uintptr_t)q & 15) == 0 && ((uintptr_t)out & 15) == 0, "q and out must be 16-byte aligned");
  if (n == 0) return FPQ_OK;
  const int grid = grid_for(n / 8, 256);
  if (dtype == FPQ_DT_BF16)
    multiply_scales_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(q, n / 8, scales, (uint32_t)group / 8, out);
  else
    multiply_scales_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(q, n / 8, scales, (uint32_t)group / 8, out);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_group_scales(const void* x, int dtype, int64_t rows, int64_t cols, int format, const float* global_scale,
                                float* scales_f32, int32_t* nan_flag, fpq_stream_t stream) {
  if (int rc = check_common(x, dtype, rows, cols, 0)) return rc;
  FPQ_CHECK_ARG(format == FPQ_FMT_MXFP4 || format == FPQ_FMT_NVFP4, "format must be FPQ_FMT_MXFP4 or FPQ_FMT_NVFP4");
  FPQ_CHECK_ARG(format != FPQ_FMT_NVFP4 || global_scale != nullptr, "NVFP4 needs a global_scale pointer");
  FPQ_CHECK_ARG(scales_f32 != nullptr && ((uintptr_t)scales_f32 & 15) == 0, "scales_f32 must be non-NULL and 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  QuantParams p{};
  p.x = x;
  p.n_chunks = rows * cols / 32;
  p.chunks_per_row = (uint32_t)(cols / 32);
  p.sf32 = scales_f32;
  p.nan_flag = nan_flag;
  p.gs = global_scale;
  return launch_mode<MODE_CODES>(0, format, dtype, p, (cudaStream_t)stream);
}

extern "C" int fpq_mse_scales(const void* x, int dtype, int64_t rows, int64_t cols, int format,
                              const float* global_scale, int iters, double max_shrink, float error_norm,
                              float* scales_f32, fpq_stream_t stream) {
  FPQ_CHECK_ARG(x && scales_f32, "NULL pointer");
  FPQ_CHECK_ARG(dtype == FPQ_DT_BF16 || dtype == FPQ_DT_F32, "bad dtype");
  FPQ_CHECK_ARG(format == FPQ_FMT_NVFP4 || format == FPQ_FMT_MXFP4, "bad format");
  FPQ_CHECK_ARG(format != FPQ_FMT_NVFP4 || global_scale != nullptr, "NVFP4 needs the tensor scale");
  FPQ_CHECK_ARG(rows >= 0 && cols > 0 && cols % 32 == 0, "cols must be a multiple of 32");
  FPQ_CHECK_ARG(iters > 0 && iters <= 100000 && max_shrink >= 0.0 && max_shrink < 1.0, "bad search parameters");
  FPQ_CHECK_ARG(((uintptr_t)x & 15) == 0, "x must be 16-byte aligned");
  if (rows == 0) return FPQ_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (format == FPQ_FMT_NVFP4)
    return launch_mse<16, true>(x, dtype, rows * cols / 16, global_scale, iters, max_shrink, error_norm, scales_f32, st);
  return launch_mse<32, false>(x, dtype, rows * cols / 32, nullptr, iters, max_shrink, error_norm, scales_f32, st);
}

extern "C" int fpq_pack_grid(const void* q, int dtype, int64_t rows, int64_t cols, uint8_t* packed,
                             fpq_stream_t stream) {
  FPQ_CHECK_ARG(q && packed, "NULL pointer");
  FPQ_CHECK_ARG(dtype == FPQ_DT_BF16 || dtype == FPQ_DT_F32, "bad dtype");
  FPQ_CHECK_ARG(rows >= 0 && cols > 0 && cols % 8 == 0, "cols must be a multiple of 8");
  FPQ_CHECK_ARG(((uintptr_t)q & 15) == 0 && ((uintptr_t)packed & 3) == 0, "bad alignment");
  if (rows == 0) return FPQ_OK;
  const int64_t n_words = rows * cols / 8;
  const int grid = grid_for(n_words, 256);
  if (dtype == FPQ_DT_BF16)
    pack_grid_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(q, n_words, reinterpret_cast<uint32_t*>(packed));
  else
    pack_grid_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(q, n_words, reinterpret_cast<uint32_t*>(packed));
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_swizzle_scales(const uint8_t* rowmajor, int64_t rows, int64_t sf_cols, uint8_t* swizzled,
                                  fpq_stream_t stream) {
  FPQ_CHECK_ARG(rowmajor && swizzled, "NULL pointer");
  FPQ_CHECK_ARG(rows > 0 && sf_cols > 0 && rows < ((int64_t)1 << 31) && sf_cols < ((int64_t)1 << 31), "bad shape");
  FPQ_CHECK_ARG(((uintptr_t)swizzled & 3) == 0, "swizzled must be 4-byte aligned");
  const uint32_t rows_pad = (uint32_t)(ceil_div64(rows, 128) * 128);
  const uint32_t tprb = (uint32_t)ceil_div64(sf_cols, 4);
  const int64_t n_words = (int64_t)rows_pad * tprb;
  swizzle_scales_kernel<<<grid_for(n_words, 256), 256, 0, (cudaStream_t)stream>>>(
      rowmajor, (uint32_t)rows, (uint32_t)sf_cols, rows_pad, tprb, reinterpret_cast<uint32_t*>(swizzled));
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

// Rotate + quantise and the FP4 GEMM in one call: what a linear layer does per forward pass.  The activations' codes and
// swizzled scale bytes go to the caller's workspace.  A decode step is bound by the host: two calls with their tensor
// wrappers and checks cost more than the two kernels.
extern "C" int64_t fpq_linear_workspace_bytes(int64_t M, int64_t K, int format) {
  if (M < 0 || K <= 0) return 0;
  const int g = format == FPQ_FMT_NVFP4 ? 16 : 32;
  const int64_t codes = (M * (K / 2) + 255) & ~(int64_t)255;
  return codes + ((M + 127) & ~(int64_t)127) * ((K / g + 3) & ~(int64_t)3);
}

extern "C" int fpq_linear_forward(const void* x_bf16, const void* up_bf16, int64_t M, int64_t N, int64_t K,
                                  int hadamard_group, int format, int quest, const float* global_scale,
                                  const uint8_t* w_codes, const uint8_t* w_scales_swizzled, const float* alpha,
                                  const void* bias_bf16, void* workspace, int64_t workspace_bytes, void* out_bf16,
                                  int32_t* error_flag, fpq_stream_t stream) {
  FPQ_CHECK_ARG(workspace != nullptr && ((uintptr_t)workspace & 255) == 0, "the workspace must be non-NULL and 256-byte aligned");
  FPQ_CHECK_ARG(workspace_bytes >= fpq_linear_workspace_bytes(M, K, format), "the workspace is too small");
  FPQ_CHECK_ARG(!quest || (format == FPQ_FMT_MXFP4 && up_bf16 == nullptr), "QuEST scales are an MXFP4 rule without the fused SiLU");
  const int g = format == FPQ_FMT_NVFP4 ? 16 : 32;
  uint8_t* codes = reinterpret_cast<uint8_t*>(workspace);
  uint8_t* sb = codes + ((M * (K / 2) + 255) & ~(int64_t)255);
  if ((K / g) % 4 != 0 && M > 0)       // scale columns up to the next multiple of four: zero (pad rows: the quantise kernel)
    FPQ_CHECK_CUDA(cudaMemsetAsync(sb, 0, (size_t)(((M + 127) & ~(int64_t)127) * ((K / g + 3) & ~(int64_t)3)), (cudaStream_t)stream));
  int rc;
  if (up_bf16)
    rc = fpq_quantize_silu_mul(x_bf16, up_bf16, M, K, hadamard_group, format, global_scale, codes, sb, FPQ_SCALES_SWIZZLED, stream);
  else if (quest)
    rc = fpq_quantize_quest(x_bf16, FPQ_DT_BF16, M, K, hadamard_group, codes, sb, FPQ_SCALES_SWIZZLED, nullptr, stream);
  else
    rc = fpq_quantize(x_bf16, FPQ_DT_BF16, M, K, hadamard_group, format, global_scale, codes, sb, FPQ_SCALES_SWIZZLED, nullptr, stream);
  if (rc != FPQ_OK) return rc;
  return fpq_gemm_fp4(codes, w_codes, sb, w_scales_swizzled, alpha, bias_bf16, out_bf16, M, N, K, format, error_flag, stream);
}
