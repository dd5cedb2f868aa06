// Integer arithmetic of the decode GEMV for one or two activation rows: weight quants as bytes, activations as four planes of
// signed base-256 digits, mma.sync.m16n8k32 (u8 / s8 x s8, int32 accumulation).
//
// Why.  The decode kernels are bound by the half-rate integer pipe (two warp instructions per clock and SM for LOP3, PRMT, SHF,
// IMAD; four for FFMA).  Turning a 4-bit quant into a 16-bit float operand costs 3.5 of them per four weights; as a byte operand
// it costs one: the low nibbles of a word are w & 0x0f0f0f0f, the high ones w & 0xf0f0f0f0 (16 q, the 1/16 goes into the scale).  The
// byte MMA runs at the instruction rate of the 16-bit one with twice the K, and an MMA has eight columns: four digits per
// activation row use four (one row) or eight (two rows) columns that were idle.
//
// Precision.  A row's activations are fixed-point numbers relative to the largest of their 256-weight super-block: x =
// xs * (d0 + 256 d1 + 256^2 d2 + 256^3 d3) with |x / xs| < 2^30.  With the largest in [2^E, 2^(E+1)) a value is rounded once, by at most
// 2^(E-30); float32 values from 2^(E-6) on, float16 from 2^(E-19) and bfloat16 from 2^(E-22) are exact.  Products and sums of a sub-block
// are exact integers; scales, super-blocks and rows are added in fp32.
// Where the large values of a super-block meet weights that are zero, only the small ones are left in the result, and the rounding is
// to be measured against them.  So planes are made only where at most a quarter of the values that are not zero lie below 2^(E-8) (16-bit
// types, whose larger values are exact: 2^(E-14)).  For the other three quarters the rounding is at most 2^-22 of the value (float32): with
// normally distributed values 2^-24 of their deviation, no more than the fp32 sums of products that this replaces.
// A super-block with a wider range than that, with an Inf, a NaN or values whose sums or digits leave the range of fp32 has no planes: its
// scale is zero, and it is multiplied weight by weight (plain()), which gives +-Inf or NaN as the products do.
//
// Every lane keeps two columns of two weight rows: lane t of a quad has digits 2 (t & 1) and 2 (t & 1) + 1.  One IMAD joins the two
// digits, one I2F and one FFMA apply the sub-block scale; the factor 256^2 of the odd lanes and xs are applied per super-block.
#pragma once
#include <type_traits>

#include "gemv_mma_common.cuh"

namespace b200gguf {
namespace planes {

constexpr int kSbBytes = 1024;                 // digit planes of one super-block of one activation row
constexpr int kScalePitch = 20;                // floats per row of the scale scratch (16 + 4: 16-byte reads of 8 rows hit all banks)

// Types with an integer path (the FP4 types keep their 16-bit operands).
template <int QT> constexpr bool has() {
  return QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q6_K || QT == QTYPE_Q8_0 || QT == QTYPE_Q4_0 || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K;
}
template <int QT> constexpr bool has_mins() { return QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q2_K; }
template <int QT> constexpr bool sub16() { return QT == QTYPE_Q6_K || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K; }    // a scale per 16 weights

template <bool SIGNED>
__device__ __forceinline__ void mma32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (SIGNED)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
  else
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
template <bool SIGNED>
__device__ __forceinline__ void mma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  if (SIGNED)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

// ---- activations -> digit planes (one warp per super-block and row; lane i holds weights 8i .. 8i+7)
// Four numbers -> their digits, plane by plane: byte i of p[c] is digit c of z[i].
__device__ __forceinline__ void transpose4(const uint32_t (&z)[4], uint32_t (&p)[4]) {
  const uint32_t a = __byte_perm(z[0], z[1], 0x5140), b = __byte_perm(z[2], z[3], 0x5140);
  const uint32_t c = __byte_perm(z[0], z[1], 0x7362), d = __byte_perm(z[2], z[3], 0x7362);
  p[0] = __byte_perm(a, b, 0x5410); p[1] = __byte_perm(a, b, 0x7632);
  p[2] = __byte_perm(c, d, 0x5410); p[3] = __byte_perm(c, d, 0x7632);
}

// xp: the 1024 bytes of this super-block; xs: its scale (zero: left to plain()); X: sums of its activations per sub-block (types with mins), or null.
// Where a piece goes follows the order in which the lanes of the MMA take the weights:
//   Q4_K, Q5_K, Q8_0: MMA j = weights 32j .. +31, lane t has weights 8t .. 8t+7 of it (8 bytes);
//   Q4_0:             MMA j = block j, lane t has weights 4t .. (low nibbles) and 16 + 4t .. (high nibbles);
//   16-weight types:  lane t has weights 4t .. of sub-block (hb, quad, u), the four quads side by side.
template <int QT, typename T>
__device__ __forceinline__ void make(const T* x, int valid, int lane, uint8_t* xp, float* xs, float* X) {
  float f[8];
  if (8 * lane < valid) {
    load8<T>(x + 8 * lane, f);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = 0.f;
  }
  float sum = 0.f;
  uint32_t bits = 0, least = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t magnitude = __float_as_uint(f[i]) & 0x7fffffffu;      // as integers: an Inf or NaN is larger than every finite value
    bits = max(bits, magnitude);
    least = min(least, magnitude);
    sum += f[i];
  }
  bits = __reduce_max_sync(0xffffffffu, bits);
  const uint32_t e = max(bits >> 23, 30u);
  const float scale = __uint_as_float((283u - e) << 23);         // 2^(29 - (e - 127)): |x| * scale < 2^30
  constexpr uint32_t kBelow = std::is_same<T, float>::value ? 8 : 14;
  const uint32_t low = (e - kBelow) << 23;
  const uint32_t lanes = __ballot_sync(0xffffffffu, least < low);        // with a value below, zeros among them
  uint32_t z[2][4], p[2][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    z[i >> 2][i & 3] = (uint32_t(__float2int_rn(f[i] * scale)) + 0x00808080u) ^ 0x00808080u;     // signed digits in [-128, 127], the top one in [-64, 64]
  transpose4(z[0], p[0]);
  transpose4(z[1], p[1]);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if constexpr (sub16<QT>()) {
      const int hb = lane >> 4, quad = (lane >> 2) & 3, u = (lane >> 1) & 1, t = 2 * (lane & 1);
      uint8_t* dst = xp + hb * 512 + c * 128 + u * 64 + t * 16 + quad * 4;
      *reinterpret_cast<uint32_t*>(dst) = p[0][c];
      *reinterpret_cast<uint32_t*>(dst + 16) = p[1][c];
    } else if constexpr (QT == QTYPE_Q4_0) {
      const int j = lane >> 2, half = (lane >> 1) & 1, t = 2 * (lane & 1);
      uint8_t* dst = xp + (j >> 1) * 256 + c * 64 + t * 16 + (j & 1) * 8 + half * 4;
      *reinterpret_cast<uint32_t*>(dst) = p[0][c];
      *reinterpret_cast<uint32_t*>(dst + 16) = p[1][c];
    } else {
      const int j = lane >> 2, t = lane & 3;
      *reinterpret_cast<uint2*>(xp + (j >> 1) * 256 + c * 64 + t * 16 + (j & 1) * 8) = make_uint2(p[0][c], p[1][c]);
    }
  }
  // largest value from 2^-97 (its last digit is 2^-126, the smallest normal number) to 2^100 (sums over a super-block stay finite), or zero;
  // looked at last, beside the stores: whatever planes a scale of zero has, they add nothing
  bool fits = bits - 0x0f000000u < 0x71800000u - 0x0f000000u || bits == 0u;
  if (__builtin_expect(__popc(lanes) > 8, 0)) {                  // else a quarter of the values at most
    uint32_t count = 0;                                          // values that are not zero, and (high half) those of them that lie below
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t magnitude = __float_as_uint(f[i]) & 0x7fffffffu;
      count += magnitude == 0u ? 0u : magnitude < low ? 0x10001u : 1u;
    }
    count = __reduce_add_sync(0xffffffffu, count);
    fits = fits && 4 * (count >> 16) <= (count & 0xffffu);
  }
  if (lane == 0) *xs = fits ? __uint_as_float((e - 29u) << 23) : 0.f;
  if constexpr (has_mins<QT>()) {
    if (!fits) sum = 0.f;
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if constexpr (sub16<QT>()) {
      if ((lane & 1) == 0) X[lane >> 1] = sum;
    } else {
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if ((lane & 3) == 0) X[lane >> 2] = sum;
    }
  }
}

// ---- one super-block of 16 weight rows on one warp
__device__ __forceinline__ float u8_float(uint32_t word, int i) { return float((word >> (8 * i)) & 0xffu); }      // one conversion with byte select
// 32-bit word at an even shared-memory address.  PHASE 0: word aligned, 2: two bytes off, -1: decided per address.
template <int PHASE>
__device__ __forceinline__ uint32_t word(const uint8_t* p) {
  if (PHASE == 0) return *reinterpret_cast<const uint32_t*>(p);
  if (PHASE == 2) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - 2);
    return __byte_perm(q[0], q[1], 0x5432);
  }
  const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (a & 2u));
  return __funnelshift_r(q[0], q[1], 8u * (a & 2u));
}
template <int PHASE>
__device__ __forceinline__ uint2 word2(const uint8_t* p) {       // two consecutive words
  if (PHASE == 0) return make_uint2(*reinterpret_cast<const uint32_t*>(p), *reinterpret_cast<const uint32_t*>(p + 4));
  const uint32_t off = PHASE == 2 ? 2u : (uint32_t(__cvta_generic_to_shared(p)) & 2u);
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p - off);
  const uint32_t w0 = q[0], w1 = q[1], w2 = q[2];
  if (PHASE == 2) return make_uint2(__byte_perm(w0, w1, 0x5432), __byte_perm(w1, w2, 0x5432));
  return make_uint2(__funnelshift_r(w0, w1, 8u * off), __funnelshift_r(w1, w2, 8u * off));
}

// bs: the block of row lane/2 (this lane decodes half of its scales); b0, b1: the blocks of rows lane/4 and lane/4 + 8 (its MMA
// rows).  ODD: these addresses are two bytes off a word boundary (types of 2-byte aligned blocks); RAG: each row has its own phase.
// xp / xs / X: digit planes, scales and sums of this super-block for activation row 0; row 1 follows at the given strides.
// blocks: valid 32-weight blocks of this super-block (8 except at the end of a row whose K is not a multiple of 256).
// res[0], res[1]: sums of rows lane/4 and lane/4 + 8 over this lane's two digits; xt: folded mins of row lane/2.
// Returns the scale of this lane's activation row.
template <int QT, int MXC, bool ODD, bool RAG>
__device__ __forceinline__ float superblock(const uint8_t* bs, const uint8_t* b0, const uint8_t* b1, float (*sS)[sub16<QT>() ? kScalePitch : 8], const uint8_t* xp,
                                           int xp_stride, const float* xs, int xs_stride, const float* X, int X_stride, int blocks, int lane,
                                           float (&res)[2], float (&xt)[MXC]) {
  constexpr int PH = RAG ? -1 : ODD ? 2 : 0;
  const int g = lane >> 2, t = lane & 3, shalf = lane & 1;
  float* srow = sS[lane >> 1];
  // ---- scales (and mins) of row lane/2, half of them per lane
  if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
    const uint4 hdr = *reinterpret_cast<const uint4*>(bs);
    const float d = half_bits_to_float(uint16_t(hdr.x & 0xffffu)), dmin = half_bits_to_float(uint16_t(hdr.x >> 16));
    // sub-blocks 0..3 keep their 6-bit fields in place; 4..7 are split across two bytes
    const uint32_t scb = shalf ? ((hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u)) : (hdr.y & 0x3f3f3f3fu);
    const uint32_t mnb = shalf ? (((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)) : (hdr.z & 0x3f3f3f3fu);
    const float dh = QT == QTYPE_Q4_K ? d * 0.0625f : d;         // Q4_K: the operands of the high nibbles are 16 q
    *reinterpret_cast<float4*>(srow + 4 * shalf) =
        make_float4(d * u8_float(scb, 0), dh * u8_float(scb, 1), d * u8_float(scb, 2), dh * u8_float(scb, 3));
#pragma unroll
    for (int c = 0; c < MXC; ++c) {
      const float4 S = *reinterpret_cast<const float4*>(X + c * X_stride + 4 * shalf);
      float mn = u8_float(mnb, 0) * S.x;
      mn = fmaf(u8_float(mnb, 1), S.y, mn);
      mn = fmaf(u8_float(mnb, 2), S.z, mn);
      mn = fmaf(u8_float(mnb, 3), S.w, mn);
      xt[c] = fmaf(dmin, mn, xt[c]);
    }
  } else if constexpr (QT == QTYPE_Q8_0 || QT == QTYPE_Q4_0) {
    constexpr int BB = QT == QTYPE_Q8_0 ? 34 : 18;
    constexpr float kUnit = QT == QTYPE_Q8_0 ? 1.f : 0.0625f;    // Q4_0: the operands are 16 (q - 8)
    float d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = 4 * shalf + i;
      d[i] = half_bits_to_float(*reinterpret_cast<const uint16_t*>(bs + BB * b)) * kUnit;
      if (RAG && b >= blocks) d[i] = 0.f;                         // past the end of the row: whatever the stage holds
    }
    *reinterpret_cast<float4*>(srow + 4 * shalf) = make_float4(d[0], d[1], d[2], d[3]);
  } else {
    // 16-weight sub-blocks: half-block shalf, scale index 8 shalf + 2 quad + u, stored [half][u][quad]
    float sc[8];
    if constexpr (QT == QTYPE_Q6_K) {
      const float d = half_bits_to_float(*reinterpret_cast<const uint16_t*>(bs + 208)) * 0.25f;      // the operands are 4 (q - 32)
      const uint2 w = word2<PH>(bs + 192 + 8 * shalf);
      const uint32_t s0 = w.x ^ 0x80808080u, s1 = w.y ^ 0x80808080u;                               // int8 + 128 as unsigned bytes
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[i] = d * (u8_float(s0, i) - 128.f);
        sc[4 + i] = d * (u8_float(s1, i) - 128.f);
      }
    } else if constexpr (QT == QTYPE_Q2_K) {
      const uint32_t dd = *reinterpret_cast<const uint32_t*>(bs + 80);
      const float d = half_bits_to_float(uint16_t(dd & 0xffffu)), dmin = half_bits_to_float(uint16_t(dd >> 16));
      const uint32_t* scp = reinterpret_cast<const uint32_t*>(bs + 8 * shalf);                       // word aligned, not more
      const uint32_t s0 = scp[0], s1 = scp[1];
      const uint32_t l0 = s0 & 0x0f0f0f0fu, l1 = s1 & 0x0f0f0f0fu, m0 = (s0 >> 4) & 0x0f0f0f0fu, m1 = (s1 >> 4) & 0x0f0f0f0fu;
      constexpr float kUnit[4] = {1.f, 0.25f, 0.0625f, 0.015625f};                                   // quad j's operands are 4^j q
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[i] = (d * kUnit[i >> 1]) * u8_float(l0, i);
        sc[4 + i] = (d * kUnit[2 + (i >> 1)]) * u8_float(l1, i);
      }
#pragma unroll
      for (int c = 0; c < MXC; ++c) {
        const float4 S0 = *reinterpret_cast<const float4*>(X + c * X_stride + 8 * shalf), S1 = *reinterpret_cast<const float4*>(X + c * X_stride + 8 * shalf + 4);
        float mn = u8_float(m0, 0) * S0.x;
        mn = fmaf(u8_float(m0, 1), S0.y, mn);
        mn = fmaf(u8_float(m0, 2), S0.z, mn);
        mn = fmaf(u8_float(m0, 3), S0.w, mn);
        mn = fmaf(u8_float(m1, 0), S1.x, mn);
        mn = fmaf(u8_float(m1, 1), S1.y, mn);
        mn = fmaf(u8_float(m1, 2), S1.z, mn);
        mn = fmaf(u8_float(m1, 3), S1.w, mn);
        xt[c] = fmaf(dmin, mn, xt[c]);
      }
    } else {                                                        // Q3_K: the operands are 32 (q - 4)
      const float d = half_bits_to_float(*reinterpret_cast<const uint16_t*>(bs + 108)) * 0.03125f;
      // 6-bit scale 8 shalf + i: low nibble in byte i (the high half of it for shalf = 1), two high bits in byte 8 + i % 4 at bit 2 (2 shalf + i / 4)
      const uint2 lw = word2<PH>(bs + 96);
      const uint32_t hw = word<PH>(bs + 104) >> (4 * shalf);
      const uint32_t s0 = ((lw.x >> (4 * shalf)) & 0x0f0f0f0fu) | ((hw & 0x03030303u) << 4);
      const uint32_t s1 = ((lw.y >> (4 * shalf)) & 0x0f0f0f0fu) | (((hw >> 2) & 0x03030303u) << 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[i] = d * (u8_float(s0, i) - 32.f);
        sc[4 + i] = d * (u8_float(s1, i) - 32.f);
      }
    }
    *reinterpret_cast<float4*>(srow + 8 * shalf) = make_float4(sc[0], sc[2], sc[4], sc[6]);
    *reinterpret_cast<float4*>(srow + 8 * shalf + 4) = make_float4(sc[1], sc[3], sc[5], sc[7]);
  }
  __syncwarp();
  const float row_scale = xs[MXC == 2 ? (t >> 1) * xs_stride : 0], lane_scale = row_scale * ((t & 1) ? 65536.f : 1.f);
  const uint8_t* px = xp + (MXC == 2 ? (g >> 2) * xp_stride : 0);
  float sum0 = 0.f, sum1 = 0.f;
  auto apply = [&](const int (&c)[4], float s0, float s1) {
    sum0 = fmaf(s0, float(c[1] * 256 + c[0]), sum0);
    sum1 = fmaf(s1, float(c[3] * 256 + c[2]), sum1);
  };
  if constexpr (sub16<QT>()) {
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
      // words of this lane: weights 4t .. 4t+3 of the two 16-weight runs u, all quads in the same bytes
      uint32_t wa[2][2], wb[2][2], ha[2], hb_[2];                   // [u][..]: Q6_K: ql of quads 0/2, 1/3; else the quants; ha / hb_: the high bits
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int l = 16 * u + 4 * t;
        if constexpr (QT == QTYPE_Q6_K) {
          wa[u][0] = word<PH>(b0 + 64 * hb + l); wa[u][1] = word<PH>(b0 + 64 * hb + 32 + l);
          wb[u][0] = word<PH>(b1 + 64 * hb + l); wb[u][1] = word<PH>(b1 + 64 * hb + 32 + l);
          ha[u] = word<PH>(b0 + 128 + 32 * hb + l) ^ 0xaaaaaaaau;    // the top bit of every two-bit field flipped: 4 (q - 32) as int8
          hb_[u] = word<PH>(b1 + 128 + 32 * hb + l) ^ 0xaaaaaaaau;
        } else if constexpr (QT == QTYPE_Q2_K) {
          wa[u][0] = word<PH>(b0 + 16 + 32 * hb + l);
          wb[u][0] = word<PH>(b1 + 16 + 32 * hb + l);
        } else {
          wa[u][0] = word<PH>(b0 + 32 + 32 * hb + l);
          wb[u][0] = word<PH>(b1 + 32 + 32 * hb + l);
          ha[u] = word<PH>(b0 + l) ^ 0xffffffffu;                    // third bit inverted: 32 (q - 4) as int8
          hb_[u] = word<PH>(b1 + l) ^ 0xffffffffu;
        }
      }
      auto operand = [&](const uint32_t (&w)[2], uint32_t h, int quad) -> uint32_t {
        if constexpr (QT == QTYPE_Q6_K) {
          const uint32_t lw = w[quad & 1], l4 = ((quad & 2) ? lw >> 2 : lw << 2) & 0x3c3c3c3cu;
          const uint32_t hs = quad == 0 ? h << 6 : quad == 1 ? h << 4 : quad == 2 ? h << 2 : h;
          return l4 | (hs & 0xc0c0c0c0u);
        } else if constexpr (QT == QTYPE_Q2_K) {
          return w[0] & (0x03030303u << (2 * quad));
        } else {
          const int bit = 4 * hb + quad;
          const uint32_t low = (quad == 3 ? w[0] >> 1 : w[0] << (5 - 2 * quad)) & 0x60606060u;
          return low | ((h << (7 - bit)) & 0x80808080u);
        }
      };
      constexpr bool kSigned = QT != QTYPE_Q2_K;
      if constexpr (MXC == 1) {
        // columns 0..3 take the digits of run u = 0, columns 4..7 those of run 1: one K = 32 MMA, lanes t < 2 get sub-block u = 0
        const int u = g >> 2;
        const uint4 xv = *reinterpret_cast<const uint4*>(px + hb * 512 + (g & 3) * 128 + u * 64 + t * 16);
        const float4 s0 = *reinterpret_cast<const float4*>(&sS[g][8 * hb + 4 * (t >> 1)]), s1 = *reinterpret_cast<const float4*>(&sS[g + 8][8 * hb + 4 * (t >> 1)]);
        const uint32_t xq[4] = {xv.x, xv.y, xv.z, xv.w};
        const float f0[4] = {s0.x, s0.y, s0.z, s0.w}, f1[4] = {s1.x, s1.y, s1.z, s1.w};
#pragma unroll
        for (int quad = 0; quad < 4; ++quad) {
          int c[4];
          mma32<kSigned>(c, operand(wa[0], ha[0], quad), operand(wb[0], hb_[0], quad), operand(wa[1], ha[1], quad), operand(wb[1], hb_[1], quad),
                         u == 0 ? xq[quad] : 0u, u == 0 ? 0u : xq[quad]);
          apply(c, f0[quad], f1[quad]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint4 xv = *reinterpret_cast<const uint4*>(px + hb * 512 + (g & 3) * 128 + u * 64 + t * 16);
          const float4 s0 = *reinterpret_cast<const float4*>(&sS[g][8 * hb + 4 * u]), s1 = *reinterpret_cast<const float4*>(&sS[g + 8][8 * hb + 4 * u]);
          const uint32_t xq[4] = {xv.x, xv.y, xv.z, xv.w};
          const float f0[4] = {s0.x, s0.y, s0.z, s0.w}, f1[4] = {s1.x, s1.y, s1.z, s1.w};
#pragma unroll
          for (int quad = 0; quad < 4; ++quad) {
            int c[4];
            mma16<kSigned>(c, operand(wa[u], ha[u], quad), operand(wb[u], hb_[u], quad), xq[quad]);
            apply(c, f0[quad], f1[quad]);
          }
        }
      }
    }
  } else {
    const float4 s0a = *reinterpret_cast<const float4*>(&sS[g][0]), s0b = *reinterpret_cast<const float4*>(&sS[g][4]);
    const float4 s1a = *reinterpret_cast<const float4*>(&sS[g + 8][0]), s1b = *reinterpret_cast<const float4*>(&sS[g + 8][4]);
    const float f0[8] = {s0a.x, s0a.y, s0a.z, s0a.w, s0b.x, s0b.y, s0b.z, s0b.w}, f1[8] = {s1a.x, s1a.y, s1a.z, s1a.w, s1b.x, s1b.y, s1b.z, s1b.w};
    uint2 qh0 = make_uint2(0u, 0u), qh1 = make_uint2(0u, 0u);
    if constexpr (QT == QTYPE_Q5_K) {                               // bit j of qh byte l: fifth bit of weight l of sub-block j
      qh0 = *reinterpret_cast<const uint2*>(b0 + 16 + 8 * t);
      qh1 = *reinterpret_cast<const uint2*>(b1 + 16 + 8 * t);
    }
#pragma unroll
    for (int G = 0; G < 4; ++G) {
      const uint4 xv = *reinterpret_cast<const uint4*>(px + G * 256 + (g & 3) * 64 + t * 16);
      if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
        constexpr int kQs = QT == QTYPE_Q4_K ? 16 : 48;
        const uint2 q0 = *reinterpret_cast<const uint2*>(b0 + kQs + 8 * t + 32 * G), q1 = *reinterpret_cast<const uint2*>(b1 + kQs + 8 * t + 32 * G);
        auto low = [&](uint32_t q, uint32_t h) -> uint32_t {
          const uint32_t v = q & 0x0f0f0f0fu;
          if constexpr (QT == QTYPE_Q4_K) return v;
          return v | ((2 * G < 4 ? h << (4 - 2 * G) : h >> (2 * G - 4)) & 0x10101010u);
        };
        auto high = [&](uint32_t q, uint32_t h) -> uint32_t {
          if constexpr (QT == QTYPE_Q4_K) return q & 0xf0f0f0f0u;   // 16 q
          return ((q >> 4) & 0x0f0f0f0fu) | ((2 * G + 1 < 4 ? h << (3 - 2 * G) : h >> (2 * G - 3)) & 0x10101010u);
        };
        int c[4];
        mma32<false>(c, low(q0.x, qh0.x), low(q1.x, qh1.x), low(q0.y, qh0.y), low(q1.y, qh1.y), xv.x, xv.y);
        apply(c, f0[2 * G], f1[2 * G]);
        mma32<false>(c, high(q0.x, qh0.x), high(q1.x, qh1.x), high(q0.y, qh0.y), high(q1.y, qh1.y), xv.z, xv.w);
        apply(c, f0[2 * G + 1], f1[2 * G + 1]);
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {                               // blocks 2G, 2G + 1; their payload starts 2 bytes in, at the other phase for odd blocks
          const int j = 2 * G + h;
          int c[4];
          if constexpr (QT == QTYPE_Q8_0) {
            constexpr int kPh[2] = {RAG ? -1 : 2, RAG ? -1 : 0};
            const uint2 q0 = h == 0 ? word2<kPh[0]>(b0 + 34 * j + 2 + 8 * t) : word2<kPh[1]>(b0 + 34 * j + 2 + 8 * t);
            const uint2 q1 = h == 0 ? word2<kPh[0]>(b1 + 34 * j + 2 + 8 * t) : word2<kPh[1]>(b1 + 34 * j + 2 + 8 * t);
            mma32<true>(c, q0.x, q1.x, q0.y, q1.y, h == 0 ? xv.x : xv.z, h == 0 ? xv.y : xv.w);
          } else {
            constexpr int kPh[2] = {RAG ? -1 : 2, RAG ? -1 : 0};
            const uint32_t q0 = h == 0 ? word<kPh[0]>(b0 + 18 * j + 2 + 4 * t) : word<kPh[1]>(b0 + 18 * j + 2 + 4 * t);
            const uint32_t q1 = h == 0 ? word<kPh[0]>(b1 + 18 * j + 2 + 4 * t) : word<kPh[1]>(b1 + 18 * j + 2 + 4 * t);
            // (q - 8) as a 4-bit two's complement number in the upper half of a byte: 16 (q - 8)
            mma32<true>(c, ((q0 << 4) ^ 0x80808080u) & 0xf0f0f0f0u, ((q1 << 4) ^ 0x80808080u) & 0xf0f0f0f0u, (q0 ^ 0x80808080u) & 0xf0f0f0f0u,
                        (q1 ^ 0x80808080u) & 0xf0f0f0f0u, h == 0 ? xv.x : xv.z, h == 0 ? xv.y : xv.w);
          }
          apply(c, f0[j], f1[j]);
        }
      }
    }
  }
  res[0] = fmaf(lane_scale, sum0, res[0]);
  res[1] = fmaf(lane_scale, sum1, res[1]);
  return row_scale;
}

// The same super-block weight by weight, as the dequantizer gives them, for activations without planes: what this lane adds to its two
// sums.  Added up in fp64, so that the result is no further off than by planes.  Q4_K [11008 x 4096], M = 1: 34 us with every super-block
// this way, 15.6 us with one of sixteen, 7.9 us with none.
// b0, b1 as above; x: the super-block of this lane's activation row, `valid` values of it; mine: whether that row has no planes here.  All
// lanes call it.
template <int QT, typename T, int MXC>
__device__ __noinline__ float2 plain(const uint8_t* b0, const uint8_t* b1, const T* x, int valid, bool mine, int t) {
  constexpr int kUnits = QTraits<QT>::kBlock / 8;                 // of eight weights, dealt to the lanes that share the row
  double sum[2] = {0., 0.};
  for (int u = MXC == 2 ? t & 1 : t; 8 * u < valid; u += MXC == 2 ? 2 : 4) {
    float f[8], w[8];
    load8<T>(x + 8 * u, f);
    decode8<QT>(b0 + u / kUnits * QTraits<QT>::kBytes, 8 * (u % kUnits), w);
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[0] = fma(double(f[i]), double(w[i]), sum[0]);
    decode8<QT>(b1 + u / kUnits * QTraits<QT>::kBytes, 8 * (u % kUnits), w);
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[1] = fma(double(f[i]), double(w[i]), sum[1]);
  }
  if (MXC == 1) {                                                 // join() counts lanes t = 0, 1
    sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 2);
    sum[1] += __shfl_xor_sync(0xffffffffu, sum[1], 2);
    mine = mine && t < 2;
  }
  return mine ? make_float2(float(sum[0]), float(sum[1])) : make_float2(0.f, 0.f);
}

// Sums of rows lane/4 and lane/4 + 8 over the digit lanes: afterwards lane t = 0 holds row 0's results (and lane t = 2 row 1's).
template <int QT, int MXC>
__device__ __forceinline__ void join(float (&res)[2]) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    res[r] += __shfl_xor_sync(0xffffffffu, res[r], 1);
    if (MXC == 1 && sub16<QT>()) res[r] += __shfl_xor_sync(0xffffffffu, res[r], 2);      // the two runs u of every sub-block pair
  }
}

}  // namespace planes
}  // namespace b200gguf
