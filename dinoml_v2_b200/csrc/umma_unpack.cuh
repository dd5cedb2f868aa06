// Packed weights -> 16-bit UMMA operand values, half a super-block (128 weights of one row) per thread: every packed byte, scale and
// header field is read by the one thread that needs it, and the barriers around it are passed once per 128 weights.
#pragma once
#include "umma_frame.cuh"

namespace b200gguf {
namespace umma {

// 4 quant bytes (values 0..255, here < 64) -> two pairs of (value - offset) * scale [+ addend].
template <typename T>
__device__ __forceinline__ void bytes_to_pairs(uint32_t u, typename Pair<T>::V off, typename Pair<T>::V scale, typename Pair<T>::V add, uint32_t* p) {
  using V = typename Pair<T>::V;
  const V a = __hsub2(as_pair<V>(__byte_perm(u, Pair<T>::kMagicBytes, 0x4140)), off);
  const V b = __hsub2(as_pair<V>(__byte_perm(u, Pair<T>::kMagicBytes, 0x4342)), off);
  p[0] = as_u32<V>(__hfma2(a, scale, add));
  p[1] = as_u32<V>(__hfma2(b, scale, add));
}

// N words starting S*2 bytes past a 16-byte aligned shared address.  Blocks of 210, 110, 84 .. bytes sit at one of 8 byte phases
// inside the staged window; S is that phase (uniform across a warp: the weight rows are 16-byte multiples).
template <int N, int S>
__device__ __forceinline__ void fetch(const uint8_t* aligned, uint32_t* out) {
  constexpr int kChunks = (4 * N + 2 * S + 15) / 16, j = S >> 1;
  uint32_t w[4 * kChunks + 1];
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const uint4 v = *reinterpret_cast<const uint4*>(aligned + 16 * c);
    w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
  }
  w[4 * kChunks] = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] = (S & 1) ? __funnelshift_r(w[j + i], w[j + i + 1], 16) : w[j + i];
}

// Packed super-block window in shared memory: the 16-byte aligned span that contains one block of every row.
// Q4_K blocks (144 B) are always aligned; a Q6_K block (210 B) starts 0..14 bytes into its window and the last
// field read (d, through a fetch at +192) ends before byte 240.  Eight Q8_0 blocks (272 B per 256 weights, always
// 16-byte aligned) are wider than a TMA box may be (256 elements), so they travel as two boxes of 144 B: blocks 0..3
// start at byte 0 of the first, blocks 4..7 at byte 8 of the second (which starts at byte 128 of the 272).  Every pitch
// is an odd number of 16-byte chunks, so 16-byte reads of 8 consecutive rows hit all 32 banks.
//   kSuper: packed bytes per 256 weights of a row; kBoxes: TMA boxes per super-block, one behind the other in its ring slot.
template <int QT> struct RawGeom;
template <> struct RawGeom<QTYPE_Q4_K> { static constexpr int kPitch = 144, kSuper = 144, kBoxes = 1; };
template <> struct RawGeom<QTYPE_Q5_K> { static constexpr int kPitch = 176, kSuper = 176, kBoxes = 1; };   // Q4_K + 32 bytes of fifth bits
template <> struct RawGeom<QTYPE_Q6_K> { static constexpr int kPitch = 240, kSuper = 210, kBoxes = 1; };
template <> struct RawGeom<QTYPE_Q8_0> { static constexpr int kPitch = 144, kSuper = 272, kBoxes = 2; };
template <> struct RawGeom<QTYPE_Q4_0> { static constexpr int kPitch = 144, kSuper = 144, kBoxes = 1; };   // 8 blocks of 18 B
template <> struct RawGeom<QTYPE_MXFP4> { static constexpr int kPitch = 144, kSuper = 136, kBoxes = 1; };  // 8 x 17 B, starts 0 / 8 bytes into its window
template <> struct RawGeom<QTYPE_Q2_K> { static constexpr int kPitch = 112, kSuper = 84, kBoxes = 1; };    // starts 0 / 4 / 8 / 12 bytes into its window
template <> struct RawGeom<QTYPE_Q3_K> { static constexpr int kPitch = 144, kSuper = 110, kBoxes = 1; };   // any even phase, like Q6_K
template <> struct RawGeom<QTYPE_NVFP4> { static constexpr int kPitch = 144, kSuper = 144, kBoxes = 1; };  // 4 blocks of 36 B

// FP4 (e2m1) codes -> 16-bit operand values, exactly.  A code s|ee|m placed on the sign bit, the two lowest exponent
// bits and the top mantissa bit of a 16-bit float IS that format's own number e2m1 * 2^(1 - bias): its subnormals give
// the codes 0 and 0.5.  Two exact multiplies follow: by k1 (which lifts the value into the normal range) and by the
// block scale.  e2m1 has 2 significant bits, an e8m0 scale none and a ue4m3 scale 4: the product is exact in either
// 16-bit type while it stays in range.  w = 4 bytes; lo / hi = the values of their low / high nibbles as two pairs.
template <typename T>
__device__ __forceinline__ void fp4_to_pairs(uint32_t w, typename Pair<T>::V k1, typename Pair<T>::V lo_scale, typename Pair<T>::V hi_scale, uint32_t* lo, uint32_t* hi) {
  using P = Pair<T>;
  using V = typename P::V;
  constexpr uint32_t kMag = (7u << P::kFp4MagPos) * 0x00010001u;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t t = __byte_perm(w, 0u, j == 0 ? 0x1404u : 0x3424u);   // bytes 2j, 2j+1 on bits 8..15 / 24..31
    // low nibble: sign on bit 11, magnitude on bits 8..10; high nibble: sign on bit 15, magnitude on bits 12..14
    uint32_t lmag;
    if constexpr (P::kFp4MagPos >= 8) lmag = t << (P::kFp4MagPos - 8); else lmag = t >> (8 - P::kFp4MagPos);
    const uint32_t l = ((t << 4) & 0x80008000u) | (lmag & kMag);
    const uint32_t h = (t & 0x80008000u) | ((t >> (12 - P::kFp4MagPos)) & kMag);
    lo[j] = as_u32<V>(__hmul2(__hmul2(as_pair<V>(l), k1), lo_scale));
    hi[j] = as_u32<V>(__hmul2(__hmul2(as_pair<V>(h), k1), hi_scale));
  }
}
// ue4m3 scale byte (NVFP4) times `mult`, where mult carries 2^120: the byte placed on exponent / mantissa bits of a float
// is value * 2^-120 (fp32 subnormals give the ue4m3 subnormals).  0x7f decodes to 0 as in the reference's host code.
__device__ __forceinline__ float ue4m3_times(uint32_t x, float mult) {
  x &= 0xffu;
  return x == 0x7fu ? 0.f : __fmul_rn(__uint_as_float((x & 0x7fu) << 20), mult);
}
// 4 int8 quants -> two 16-bit pairs of q * d, each rounded once.  With u = q + 128 in byte 1 of a float's mantissa,
// f = 2^23 + 256 u, and f * (d / 256) - (2^23 + 2^15) * (d / 256) = q * d with every term exact in fp32.
template <typename T>
__device__ __forceinline__ void q8_to_pairs(uint32_t u, float d256, float c, uint32_t* p) {
  using P = Pair<T>;
  const uint32_t v = u ^ 0x80808080u;
  const float f0 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7404));
  const float f1 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7414));
  const float f2 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7424));
  const float f3 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7434));
  p[0] = as_u32<typename P::V>(P::pack(fmaf(f0, d256, c), fmaf(f1, d256, c)));
  p[1] = as_u32<typename P::V>(P::pack(fmaf(f2, d256, c), fmaf(f3, d256, c)));
}

// Half `hb` of a super-block of one row.  load() copies its packed words to registers (part p of kLoads before groups 4 p / kLoads on), from
// the row's window of the staged bytes; group(i): weights 32 i .. 32 i + 31 as 16 pairs.
template <int QT, typename T> struct Half {
  using P = Pair<T>;
  using V = typename P::V;
  static constexpr int kLoads = QT == QTYPE_Q8_0 ? 2 : 1, kSuper = RawGeom<QT>::kSuper;
  static constexpr bool kRuns = QT == QTYPE_Q6_K || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K;
  static constexpr bool kHigh = QT == QTYPE_Q5_K || QT == QTYPE_Q6_K || QT == QTYPE_Q3_K;
  uint32_t q[QT == QTYPE_NVFP4 ? 18 : QT == QTYPE_Q2_K || QT == QTYPE_Q3_K ? 8 : 16], h[kHigh ? 8 : 1];
  uint32_t sc[QT == QTYPE_Q3_K ? 3 : QT == QTYPE_Q4_0 || QT == QTYPE_MXFP4 ? 4 : 2];
  float d, dmin;
  int half;

  template <int S> __device__ __forceinline__ void load_runs(const uint8_t* row, int hb) {      // the types of even byte phases
    if constexpr (QT == QTYPE_Q6_K) {          // ql[128], qh[64], 16 int8 scales, d
      uint32_t tail[5];
      fetch<16, S>(row + 64 * hb, q);
      fetch<8, S>(row + 128 + 32 * hb, h);
      fetch<5, S>(row + 192, tail);
      sc[0] = hb ? tail[2] : tail[0];
      sc[1] = hb ? tail[3] : tail[1];
      d = half_bits_to_float(uint16_t(tail[4] & 0xffffu));
    } else if constexpr (QT == QTYPE_Q2_K) {   // scales[16], qs[64], d, dmin
      uint32_t head[4], tail[1];
      fetch<8, S>(row + 16 + 32 * hb, q);
      fetch<4, S>(row, head);
      fetch<1, S>(row + 80, tail);
      sc[0] = hb ? head[2] : head[0];
      sc[1] = hb ? head[3] : head[1];
      d = half_bits_to_float(uint16_t(tail[0] & 0xffffu));
      dmin = half_bits_to_float(uint16_t(tail[0] >> 16));
    } else {                                   // Q3_K: hmask[32], qs[64], 12 scale bytes, d
      uint32_t tail[4];
      fetch<8, S>(row + 32 + 32 * hb, q);
      fetch<8, S>(row, h);
      fetch<4, S>(row + 96, tail);
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] >>= 4 * hb;             // the third bits of this half on bits 0..3
      // 6-bit scale number 8 hb + 2 j + u: low nibble in byte 2 j + u (its high half for hb = 1), the two high bits in byte 8 + 2 (j % 2) + u
      // at bit 2 (2 hb + j / 2)
      sc[0] = ((tail[0] >> (4 * hb)) & 0x0f0f0f0fu) | (((tail[2] >> (4 * hb)) & 0x03030303u) << 4);
      sc[1] = ((tail[1] >> (4 * hb)) & 0x0f0f0f0fu) | (((tail[2] >> (4 * hb + 2)) & 0x03030303u) << 4);
      d = half_bits_to_float(uint16_t(tail[3] & 0xffffu));
    }
  }
  template <int R0> __device__ __forceinline__ void load_blocks(const uint8_t* base) {          // Q4_0, MXFP4: four blocks from byte R0 on
    constexpr int BB = QTraits<QT>::kBytes, kWords = (R0 + 4 * BB + 15) / 16 * 4;
    uint32_t w[kWords + 1];
#pragma unroll
    for (int c = 0; c < kWords / 4; ++c) {
      const uint4 v = *reinterpret_cast<const uint4*>(base + 16 * c);
      w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
    }
    w[kWords] = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int oe = R0 + BB * b, o = oe + BB - 16, sh = 8 * (o & 3);
      sc[b] = w[oe >> 2] >> (8 * (oe & 3));
#pragma unroll
      for (int i = 0; i < 4; ++i) q[4 * b + i] = sh ? __funnelshift_r(w[(o >> 2) + i], w[(o >> 2) + i + 1], sh) : w[(o >> 2) + i];
    }
  }
  template <int B0> __device__ __forceinline__ void load_bytes(const uint8_t* box) {            // Q8_0: two blocks from byte B0 of the box on
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      constexpr int kAt0 = B0 + 2, kAt1 = B0 + 36;
      sc[b] = *reinterpret_cast<const uint16_t*>(box + B0 + 34 * b);
      if (b == 0) fetch<8, (kAt0 & 15) / 2>(box + (kAt0 & ~15), q); else fetch<8, (kAt1 & 15) / 2>(box + (kAt1 & ~15), q + 8);
    }
  }

  __device__ __forceinline__ void load(const uint8_t* row, int sb, int hb, int part) {
    half = hb;
    if constexpr (kRuns) {
      const int phase = ((sb * kSuper) & 15) >> 1;              // rows are 16-byte multiples: the same phase in every row
      if constexpr (QT == QTYPE_Q2_K) {
        switch (phase >> 1) {                                   // 84-byte blocks: multiples of four
          case 0: load_runs<0>(row, hb); break;
          case 1: load_runs<2>(row, hb); break;
          case 2: load_runs<4>(row, hb); break;
          default: load_runs<6>(row, hb); break;
        }
      } else {
        switch (phase) {
          case 0: load_runs<0>(row, hb); break;
          case 1: load_runs<1>(row, hb); break;
          case 2: load_runs<2>(row, hb); break;
          case 3: load_runs<3>(row, hb); break;
          case 4: load_runs<4>(row, hb); break;
          case 5: load_runs<5>(row, hb); break;
          case 6: load_runs<6>(row, hb); break;
          default: load_runs<7>(row, hb); break;
        }
      }
    } else if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
      const uint4 hdr = *reinterpret_cast<const uint4*>(row);
      d = half_bits_to_float(uint16_t(hdr.x & 0xffffu));
      dmin = half_bits_to_float(uint16_t(hdr.x >> 16));
      // sub-blocks 0..3 keep their 6-bit fields in place; 4..7 are split across two bytes
      sc[0] = hb ? (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3f3f3f3fu;
      sc[1] = hb ? ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u) : hdr.z & 0x3f3f3f3fu;
      fetch<16, 0>(row + (QT == QTYPE_Q5_K ? 48 : 16) + 64 * hb, q);
      if constexpr (QT == QTYPE_Q5_K) {       // bit 4 hb + i of qh byte l: fifth bit of weight l of group i
        fetch<8, 0>(row + 16, h);
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] >>= 4 * hb;
      }
    } else if constexpr (QT == QTYPE_Q8_0) {                    // row: of box hb
      if (hb == 0) { if (part == 0) load_bytes<0>(row); else load_bytes<68>(row); }
      else { if (part == 0) load_bytes<8>(row); else load_bytes<76>(row); }
    } else if constexpr (QT == QTYPE_NVFP4) {                   // two blocks of four ue4m3 scales and 32 bytes of nibbles, from byte 72 hb on
      if (hb == 0) fetch<18, 0>(row, q); else fetch<18, 4>(row + 64, q);
    } else {
      const int at = ((sb * kSuper) & 15) + 4 * QTraits<QT>::kBytes * hb;      // the half's four blocks start here in the window
      const uint8_t* base = row + (at & ~15);
      if constexpr (QT == QTYPE_Q4_0) {
        if (at & 15) load_blocks<8>(base); else load_blocks<0>(base);
      } else {
        switch (at & 15) {
          case 0: load_blocks<0>(base); break;
          case 4: load_blocks<4>(base); break;
          case 8: load_blocks<8>(base); break;
          default: load_blocks<12>(base); break;
        }
      }
    }
  }

  __device__ __forceinline__ float byte_of(uint32_t w, int i) const { return float((w >> (8 * i)) & 0xffu); }
  __device__ __forceinline__ void group(int i, uint32_t (&o)[16]) const {
    if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
      const V off = P::splat(P::kMagic), s = P::splat(d * byte_of(sc[0], i)), mn = P::splat(-(dmin * byte_of(sc[1], i)));
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t w = q[8 * (i >> 1) + k];
        uint32_t n = (i & 1 ? w >> 4 : w) & 0x0f0f0f0fu;
        if constexpr (QT == QTYPE_Q5_K) n |= (h[k] << (4 - i)) & 0x10101010u;
        bytes_to_pairs<T>(n, off, s, mn, o + 2 * k);
      }
    } else if constexpr (QT == QTYPE_Q6_K) {
      // quad i: ql bytes 0..31 (even) or 32..63 (odd) of the half, low or high nibbles; its two high bits at bit 2 i of the qh bytes
      const V off = P::splat(P::kMagic + 32.f), zero = P::splat(0.f);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const V s = P::splat(d * float(int(int8_t(sc[i >> 1] >> (8 * (2 * (i & 1) + u))))));
#pragma unroll
        for (int k = 4 * u; k < 4 * u + 4; ++k) {
          const uint32_t l4 = (q[8 * (i & 1) + k] >> (i & 2 ? 4 : 0)) & 0x0f0f0f0fu;
          const uint32_t hs = i == 0 ? h[k] << 4 : i == 1 ? h[k] << 2 : i == 2 ? h[k] : h[k] >> 2;
          bytes_to_pairs<T>(l4 | (hs & 0x30303030u), off, s, zero, o + 2 * k);
        }
      }
    } else if constexpr (QT == QTYPE_Q2_K || QT == QTYPE_Q3_K) {
      // bits 2 i, 2 i + 1 of the qs bytes; Q3_K: plus bit i of the mask bytes as a third bit, less 4
      const V off = P::splat(P::kMagic + (QT == QTYPE_Q3_K ? 4.f : 0.f));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t b = (sc[i >> 1] >> (8 * (2 * (i & 1) + u))) & 0xffu;
        V s, a;
        if constexpr (QT == QTYPE_Q2_K) { s = P::splat(d * float(b & 0x0fu)); a = P::splat(-(dmin * float(b >> 4))); }
        else { s = P::splat(d * float(int(b) - 32)); a = P::splat(0.f); }
#pragma unroll
        for (int k = 4 * u; k < 4 * u + 4; ++k) {
          uint32_t n = (q[k] >> (2 * i)) & 0x03030303u;
          if constexpr (QT == QTYPE_Q3_K) n |= (i <= 2 ? h[k] << (2 - i) : h[k] >> (i - 2)) & 0x04040404u;
          bytes_to_pairs<T>(n, off, s, a, o + 2 * k);
        }
      }
    } else if constexpr (QT == QTYPE_Q8_0) {
      const float d256 = half_bits_to_float(uint16_t(sc[i & 1])) * (1.f / 256.f);
      const float c = -8421376.f * d256;        // -(2^23 + 2^15) * d / 256, exact
#pragma unroll
      for (int k = 0; k < 8; ++k) q8_to_pairs<T>(q[8 * (i & 1) + k], d256, c, o + 2 * k);
    } else if constexpr (QT == QTYPE_Q4_0) {
      const V off = P::splat(P::kMagic + 8.f), zero = P::splat(0.f), s = P::splat(half_bits_to_float(uint16_t(sc[i] & 0xffffu)));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        bytes_to_pairs<T>(q[4 * i + k] & 0x0f0f0f0fu, off, s, zero, o + 2 * k);
        bytes_to_pairs<T>((q[4 * i + k] >> 4) & 0x0f0f0f0fu, off, s, zero, o + 8 + 2 * k);
      }
    } else if constexpr (QT == QTYPE_MXFP4) {
      const V k1 = P::splat(P::kFp4Up), s = P::splat(__fmul_rn(e8m0_half(sc[i] & 0xffu), 2.f * P::kFp4Rest));    // 2^(e - 127), less what k1 already gave
#pragma unroll
      for (int k = 0; k < 4; ++k) fp4_to_pairs<T>(q[4 * i + k], k1, s, s, o + 2 * k, o + 8 + 2 * k);
    } else {
      // NVFP4: sub-blocks 2 (i % 2), + 1 of block i / 2: 8 bytes each, low nibbles = the first 8 weights
      const V k1 = P::splat(P::kFp4Up);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const V s = P::splat(ue4m3_times(q[9 * (i >> 1)] >> (8 * (2 * (i & 1) + u)), 0x1p120f * P::kFp4Rest));
#pragma unroll
        for (int k = 0; k < 2; ++k) fp4_to_pairs<T>(q[9 * (i >> 1) + 1 + 2 * (2 * (i & 1) + u) + k], k1, s, s, o + 8 * u + 2 * k, o + 8 * u + 4 + 2 * k);
      }
    }
  }
};

}  // namespace umma
}  // namespace b200gguf
