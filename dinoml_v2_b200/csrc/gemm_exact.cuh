// Fused GGUF gemm_rcr that rounds neither weights nor activations, from three rows on ("simt" family): C[M,N] = A[M,K] * dequant(W[N,K])^T
// (+ bias) for float32 activations and for weight rows that are not multiples of 16 bytes, on mma.sync tensor cores.
//
// The quants are small integers (FP4 codes small binary fractions), exact as 16-bit MMA operands.  A float32 activation is the exact
// sum of three bfloat16 numbers, one MMA each; a 16-bit activation is its own operand.  The MMA of a group of 16 weights (one K
// step) yields the exact products summed in fp32, and the group's scale and min are applied to that sum in fp32: no operand is rounded,
// as in the CUDA-core kernel this replaces (which reads the whole weight again for every four activation rows: Q6_K [4096 x 11008],
// M = 333: 2626 us).
//
// A CTA of 8 warps owns ROWS weight rows x BT activation rows and walks K in super-blocks of 256:
//   * packed bytes: every row's 16-byte aligned window around its super-block, 16-byte cp.async (rows have phases of their own);
//   * per half super-block each thread decodes 64 (or 32) weights of one row into the operand tile and its scales; the next
//     super-block's bytes are requested as soon as the second half is decoded;
//   * warps 4 x 2 take ROWS/4 x BT/2 of the tile with ldmatrix operands;
//   * with few tiles K is cut across a cluster of up to 8 CTAs whose sums meet through distributed shared memory.
// Two CTAs share an SM (< 113 KB each), so that one decodes while the other keeps the tensor pipe busy.
//
// A result that is not finite (or, with float32 activations, smaller than 2^-100) is computed again weight by weight: an infinite
// activation has no three parts, and a quant times an activation may leave the range of fp32 before the scale brings it back.
#pragma once
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "gemv_mma_common.cuh"

namespace b200gguf {
namespace stream { int sm_count(); }             // gemv_stream.cu

namespace exact {

constexpr int kThreads = 256;
constexpr int kHalfK = 128;                      // K per operand tile
constexpr int kPitchB = (kHalfK + 8) * 2;        // bytes of an operand row: 272, ldmatrix rows on distinct banks

template <int QT> constexpr int sb_bytes() { return 256 / QTraits<QT>::kBlock * QTraits<QT>::kBytes; }
template <int QT> constexpr int raw_pitch() { return (sb_bytes<QT>() + 15 + 15) / 16 * 16 + (((sb_bytes<QT>() + 30) / 16) % 2 == 0 ? 16 : 0); }   // an odd number of 16-byte chunks
template <int QT> constexpr bool has_mins() { return QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q2_K; }
template <typename T> using Operand = typename std::conditional<std::is_same<T, __half>::value, __half, __nv_bfloat16>::type;
template <typename T> constexpr int x_planes() { return std::is_same<T, float>::value ? 3 : 1; }

template <int QT, typename T, int ROWS, int BT> constexpr size_t smem_bytes() {
  return size_t(ROWS) * raw_pitch<QT>() + size_t(ROWS) * kPitchB + size_t(x_planes<T>()) * BT * kPitchB + size_t(8) * ROWS * sizeof(float) * (has_mins<QT>() ? 2 : 1) +
         (has_mins<QT>() ? size_t(8) * BT * sizeof(float) : 0);
}

// 16 consecutive bytes from any shared-memory address.
__device__ __forceinline__ void lds16(const uint8_t* p, uint32_t (&w)[4]) {
  const uint32_t off = uint32_t(__cvta_generic_to_shared(p)) & 3u;
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p - off);
  uint32_t v[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) v[i] = q[i];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(v[i], v[i + 1], 8u * off);
}

// Four unsigned bytes less an offset -> two operand pairs, exact (bytes below 128 for bfloat16, any for float16).
template <typename O>
__device__ __forceinline__ void bytes_minus(uint32_t w, int off, uint32_t& p01, uint32_t& p23) {
  const uint32_t a = __byte_perm(w, MmaType<O>::kMagicBytes, 0x4140), b = __byte_perm(w, MmaType<O>::kMagicBytes, 0x4342);
  if constexpr (std::is_same<O, __half>::value) {
    const __half2 o = __float2half2_rn(1024.f + float(off));
    const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&a), o), y = __hsub2(*reinterpret_cast<const __half2*>(&b), o);
    p01 = *reinterpret_cast<const uint32_t*>(&x);
    p23 = *reinterpret_cast<const uint32_t*>(&y);
  } else {
    const __nv_bfloat162 o = __float2bfloat162_rn(128.f + float(off));
    const __nv_bfloat162 x = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), o), y = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&b), o);
    p01 = *reinterpret_cast<const uint32_t*>(&x);
    p23 = *reinterpret_cast<const uint32_t*>(&y);
  }
}
template <typename O> __device__ __forceinline__ uint32_t pack(float lo, float hi) {
  if constexpr (std::is_same<O, __half>::value) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
// Offset of a type's quants as unsigned bytes: weight = scale * (byte - offset) - min.  FP4 codes become 12 + 2 * e2m1.
template <int QT> constexpr int byte_offset() {
  return QT == QTYPE_Q8_0 ? 128 : QT == QTYPE_Q6_K ? 32 : QT == QTYPE_Q4_0 ? 8 : QT == QTYPE_Q3_K ? 4 : (QT == QTYPE_MXFP4 || QT == QTYPE_NVFP4) ? 12 : 0;
}
// Four FP4 codes (low nibbles of the bytes, high nibbles zero) -> bytes 12 + 2 * e2m1: look-ups of the eight magnitudes, both signs.
__device__ __forceinline__ uint32_t fp4_bytes(uint32_t w) {
  const uint32_t mag = w & 0x07070707u;
  const uint32_t sel = __byte_perm(mag | (mag >> 4), 0u, 0x4420);
  const uint32_t pos = __byte_perm(0x0F0E0D0Cu, 0x18141210u, sel), neg = __byte_perm(0x090A0B0Cu, 0x00040608u, sel);
  const uint32_t sign = ((w >> 3) & 0x01010101u) * 0xffu;
  return (pos & ~sign) | (neg & sign);
}

// NJ groups of 16 weights of the super-block at p that lie 32 apart: weights 128 hb + 32 j + 16 u + 0..15, j = j0 .. j0 + NJ - 1 (NJ = 2 or 4,
// j0 = 0 or 2).  Each packed word is read once for all groups that it serves.
template <int QT, int NJ> struct Unit {
  static constexpr bool kHigh = QT == QTYPE_Q5_K || QT == QTYPE_Q6_K || QT == QTYPE_Q3_K;
  static constexpr int kWords = (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) ? NJ / 2 : QT == QTYPE_Q6_K ? 2 : (QT == QTYPE_Q2_K || QT == QTYPE_Q3_K) ? 1 : NJ;
  uint32_t w[kWords][4], h[kHigh ? 4 : 1];
  float scale[NJ], mn[NJ];
  int hb, j0, u;

  __device__ __forceinline__ void load(const uint8_t* p, int hb_, int j0_, int u_) {
    hb = hb_; j0 = j0_; u = u_;
#pragma unroll
    for (int i = 0; i < NJ; ++i) mn[i] = 0.f;
    if constexpr (QT == QTYPE_Q8_0) {
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const uint8_t* b = p + 34 * (4 * hb + j0 + i);
        scale[i] = half_at(b);
        lds16(b + 2 + 16 * u, w[i]);
      }
    } else if constexpr (QT == QTYPE_Q4_0 || QT == QTYPE_MXFP4) {
      constexpr int BB = QT == QTYPE_Q4_0 ? 18 : 17;
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const uint8_t* b = p + BB * (4 * hb + j0 + i);
        scale[i] = QT == QTYPE_Q4_0 ? half_at(b) : e8m0_half(b[0]);
        lds16(b + BB - 16, w[i]);
      }
    } else if constexpr (QT == QTYPE_NVFP4) {
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const uint8_t* b = p + 36 * (2 * hb + ((j0 + i) >> 1));
        const int sub = 2 * ((j0 + i) & 1) + u;
        scale[i] = ue4m3_half(b[sub]);
        lds16(b + 4 + 8 * sub, w[i]);            // 8 bytes of this sub-block (and 8 of the next)
      }
    } else if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
      const float d = half_at(p), dmin = half_at(p + 2);
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        int sc, m;
        k4_scale_min(4 * hb + j0 + i, p + 4, sc, m);
        scale[i] = d * float(sc);
        mn[i] = dmin * float(m);
      }
#pragma unroll
      for (int i = 0; i < NJ / 2; ++i) lds16(p + (QT == QTYPE_Q4_K ? 16 : 48) + 32 * (2 * hb + (j0 >> 1) + i) + 16 * u, w[i]);
      if constexpr (QT == QTYPE_Q5_K) lds16(p + 16 + 16 * u, h);
    } else if constexpr (QT == QTYPE_Q6_K) {
      const float d = half_at(p + 208);
#pragma unroll
      for (int i = 0; i < NJ; ++i) scale[i] = d * float(int(int8_t(p[192 + 8 * hb + 2 * (j0 + i) + u])));
      lds16(p + 64 * hb + 16 * u, w[0]);
      lds16(p + 64 * hb + 32 + 16 * u, w[1]);
      lds16(p + 128 + 32 * hb + 16 * u, h);
    } else if constexpr (QT == QTYPE_Q2_K) {
      const float d = half_at(p + 80), dmin = half_at(p + 82);
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const uint32_t s = p[8 * hb + 2 * (j0 + i) + u];
        scale[i] = d * float(s & 0x0fu);
        mn[i] = dmin * float(s >> 4);
      }
      lds16(p + 16 + 32 * hb + 16 * u, w[0]);
    } else {
      const float d = half_at(p + 108);
#pragma unroll
      for (int i = 0; i < NJ; ++i) scale[i] = d * float(q3k_scale(p + 96, 8 * hb + 2 * (j0 + i) + u) - 32);
      lds16(p + 32 + 32 * hb + 16 * u, w[0]);
      lds16(p + 16 * u, h);
    }
  }
  // Word k (weights 4k .. 4k+3) of group i as unsigned bytes.
  __device__ __forceinline__ uint32_t bytes(int i, int k) const {
    const int j = j0 + i;
    if constexpr (QT == QTYPE_Q8_0) return w[i][k] ^ 0x80808080u;
    else if constexpr (QT == QTYPE_Q4_0) return (w[i][k] >> (4 * u)) & 0x0f0f0f0fu;
    else if constexpr (QT == QTYPE_MXFP4) return fp4_bytes((w[i][k] >> (4 * u)) & 0x0f0f0f0fu);
    else if constexpr (QT == QTYPE_NVFP4) return fp4_bytes((w[i][k & 1] >> (k < 2 ? 0 : 4)) & 0x0f0f0f0fu);
    else if constexpr (QT == QTYPE_Q4_K) return (w[i >> 1][k] >> (4 * (i & 1))) & 0x0f0f0f0fu;
    else if constexpr (QT == QTYPE_Q5_K) return ((w[i >> 1][k] >> (4 * (i & 1))) & 0x0f0f0f0fu) | (((h[k] >> (4 * hb + j)) & 0x01010101u) << 4);
    else if constexpr (QT == QTYPE_Q6_K) return ((w[i & 1][k] >> (2 * (j & 2))) & 0x0f0f0f0fu) | (((h[k] >> (2 * j)) & 0x03030303u) << 4);
    else if constexpr (QT == QTYPE_Q2_K) return (w[0][k] >> (2 * j)) & 0x03030303u;
    else return ((w[0][k] >> (2 * j)) & 0x03030303u) | (((h[k] >> (4 * hb + j)) & 0x01010101u) << 2);
  }
};
// Four such bytes less the type's offset -> two operand pairs, exact.
template <int QT, typename O>
__device__ __forceinline__ void byte_pairs(uint32_t w, uint32_t& p01, uint32_t& p23) {
  if constexpr (QT == QTYPE_Q8_0 && !std::is_same<O, __half>::value) {     // bytes above 127 do not fit the bfloat16 pattern 0x43qq
    p01 = pack<O>(byte_to_float(w, 0) - 128.f, byte_to_float(w, 1) - 128.f);
    p23 = pack<O>(byte_to_float(w, 2) - 128.f, byte_to_float(w, 3) - 128.f);
  } else {
    bytes_minus<O>(w, byte_offset<QT>(), p01, p23);
  }
}

__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

template <int QT, typename T, int ROWS, int BT>
__global__ void __launch_bounds__(kThreads, 2)
gemm_exact_kernel(const T* __restrict__ x, const uint8_t* __restrict__ w, const T* __restrict__ bias, T* __restrict__ y, int m, int n, int k) {
  using O = Operand<T>;
  constexpr int PL = x_planes<T>(), MI = ROWS / 64, NI = BT / 16, kRawPitch = raw_pitch<QT>();
  constexpr bool kMins = has_mins<QT>();
  constexpr int kPer = (QT == QTYPE_Q6_K || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K || QT == QTYPE_NVFP4) ? 1 : 2;    // K steps that share a scale
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* raw = smem;                                            // [ROWS][kRawPitch]
  uint8_t* sA = raw + ROWS * kRawPitch;                           // [ROWS][kPitchB]
  uint8_t* sB = sA + ROWS * kPitchB;                              // [PL][BT][kPitchB]
  float* sS = reinterpret_cast<float*>(sB + PL * BT * kPitchB);   // [8 groups][ROWS] scales, then mins
  float* sM = sS + 8 * ROWS;
  float* sX = sM + 8 * ROWS;                                      // [8 groups][BT] activation sums (types with mins)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * ROWS, m0 = blockIdx.y * BT;
  const int64_t row_bytes = int64_t(k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes;
  // this CTA's super-blocks: one of gridDim.z (= cluster size) slices of K
  const int nsb = (k + 255) >> 8, per_slice = (nsb + int(gridDim.z) - 1) / int(gridDim.z);
  const int h_begin = 2 * int(blockIdx.z) * per_slice, halves = min((k + kHalfK - 1) / kHalfK, h_begin + 2 * per_slice);

  // packed bytes of super-block c: TPR threads per row, 16-byte chunks of the row's window in turn
  constexpr int TPR = kThreads / ROWS;
  const int crow = tid / TPR;
  const uint8_t* wrow = w + int64_t(min(n0 + crow, n - 1)) * row_bytes;
  auto issue_raw = [&](int c) {
    const uint8_t* src = wrow + int64_t(c) * sb_bytes<QT>();
    const int phase = int(reinterpret_cast<uintptr_t>(src) & 15);
    const int piece = int(min(int64_t(sb_bytes<QT>()), row_bytes - int64_t(c) * sb_bytes<QT>()));
    const int chunks = (phase + piece + 15) >> 4;
    const uint32_t dst = uint32_t(__cvta_generic_to_shared(raw + crow * kRawPitch));
    for (int i = tid % TPR; i < chunks; i += TPR) cp_async16(dst + 16 * i, src - phase + 16 * i);
  };
  // activations of half h: units of 8 values
  constexpr int kUnits = BT * (kHalfK / 8) / kThreads;
  float4 xf[PL == 3 ? kUnits : 1][2];
  auto fetch_x = [&](int h) {
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int unit = tid + i * kThreads, row = unit >> 4, k8 = unit & 15;
      const int kk = h * kHalfK + 8 * k8;
      const bool in = m0 + row < m && kk < k;
      if constexpr (PL == 3) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + int64_t(m0 + row) * k + kk);
        xf[i][0] = in ? __ldg(p) : z;
        xf[i][1] = in ? __ldg(p + 1) : z;
      } else {
        uint8_t* dst = sB + row * kPitchB + 16 * k8;
        if (in) cp_async16(uint32_t(__cvta_generic_to_shared(dst)), x + int64_t(m0 + row) * k + kk);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  auto store_x = [&]() {                       // float32: three bfloat16 numbers whose sum is the value
    if constexpr (PL == 3) {
#pragma unroll
      for (int i = 0; i < kUnits; ++i) {
        const int unit = tid + i * kThreads, row = unit >> 4, k8 = unit & 15;
        float v[8] = {xf[i][0].x, xf[i][0].y, xf[i][0].z, xf[i][0].w, xf[i][1].x, xf[i][1].y, xf[i][1].z, xf[i][1].w};
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) {
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            o[j] = pack<O>(v[2 * j], v[2 * j + 1]);
            v[2 * j] -= __uint_as_float(o[j] << 16);
            v[2 * j + 1] -= __uint_as_float(o[j] & 0xffff0000u);
          }
          *reinterpret_cast<uint4*>(sB + (pl * BT + row) * kPitchB + 16 * k8) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
  };

  float res[MI][NI][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) res[i][j][q] = 0.f;

  float zero4[4];
  opaque_zero4(zero4);
  const int wm = warp & 3, wn = warp >> 2, g = lane >> 2, t = lane & 3;
  const uint32_t a_addr = uint32_t(__cvta_generic_to_shared(sA + (wm * (ROWS / 4) + (lane & 15)) * kPitchB + (lane >> 4) * 16));
  const uint32_t b_addr = uint32_t(__cvta_generic_to_shared(sB + (wn * (BT / 2) + (lane & 7) + ((lane >> 4) << 3)) * kPitchB + ((lane >> 3) & 1) * 16));

  if (h_begin < halves) {
    issue_raw(h_begin >> 1);
    fetch_x(h_begin);
  }
  cp_async_commit();
  for (int h = h_begin; h < halves; ++h) {
    store_x();
    cp_async_wait<0>();
    __syncthreads();                             // bytes and activations of this half are here
    {
      // decode: ROWS * 8 groups of 16 weights
      const int c = h >> 1;
      constexpr int NJ = ROWS * 2 >= kThreads ? 4 : 2;            // ROWS * 8 / NJ units, one per thread
      static_assert(ROWS * 8 / NJ == kThreads, "one unit per thread");
      const int row = tid / (8 / NJ), part = tid % (8 / NJ), u = part & 1;
      const uint8_t* src = w + int64_t(min(n0 + row, n - 1)) * row_bytes + int64_t(c) * sb_bytes<QT>();
      Unit<QT, NJ> unit;
      unit.load(raw + row * kRawPitch + (reinterpret_cast<uintptr_t>(src) & 15), h & 1, NJ == 4 ? 0 : part & 2, u);
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const int grp = 2 * (unit.j0 + i) + u;
        uint32_t o[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) byte_pairs<QT, O>(unit.bytes(i, q), o[2 * q], o[2 * q + 1]);
        uint4* dst = reinterpret_cast<uint4*>(sA + row * kPitchB + 32 * grp);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        const bool in = h * kHalfK + 16 * grp < k;               // past the end of the row: whatever the buffer holds
        sS[grp * ROWS + row] = in ? unit.scale[i] : 0.f;
        if constexpr (kMins) sM[grp * ROWS + row] = in ? unit.mn[i] : 0.f;
      }
      if constexpr (kMins) {
        for (int u = tid; u < BT * 8; u += kThreads) {
          const int row = u >> 3, grp = u & 7;
          float sum = 0.f;
#pragma unroll
          for (int pl = PL - 1; pl >= 0; --pl) {
            const uint4* p = reinterpret_cast<const uint4*>(sB + (pl * BT + row) * kPitchB + 32 * grp);
            sum += MmaType<O>::sum8(p[0]) + MmaType<O>::sum8(p[1]);
          }
          sX[grp * BT + row] = sum;
        }
      }
    }
    __syncthreads();
    if ((h & 1) && h + 1 < halves) issue_raw((h + 1) >> 1);      // both halves of the super-block are decoded
    if (PL == 3 && h + 1 < halves) fetch_x(h + 1);
#pragma unroll 1
    for (int gg = 0; gg < 8; gg += kPer) {        // not unrolled: hoisted operand loads spill
      uint32_t a[kPer][MI][4];
#pragma unroll
      for (int s = 0; s < kPer; ++s)
#pragma unroll
        for (int i = 0; i < MI; ++i) ldmatrix4(a_addr + i * 16 * kPitchB + (gg + s) * 32, a[s][i]);
      float sc[MI][2];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int r = wm * (ROWS / 4) + i * 16 + g;
        sc[i][0] = sS[gg * ROWS + r];
        sc[i][1] = sS[gg * ROWS + r + 8];
      }
      // 16 activation rows at a time: few live accumulators, so that 64 of them per warp fit beside the results
#pragma unroll
      for (int jj = 0; jj < NI / 2; ++jj) {
        float acc[MI][2][4];
#pragma unroll
        for (int s = 0; s < kPer; ++s)
#pragma unroll
          for (int pl = PL - 1; pl >= 0; --pl) {                 // the small parts first
            uint32_t b[4];
            ldmatrix4(b_addr + (pl * BT + jj * 16) * kPitchB + (gg + s) * 32, b);
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                if (s == 0 && pl == PL - 1) MmaType<O>::mma_c(acc[i][j], a[s][i], b[2 * j], b[2 * j + 1], zero4);
                else MmaType<O>::mma(acc[i][j], a[s][i], b[2 * j], b[2 * j + 1]);
              }
          }
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float (&r)[4] = res[i][2 * jj + j];
            r[0] = fmaf(sc[i][0], acc[i][j][0], r[0]);
            r[1] = fmaf(sc[i][0], acc[i][j][1], r[1]);
            r[2] = fmaf(sc[i][1], acc[i][j][2], r[2]);
            r[3] = fmaf(sc[i][1], acc[i][j][3], r[3]);
          }
        if constexpr (kMins) {
#pragma unroll
          for (int s = 0; s < kPer; ++s)
#pragma unroll
            for (int i = 0; i < MI; ++i) {
              const int row = wm * (ROWS / 4) + i * 16 + g;
              const float m0v = sM[(gg + s) * ROWS + row], m1v = sM[(gg + s) * ROWS + row + 8];
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const float2 X = *reinterpret_cast<const float2*>(&sX[(gg + s) * BT + wn * (BT / 2) + (2 * jj + j) * 8 + 2 * t]);
                float (&r)[4] = res[i][2 * jj + j];
                r[0] = fmaf(-m0v, X.x, r[0]);
                r[1] = fmaf(-m0v, X.y, r[1]);
                r[2] = fmaf(-m1v, X.x, r[2]);
                r[3] = fmaf(-m1v, X.y, r[3]);
              }
            }
        }
      }
    }
    __syncthreads();                             // the operand tiles may be overwritten
    if (PL == 1 && h + 1 < halves) fetch_x(h + 1);
    cp_async_commit();
  }

  // The sums go through shared memory (row pitch ROWS + 4: the two token rows of a lane pair on distinct banks), where the CTAs of a
  // cluster add their slices, each a part of the tile in slice order, and rows of the output are stored whole.
  cp_async_wait<0>();
  __syncthreads();
  constexpr int kSumPitch = ROWS + 4;
  float* sums = reinterpret_cast<float*>(smem);                   // [BT][kSumPitch]
  static_assert(size_t(BT) * kSumPitch * sizeof(float) <= smem_bytes<QT, T, ROWS, BT>(), "sums");
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        sums[(wn * (BT / 2) + j * 8 + 2 * t + (q & 1)) * kSumPitch + wm * (ROWS / 4) + i * 16 + g + 8 * (q >> 1)] = res[i][j][q];
  const int slices = int(gridDim.z);
  if (slices > 1) cluster_barrier(); else __syncthreads();
  bool again = false;
  for (int idx = int(blockIdx.z) * kThreads + tid; idx < ROWS * BT; idx += slices * kThreads) {
    const int r = idx % ROWS, col = idx / ROWS;
    if (n0 + r >= n || m0 + col >= m) continue;
    float* at = &sums[col * kSumPitch + r];
    float v = 0.f;
    if (slices > 1)
      for (int z = 0; z < slices; ++z) v += ld_cluster_f32(at, uint32_t(z));
    else
      v = *at;
    if (bias != nullptr) v += MmaType<T>::to_float(bias[n0 + r]);
    y[int64_t(m0 + col) * n + n0 + r] = MmaType<T>::from_float(v);
    again = again || !(fabsf(v) < INFINITY) || (PL == 3 && v != 0.f && fabsf(v) < 0x1p-100f);
  }
  // float32 activations beyond what three bfloat16 numbers, or their sums with quants, hold: not results of the tiles
  static_assert(kThreads % ROWS == 0, "a thread's results are one weight row's");
  if (again) {
    const int idx = int(blockIdx.z) * kThreads + tid, r = idx % ROWS, col = idx / ROWS, step = slices * (kThreads / ROWS);
    const int cols = min(BT, m - m0);            // of this tile; this thread stored col, col + step, ..
    redo<QT, T, PL == 3>(y + int64_t(m0 + col) * n + n0 + r, int64_t(step) * n, x + int64_t(m0 + col) * k, int64_t(step) * k, w + int64_t(n0 + r) * row_bytes,
                         bias != nullptr ? MmaType<T>::to_float(bias[n0 + r]) : 0.f, (cols - col + step - 1) / step, k);
  }
  if (slices > 1) cluster_barrier();           // nobody leaves while its sums may still be read
}

template <int QT, typename T, int ROWS, int BT>
int launch_tile(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  constexpr size_t smem = smem_bytes<QT, T, ROWS, BT>();
  static_assert(smem <= 113 * 1024, "two CTAs per SM");
  auto kern = gemm_exact_kernel<QT, T, ROWS, BT>;
  static SmemOptIn granted;
  if (!smem_opt_in(kern, smem, granted)) return RC_LAUNCH;
  const int tiles = (n + ROWS - 1) / ROWS, m_tiles = (m + BT - 1) / BT, nsb = (k + 255) / 256;
  if (m_tiles > 65535) return RC_RANGE;
  // The number of K slices with the shortest walk: rounds of two CTAs per SM times super-blocks per slice (a slice costs about two
  // super-blocks more for its start and the exchange of sums).
  const int64_t slots = 2 * stream::sm_count();
  int slices = 1;
  int64_t best = INT64_MAX;
  for (int z = 1; z <= 8 && z <= nsb; ++z) {
    const int64_t walk = ((int64_t(tiles) * m_tiles * z + slots - 1) / slots) * ((nsb + z - 1) / z + 2);
    if (walk < best) { best = walk; slices = z; }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(tiles), unsigned(m_tiles), unsigned(slices));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = unsigned(slices);
  cfg.attrs = attr;
  cfg.numAttrs = slices > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<const T*>(a), static_cast<const uint8_t*>(b), static_cast<const T*>(bias), static_cast<T*>(c), m, n,
                            k) == cudaSuccess ? RC_OK : RC_LAUNCH;
}

// 128 x 128 tiles above 64 activation rows, 128 x 64 above 32 (float32: 128 x 32, for its three operand planes) where that gives a
// quarter of the SMs a tile, else 64 x 32.
template <int QT, typename T>
int launch(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  constexpr bool kPlanes = x_planes<T>() == 3;
  const int64_t row_tiles = (n + 127) / 128, quarter = stream::sm_count() / 4;
  if constexpr (!kPlanes) {
    if (m > 64 && row_tiles * ((m + 127) / 128) >= quarter) return launch_tile<QT, T, 128, 128>(a, b, bias, c, m, n, k, s);
    if (m > 32 && row_tiles * ((m + 63) / 64) >= quarter) return launch_tile<QT, T, 128, 64>(a, b, bias, c, m, n, k, s);
  } else {
    if (row_tiles * ((m + 31) / 32) >= quarter) return launch_tile<QT, T, 128, 32>(a, b, bias, c, m, n, k, s);
  }
  return launch_tile<QT, T, 64, 32>(a, b, bias, c, m, n, k, s);
}

}  // namespace exact
}  // namespace b200gguf
