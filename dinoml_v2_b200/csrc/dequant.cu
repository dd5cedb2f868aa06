// Standalone GGUF dequantize kernel: packed blocks -> dense f32 / f16 / bf16, bit-exact.
//
// Replaces the un-vendored libgguf device entry the reference's generated module declares at
// src/dinoml/templates/gpu_module.cu.j2:35-42 and calls from src/dinoml/lowering/ops/gemm.py:745,
// keeping its name and argument list so the generated launch text links unchanged.
//
// HBM-bound and write-dominated (Q4_K -> f32 writes 7.1 bytes per byte read).  One kernel for the nine types and three outputs: an item
// is R consecutive packed bytes and every run of R weights that they hold, so each packed byte is loaded once and each run is one
// streaming store of whole 32-byte sectors.  What was measured, [11008 x 4096] in a graph, buffers of more than the L2 in turn, before
// (one 8-weight unit per thread, or items with 8-weight runs, two per thread) -> now, us:
//                f16                          f32
//   Q4_K    20.5 -> 18.6  (6.2 TB/s)    42.7 -> 33.8  (6.1 TB/s)
//   Q5_K    28.9 -> 19.9                52.1 -> 34.7
//   Q6_K    25.0 -> 22.0                50.4 -> 35.9
//   Q8_0    28.7 -> 23.0                45.2 -> 36.8
//   Q4_0    21.3 -> 19.3                46.9 -> 33.2
//   Q2_K    18.9 -> 17.6                38.5 -> 32.2
//   Q3_K    23.5 -> 19.3                48.9 -> 33.3
//   MXFP4   24.7 -> 19.2                46.2 -> 32.9
//   NVFP4   24.8 -> 20.5                47.0 -> 32.9
// and [512 x 2048], where the launch counts: 2.1 - 2.9 -> 1.5 - 1.9 (f16), 2.8 - 4.7 -> 2.0 - 2.5 (f32).  Where it came from:
//   * a 256-bit store per run: as two 128-bit stores, each half fills its sectors (f32: 43 -> 34);
//   * four quants decoded at a time: masks and shifts for four bytes at once, then one byte permute (0x4B0000qq is 2^23 + q) and one exact
//     subtraction per weight instead of shift, mask and conversion (Q5_K 28.9 -> 20.7);
//   * words for blocks that start at any address, shifted into place, instead of bytes or halves (MXFP4 24.7 -> 19.9);
//   * programmatic dependent launch, 0.3 - 0.4 us per call: the next kernel's CTAs are let in once a CTA holds its packed bytes.  From the first
//     instruction on they would fill the SMs that happen to be free, and a small grid ends up uneven (Q2_K [2048 x 4096] 4.7 -> 5.2).
// Decoding uses explicitly rounded fp32 operations, those of decode8<QT> in its order (bit-exact).
#include "gguf_common.cuh"

#include <type_traits>

namespace b200gguf {

constexpr int kDequantThreads = 256;

// 32 bytes of output of one thread, streaming: one 256-bit store where the output starts at a 32-byte boundary (every run then
// does), else two of 128 bits.
__device__ __forceinline__ void store32(void* p, const uint32_t (&v)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.cs.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
  } else {
    __stcs(static_cast<uint4*>(p), make_uint4(v[0], v[1], v[2], v[3]));
    __stcs(static_cast<uint4*>(p) + 1, make_uint4(v[4], v[5], v[6], v[7]));
  }
}

// N words of packed bytes from p.  A: alignment of p.  1: any address; the aligned words around p are shifted into place, except where
// `edge` says that such a word holds bytes outside the buffer.  0: any address in shared memory (with four bytes after the last).
template <int N, int A>
__device__ __forceinline__ void load_words(const uint8_t* __restrict__ p, bool edge, uint32_t (&v)[N]) {
  if constexpr (A == 16 && N == 4) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else if constexpr (A == 16 && N == 2) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
    v[0] = q.x; v[1] = q.y;
  } else if constexpr (A == 0) {
    const int off = int(__cvta_generic_to_shared(p)) & 3;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p - off);
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) r[i] = w[i];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __funnelshift_r(r[i], r[i + 1], 8 * off);
  } else if constexpr (A >= 4) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
  } else {
    if (edge) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        v[i] = uint32_t(p[4 * i]) | uint32_t(p[4 * i + 1]) << 8 | uint32_t(p[4 * i + 2]) << 16 | uint32_t(p[4 * i + 3]) << 24;
      return;
    }
    const int off = int(reinterpret_cast<uintptr_t>(p) & 3);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p - off);
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = __ldg(w + i);
    r[N] = off ? __ldg(w + N) : 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __funnelshift_r(r[i], r[i + 1], 8 * off);
  }
}
__device__ __forceinline__ float half_of(uint32_t word, int hi) { return half_bits_to_float(uint16_t(hi ? word >> 16 : word & 0xffffu)); }
// Four FP4 codes (high nibbles of the bytes zero) -> bytes 12 + twice the value: look-ups of the eight magnitudes, both signs.
__device__ __forceinline__ uint32_t fp4_biased(uint32_t w) {
  const uint32_t mag = w & 0x07070707u;
  const uint32_t sel = __byte_perm(mag | (mag >> 4), 0u, 0x4420);
  const uint32_t pos = __byte_perm(0x0F0E0D0Cu, 0x18141210u, sel), neg = __byte_perm(0x090A0B0Cu, 0x00040608u, sel);
  const uint32_t sign = ((w >> 3) & 0x01010101u) * 0xffu;
  return (pos & ~sign) | (neg & sign);
}

// Geometry of a type's items (R: weights per run).
//   Q4_0 / MXFP4: R of a block's 16 bytes: low nibbles = weights 0 .. 15, high nibbles = weights 16 .. 31
//   Q8_0:         R weights
//   NVFP4:        one sub-block: low nibbles = its first 8 weights, high nibbles = the other 8
//   Q4_K / Q5_K:  R of the 32 bytes of a 64-weight group: low nibbles its first half, high nibbles the other; Q5_K: and R bytes of qh
//   Q6_K:         R of the 32 ql bytes that hold 32-weight quarters `half` and `half` + 2 of a 128-weight half, and R bytes of qh
//   Q2_K / Q3_K:  R of the 32 bytes of a 128-weight half: bit pairs j = 0..3 are runs 32 apart; Q3_K: and R mask bytes
template <int QT, int R> struct ItemGeom {
  static constexpr bool k16 = QT == QTYPE_NVFP4 && R == 16;         // a sub-block's 8 bytes are its 16 weights
  static constexpr int kRuns = QT == QTYPE_Q8_0 ? 1 : QT == QTYPE_Q6_K ? 2 : (QT == QTYPE_Q2_K || QT == QTYPE_Q3_K) ? 4
                             : QT == QTYPE_NVFP4 ? 16 / R : 2;
  static constexpr int kItems = QTraits<QT>::kBlock / (kRuns * R);  // per block
  // alignment that every block has in a buffer that has it
  static constexpr int kAlign = (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) ? 16 : (QT == QTYPE_Q2_K || QT == QTYPE_NVFP4) ? 4 : 1;
  static constexpr int kBias = QT == QTYPE_Q8_0 ? 128 : QT == QTYPE_Q6_K ? 32 : QT == QTYPE_Q4_0 ? 8 : QT == QTYPE_Q3_K ? 4
                             : (QT == QTYPE_MXFP4 || QT == QTYPE_NVFP4) ? 12 : 0;
  static constexpr bool kMin = QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q2_K;
};

// Weights per run: 32 bytes of output.  16-bit Q2_K and Q3_K, whose items hold four runs, take 8 (16-byte stores): with 16 a matrix has too
// few threads (Q2_K [2048 x 4096] 5.4 -> 4.7 us, Q3_K 5.1 -> 4.7; [11008 x 4096] equal).
template <int QT, typename T> constexpr int run_of() { return sizeof(T) == 4 || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K ? 8 : 16; }

template <int QT, typename T, int A> struct Item {
  static constexpr int R = run_of<QT, T>(), N = R / 4;
  using G = ItemGeom<QT, R>;
  static constexpr int kQ = QT == QTYPE_NVFP4 ? 2 : N;              // words of quants
  static constexpr bool kHigh = QT == QTYPE_Q5_K || QT == QTYPE_Q6_K || QT == QTYPE_Q3_K;
  uint32_t q[kQ], h[kHigh ? N : 1], s[4];

  __device__ __forceinline__ void load(const uint8_t* __restrict__ b, int item, bool edge) {
    if constexpr (QT == QTYPE_Q4_0) {
      s[0] = uint32_t(b[0]) | uint32_t(b[1]) << 8;
      load_words<N, A>(b + 2 + R * item, edge, q);
    } else if constexpr (QT == QTYPE_Q8_0) {
      s[0] = ld_u16(b);
      load_words<N, A>(b + 2 + R * item, edge, q);
    } else if constexpr (QT == QTYPE_MXFP4) {
      s[0] = b[0];
      load_words<N, A>(b + 1 + R * item, edge, q);
    } else if constexpr (QT == QTYPE_NVFP4) {
      const int sub = G::k16 ? item : item >> (G::kRuns == 2 ? 0 : 1);
      s[0] = b[sub];
      load_words<2, A>(b + 4 + 8 * sub, edge, q);
    } else if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
      constexpr int kQs = QT == QTYPE_Q4_K ? 16 : 48, P = 32 / R;
      load_words<4, A>(b, edge, s);
      load_words<N, A>(b + kQs + 32 * (item / P) + R * (item % P), edge, q);
      if constexpr (QT == QTYPE_Q5_K) load_words<N, A>(b + 16 + R * (item % P), edge, h);
    } else {
      constexpr int P = 32 / R;
      if constexpr (QT == QTYPE_Q6_K) {
        const int hb = item / (2 * P), half = item / P & 1, l0 = R * (item % P);
        uint32_t sc[2];
        load_words<2, A>(b + 192 + 8 * hb, edge, sc);
        s[0] = sc[0]; s[1] = sc[1];
        s[3] = ld_u16(b + 208);
        load_words<N, A>(b + 64 * hb + 32 * half + l0, edge, q);
        load_words<N, A>(b + 128 + 32 * hb + l0, edge, h);
      } else if constexpr (QT == QTYPE_Q2_K) {
        const int hb = item / P, l0 = R * (item % P);
        uint32_t sc[2];
        load_words<2, A>(b + 8 * hb, edge, sc);
        s[0] = sc[0]; s[1] = sc[1];
        uint32_t d[1];
        load_words<1, A>(b + 80, edge, d);
        s[3] = d[0];
        load_words<N, A>(b + 16 + 32 * hb + l0, edge, q);
      } else {
        const int hb = item / P, l0 = R * (item % P);
        uint32_t sc[3];
        load_words<3, A>(b + 96, edge, sc);
        s[0] = sc[0]; s[1] = sc[1]; s[2] = sc[2];
        s[3] = uint32_t(b[108]) | uint32_t(b[109]) << 8;
        load_words<N, A>(b + 32 + 32 * hb + l0, edge, q);
        load_words<N, A>(b + l0, edge, h);
      }
    }
  }

  // Run j: its first output in the block, its scale and min (products rounded as decode8<QT>'s) and its weights as biased bytes.
  __device__ __forceinline__ int first(int item, int j) const {
    constexpr int P = 32 / R;
    if constexpr (QT == QTYPE_Q8_0) return R * item;
    else if constexpr (QT == QTYPE_Q4_0 || QT == QTYPE_MXFP4) return R * item + 16 * j;
    else if constexpr (QT == QTYPE_NVFP4) return 16 * item + 8 * j;
    else if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) return 64 * (item / P) + R * (item % P) + 32 * j;
    else if constexpr (QT == QTYPE_Q6_K) return 128 * (item / (2 * P)) + 32 * (item / P & 1) + R * (item % P) + 64 * j;
    else return 128 * (item / P) + R * (item % P) + 32 * j;
  }
  __device__ __forceinline__ void scale(int item, int j, float& ds, float& dm) const {
    dm = 0.f;
    if constexpr (QT == QTYPE_Q4_0 || QT == QTYPE_Q8_0) ds = half_of(s[0], 0);
    else if constexpr (QT == QTYPE_MXFP4) ds = e8m0_half(s[0]);
    else if constexpr (QT == QTYPE_NVFP4) ds = ue4m3_half(s[0]);
    else if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) {
      // 6-bit (scale, min) of sub-block 2g + j: in place for the first four, split across two bytes after
      const int g = item / (32 / R), sh = 16 * (g & 1) + 8 * j;
      const uint32_t sc = g < 2 ? s[1] >> sh & 0x3fu : (s[3] >> sh & 0x0fu) | (s[1] >> sh >> 2 & 0x30u);
      const uint32_t mn = g < 2 ? s[2] >> sh & 0x3fu : (s[3] >> sh >> 4 & 0x0fu) | (s[2] >> sh >> 2 & 0x30u);
      ds = __fmul_rn(half_of(s[0], 0), float(sc));
      dm = __fmul_rn(half_of(s[0], 1), float(mn));
    } else {
      const int hb = item / (32 / R), u = (R * (item % (32 / R))) >> 4, i4 = 2 * (j & 1) + u;     // sub-block 8 hb + 2 j + u
      if constexpr (QT == QTYPE_Q6_K) {
        ds = __fmul_rn(half_of(s[3], 0), float(int(int8_t(s[j] >> (8 * (2 * (item / (32 / R) & 1) + u))))));
      } else if constexpr (QT == QTYPE_Q2_K) {
        const uint32_t b = s[j >> 1] >> (8 * i4);
        ds = __fmul_rn(half_of(s[3], 0), float(b & 0x0fu));
        dm = __fmul_rn(half_of(s[3], 1), float(b >> 4 & 0x0fu));
      } else {
        // sub-block 4 qd + i4: low nibble in byte (4 qd + i4) % 8 (its high half from sub-block 8 on), two high bits in byte 8 + i4 at 2 qd
        const uint32_t low = s[j >> 1] >> (8 * i4 + 4 * hb) & 0x0fu, high = s[2] >> (8 * i4 + 2 * (2 * hb + (j >> 1))) & 0x03u;
        ds = __fmul_rn(half_of(s[3], 0), float(int(low | high << 4) - 32));
      }
    }
  }
  __device__ __forceinline__ uint32_t bytes(int item, int j, int k) const {
    if constexpr (QT == QTYPE_Q8_0) return q[k] ^ 0x80808080u;
    else if constexpr (QT == QTYPE_Q4_0) return q[k] >> (4 * j) & 0x0f0f0f0fu;
    else if constexpr (QT == QTYPE_MXFP4) return fp4_biased(q[k] >> (4 * j) & 0x0f0f0f0fu);
    else if constexpr (QT == QTYPE_NVFP4) return fp4_biased((G::k16 ? q[k & 1] >> (2 * (k & 2)) : q[k & 1] >> (4 * j)) & 0x0f0f0f0fu);
    else if constexpr (QT == QTYPE_Q4_K) return q[k] >> (4 * j) & 0x0f0f0f0fu;
    else if constexpr (QT == QTYPE_Q5_K) return (q[k] >> (4 * j) & 0x0f0f0f0fu) | (h[k] >> (2 * (item / (32 / R)) + j) & 0x01010101u) << 4;
    else if constexpr (QT == QTYPE_Q6_K) return (q[k] >> (4 * j) & 0x0f0f0f0fu) | (h[k] >> (4 * j + 2 * (item / (32 / R) & 1)) & 0x03030303u) << 4;
    else if constexpr (QT == QTYPE_Q2_K) return q[k] >> (2 * j) & 0x03030303u;
    else return (q[k] >> (2 * j) & 0x03030303u) | (h[k] >> (4 * (item / (32 / R)) + j) & 0x01010101u) << 2;
  }
  __device__ __forceinline__ void emit(T* dst, int item, bool wide) const {
#pragma unroll
    for (int j = 0; j < G::kRuns; ++j) {
      float ds, dm;
      scale(item, j, ds, dm);
      uint32_t v[R * int(sizeof(T)) / 4];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const uint32_t by = bytes(item, j, k);
        float w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // byte q as a float: 0x4B0000qq is 2^23 + q, and the difference is exact
          const float x = __fsub_rn(__uint_as_float(__byte_perm(by, 0x4B000000u, 0x7440u + e)), float(8388608 + G::kBias));
          w[e] = G::kMin ? __fsub_rn(__fmul_rn(ds, x), dm) : __fmul_rn(ds, x);
        }
        if constexpr (sizeof(T) == 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) v[4 * k + e] = __float_as_uint(w[e]);
        } else if constexpr (std::is_same<T, __half>::value) {
          const __half2 a = __floats2half2_rn(w[0], w[1]), c = __floats2half2_rn(w[2], w[3]);
          v[2 * k] = *reinterpret_cast<const uint32_t*>(&a); v[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&c);
        } else {
          const __nv_bfloat162 a = __floats2bfloat162_rn(w[0], w[1]), c = __floats2bfloat162_rn(w[2], w[3]);
          v[2 * k] = *reinterpret_cast<const uint32_t*>(&a); v[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&c);
        }
      }
      if constexpr (R * sizeof(T) == 32) store32(dst + first(item, j), v, wide);
      else __stcs(reinterpret_cast<uint4*>(dst + first(item, j)), make_uint4(v[0], v[1], v[2], v[3]));
    }
  }
};

// Items per thread.  Two for 16-bit NVFP4, whose item is a single store of few instructions: [28672 x 8192] 96 us, 105 with one ([2048 x 4096]
// 5.1 / 5.0).  One elsewhere: Q8_0 [2048 x 4096] 5.8 -> 5.7 (f16), 8.8 -> 8.2 (f32), Q4_K 4.6 -> 5.2 with two.
template <int QT, typename T> constexpr int items_per_thread() { return QT == QTYPE_NVFP4 && sizeof(T) == 2 ? 2 : 1; }

// A: alignment of the packed buffer where all its blocks keep it (16: Q4_K and Q5_K; 4: also Q2_K and NVFP4), 1: any start and block size,
// 0: Q6_K from a 16-byte boundary, through shared memory.  An item of Q6_K is 3 misaligned pieces of its block; a CTA's 32 or 16 blocks
// in 16-byte loads first cost a barrier and save the rest: [11008 x 4096] f16 25.0 -> 22.0 us, f32 37.0 -> 35.9, [512 x 2048] f32 3.1 -> 2.4.
// The other types with odd blocks have shorter pieces and lose by it: Q8_0 f16 23.4 -> 24.5, Q3_K 19.3 -> 20.7, MXFP4 19.2 -> 20.9, Q4_0 equal.
template <int QT, typename T, int A>
__global__ void __launch_bounds__(kDequantThreads)
dequant_kernel(const uint8_t* __restrict__ in, T* __restrict__ out, int64_t total_items, int64_t first_edge, int64_t last_edge, bool wide) {
  using G = ItemGeom<QT, run_of<QT, T>()>;
  constexpr int kPer = items_per_thread<QT, T>();
  asm volatile("griddepcontrol.wait;\n" ::: "memory");          // the packed bytes may be the preceding kernel's output
  if constexpr (A == 0) {
    constexpr int kBlocks = kDequantThreads / G::kItems, kBytes = kBlocks * QTraits<QT>::kBytes, kVec = kBytes / 16;
    static_assert(kPer == 1 && kBytes % 16 == 0, "");
    __shared__ __align__(16) uint8_t stage[kBytes + 16];
    const int64_t blk0 = int64_t(blockIdx.x) * kBlocks, blocks = total_items / G::kItems;
    const uint8_t* src = in + blk0 * QTraits<QT>::kBytes;
    const int bytes = blocks - blk0 >= kBlocks ? kBytes : int(blocks - blk0) * QTraits<QT>::kBytes, vecs = bytes / 16;
#pragma unroll
    for (int i = 0; i < (kVec + kDequantThreads - 1) / kDequantThreads; ++i) {
      const int at = i * kDequantThreads + threadIdx.x;
      if (at < vecs) *reinterpret_cast<uint4*>(stage + 16 * at) = __ldg(reinterpret_cast<const uint4*>(src) + at);
    }
    for (int at = 16 * vecs + threadIdx.x; at < bytes; at += kDequantThreads) stage[at] = src[at];
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int blk = threadIdx.x / G::kItems, item = threadIdx.x % G::kItems;
    if (blk0 + blk < blocks) {
      Item<QT, T, A> one;
      one.load(stage + blk * QTraits<QT>::kBytes, item, false);
      one.emit(out + (blk0 + blk) * QTraits<QT>::kBlock, item, wide);
    }
  } else {
    const int64_t base = int64_t(blockIdx.x) * (kPer * kDequantThreads) + threadIdx.x;
    Item<QT, T, A> it[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int64_t at = base + i * kDequantThreads, blk = at / G::kItems;
      if (at < total_items) it[i].load(in + blk * QTraits<QT>::kBytes, int(at % G::kItems), blk == first_edge || blk == last_edge);
    }
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int64_t at = base + i * kDequantThreads, blk = at / G::kItems;
      if (at < total_items) it[i].emit(out + blk * QTraits<QT>::kBlock, int(at % G::kItems), wide);
    }
  }
}

template <int QT, typename T, int A>
static int launch_items(const void* in, void* out, int64_t weights, cudaStream_t stream) {
  using G = ItemGeom<QT, run_of<QT, T>()>;
  constexpr int kPer = items_per_thread<QT, T>();
  const int64_t items = weights / QTraits<QT>::kBlock * G::kItems, per_cta = int64_t(kDequantThreads) * kPer;
  const int64_t grid = (items + per_cta - 1) / per_cta;
  if (grid > 0x7fffffffLL) return RC_RANGE;
  // blocks whose first or last aligned word holds bytes outside the buffer (only A == 1 looks)
  const uintptr_t begin = reinterpret_cast<uintptr_t>(in);
  const int64_t blocks = weights / QTraits<QT>::kBlock, first_edge = begin & 3 ? 0 : -1;
  const int64_t last_edge = (begin + uintptr_t(blocks) * QTraits<QT>::kBytes) & 3 ? blocks - 1 : -1;
  const bool wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(kDequantThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, dequant_kernel<QT, T, A>, static_cast<const uint8_t*>(in), static_cast<T*>(out), items, first_edge,
                                           last_edge, wide);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? RC_OK : RC_LAUNCH;
}

template <int QT, typename T>
static int launch_dequant(const void* in, void* out, int64_t rows, int64_t n_per_row, cudaStream_t stream) {
  using G = ItemGeom<QT, run_of<QT, T>()>;
  const uintptr_t at = reinterpret_cast<uintptr_t>(in);
  if constexpr (G::kAlign == 16)
    if ((at & 15) == 0) return launch_items<QT, T, 16>(in, out, rows * n_per_row, stream);
  if constexpr (G::kAlign >= 4)
    if ((at & 3) == 0) return launch_items<QT, T, 4>(in, out, rows * n_per_row, stream);
  if constexpr (QT == QTYPE_Q6_K)
    if ((at & 15) == 0) return launch_items<QT, T, 0>(in, out, rows * n_per_row, stream);
  if constexpr (QT == QTYPE_Q4_K) return RC_ALIGN;                  // the entry has refused these
  else return launch_items<QT, T, 1>(in, out, rows * n_per_row, stream);
}

template <int QT>
static int launch_dequant_dtype(const void* in, void* out, int64_t rows, int64_t n_per_row, int out_dtype,
                                cudaStream_t stream) {
  switch (out_dtype) {
    case OUT_F32: return launch_dequant<QT, float>(in, out, rows, n_per_row, stream);
    case OUT_F16: return launch_dequant<QT, __half>(in, out, rows, n_per_row, stream);
    case OUT_BF16: return launch_dequant<QT, __nv_bfloat16>(in, out, rows, n_per_row, stream);
    default: return RC_DTYPE;
  }
}

int dequantize_rows(const void* dev_in, int64_t qtype, int64_t rows, int64_t n_per_row, int output_dtype,
                    void* dev_out, cudaStream_t stream) {
  if (dev_in == nullptr || dev_out == nullptr) return RC_NULL;
  if (rows <= 0 || n_per_row <= 0) return RC_DIMS;
  const int bs = qtype_block_size(qtype);
  if (bs == 0) return RC_QTYPE;
  if (n_per_row % bs) return RC_KBLOCK;
  const uintptr_t in_a = reinterpret_cast<uintptr_t>(dev_in), out_a = reinterpret_cast<uintptr_t>(dev_out);
  if ((in_a & uintptr_t(qtype_alignment(qtype) - 1)) || (out_a & 15)) return RC_ALIGN;
  switch (qtype) {
    case QTYPE_Q8_0: return launch_dequant_dtype<QTYPE_Q8_0>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q4_K: return launch_dequant_dtype<QTYPE_Q4_K>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q6_K: return launch_dequant_dtype<QTYPE_Q6_K>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q4_0: return launch_dequant_dtype<QTYPE_Q4_0>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q5_K: return launch_dequant_dtype<QTYPE_Q5_K>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q2_K: return launch_dequant_dtype<QTYPE_Q2_K>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_Q3_K: return launch_dequant_dtype<QTYPE_Q3_K>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_MXFP4: return launch_dequant_dtype<QTYPE_MXFP4>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    case QTYPE_NVFP4: return launch_dequant_dtype<QTYPE_NVFP4>(dev_in, dev_out, rows, n_per_row, output_dtype, stream);
    default: return RC_QTYPE;
  }
}

}  // namespace b200gguf
