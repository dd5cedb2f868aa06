// Persistent decode GEMV ("stream" variant), M = 1..8, float16 / bfloat16 activations, tensor cores: Q4_K, Q5_K, Q6_K, Q4_0, Q2_K,
// Q3_K, MXFP4 and NVFP4 weights.
//
// C[M,N] = A[M,K] * dequant(W[N,K])^T (+ bias), W streamed once from HBM as packed GGUF blocks (Q4_K 144 B, Q6_K 210 B per
// 256 weights).  Two arithmetics on one data path:
//   * M <= 2 (every type but the FP4 ones): byte operands against digit planes of the activations, gemv_int_planes.cuh.  Bound by
//     HBM and the latencies around a launch: [28672 x 4096] Q4_K, M = 1, 66 MB: 16.0 us = 4.1 TB/s (21.2 with 16-bit operands); the same
//     copies without arithmetic take 12.6 us;
//   * M = 3 .. 8, and the FP4 types at every M: quants become 16-bit floats 128+q / 1024+q, mma.sync.m16n8k16 with fp32 accumulation,
//     per-sub-block scales applied in fp32, the offsets folded against activation sums.  Bound by the half-rate integer pipe.
// How the bytes move and how the work is cut:
//   * grid = one CTA per SM (or two).  The work of a launch is a line of units (16-row tile t, K chunk of 8 super-blocks),
//     tile-major; CTA c owns the contiguous range [c * U / G, (c + 1) * U / G), so every CTA moves the same number of bytes
//     whatever the tile count (688 tiles on 296 CTAs would otherwise be 2 or 3 tiles each).  A CTA walks its range from
//     the highest unit down: a tile cut between two CTAs is the FIRST thing the lower-numbered CTA computes (it leaves
//     its partial sums, 16 x M words that carry their own flag, in a small global workspace) and the LAST thing the
//     higher-numbered one computes (it adds the partial, empties the words and stores) - no waiting in practice, the
//     dependency points to a lower-numbered CTA, which is dispatched first, and the summation order is fixed.  One
//     prologue (activation sums) per CTA instead of one per tile;
//   * one producer warp issues, per (tile, K chunk of 8 super-blocks), one 2-D box of 16 weight rows (cp.async.bulk.tensor; ragged
//     rows, Q8_0 and the first lap of the ring: a 1-D bulk copy per row) into a ring of D shared-memory stages; a stage is "full" when its bytes have landed
//     (mbarrier transaction count) and "empty" when its 8 consumer warps have arrived.  The ring runs across tile
//     boundaries.  No thread spends issue slots on per-16-byte copies and no CTA barrier sits in the loop;
//   * NG groups of 8 consumer warps take the stages round-robin (warp w of a group unpacks super-block w of the chunk
//     for all 16 rows), accumulate over the chunks of a tile and hand their partial rows to the epilogue warp through
//     a double-buffered shared-memory area guarded by mbarriers; the epilogue warp adds the partials in a fixed order,
//     applies bias / the gated activation and stores (also to peer buffers for the sharded path);
//   * programmatic dependent launch: the producer starts streaming the (constant) weights at once, everything that
//     reads activations or writes outputs first waits for the preceding kernel (griddepcontrol.wait).  With the
//     one-CTA-per-SM grid and at most half of an SM's shared memory and registers per CTA, the next launch's CTAs sit
//     beside this launch's and fill their rings while this one finishes.
// Every wait (mbarriers, partial sums) is bounded; one that gives up records a code (11..15) in the library's
// status word, raises the CTA's abort flag, the producer waits for the copies it has in flight, and every role returns.
//
// Behavioural ancestor in the reference: the small-M kernels of the fused prototype
// (kernels/rocm/src/ck_gguf_q8_gemm.hip:1009-1166); the reference's CUDA path dequantizes the whole weight and runs a
// dense Sm80 GEMM instead (src/dinoml/lowering/ops/gemm.py:729-749).
#pragma once
#include <type_traits>

#include "gemv_int_planes.cuh"
#include "gemv_q6k_common.cuh"
#include "gemv_stream_common.cuh"
#include "scratch_sets.h"
#include "tensor_map.cuh"

namespace b200gguf {

int check_gemm_args(const void* a, const void* b, const void* c, int qtype, int dtype, int m, int n, int k);

namespace stream {

constexpr int kRows = 16;                       // weight rows per tile (one MMA M-tile)
constexpr int kKC = 8;                          // super-blocks per row per stage: one per consumer warp of a group
// Bytes per super-block and shared-memory row pitch of a stage.  Q4_K: 8 x 144 + 32 = 1184 B, so that the 8-byte reads of 4
// rows x 4 lanes (a half-warp) hit 32 distinct banks.  Q6_K: 8 x 210 = 1680 B is 16 (mod 128) by itself, which spreads the
// 4-byte reads of 8 rows x 4 lanes over all banks; a block starts 2 bytes off a word boundary in every odd super-block.
template <int QT> struct Geom;
template <> struct Geom<QTYPE_Q4_K> { static constexpr int kSbBytes = 144, kPitch = kKC * 144 + 32; };
template <> struct Geom<QTYPE_Q6_K> { static constexpr int kSbBytes = 210, kPitch = kKC * 210; };
// Q5_K = the Q4_K block with 32 more bytes (one high bit per weight) between the scales and the nibbles: same 8-byte reads,
// 8 x 176 + 32 = 1440 B is 32 (mod 128) like the Q4_K pitch.
template <> struct Geom<QTYPE_Q5_K> { static constexpr int kSbBytes = 176, kPitch = kKC * 176 + 32; };
// The further types: packed bytes per 256 weights of a row; the pitch is the stage piece made an odd multiple of 16 B (the
// 4-byte reads of 8 rows x 4 lanes then hit 32 distinct banks).
template <int BYTES> struct PaddedGeom { static constexpr int kSbBytes = BYTES, kPitch = kKC * BYTES + ((kKC * BYTES) % 32 == 16 ? 0 : 16); };
template <> struct Geom<QTYPE_Q4_0> : PaddedGeom<8 * 18> {};
template <> struct Geom<QTYPE_Q2_K> : PaddedGeom<84> {};
template <> struct Geom<QTYPE_Q3_K> : PaddedGeom<110> {};
template <> struct Geom<QTYPE_MXFP4> : PaddedGeom<8 * 17> {};
template <> struct Geom<QTYPE_NVFP4> : PaddedGeom<4 * 36> {};
template <> struct Geom<QTYPE_Q8_0> : PaddedGeom<8 * 34> {};
// RAG: weight rows that are not multiples of 16 bytes.  A row's piece then starts up to 15 bytes into the 16-byte aligned window
// that is copied, at a phase of its own.
template <int QT, bool RAG> constexpr int stage_pitch() { return RAG ? (kKC * Geom<QT>::kSbBytes + 30 + 15) / 16 * 16 : Geom<QT>::kPitch; }
// Whether a stage is fetched as one 2-D box over the weight (8-byte elements, at most 256 of them per row): a bulk copy per row takes 30 ns
// on an SM's copy unit whatever its length, which capped the stream at 5.7 TB/s.  The first lap of the ring still goes row by row: the
// rows land sooner and the map's own fetch is hidden (Q4_K, M = 1: [11008 x 4096] 8.7 us with boxes alone, 7.9 row by row; 2 x
// [28672 x 8192] 47.2 against 55.1).
template <int QT, bool RAG> constexpr bool tiled_copy() { return !RAG && stage_pitch<QT, RAG>() <= 256 * 8; }
// The integer arithmetic of gemv_int_planes.cuh serves the types that have it for one and two activation rows.
template <int QT, int MXC> constexpr bool int_path() { return MXC <= 2 && planes::has<QT>(); }
// Q4_0 and MXFP4 (32-weight blocks: a scale and 16 bytes of nibbles), NVFP4, Q2_K and Q3_K run on tensor cores like Q4_K.
template <int QT> constexpr bool is_blk32() { return QT == QTYPE_Q4_0 || QT == QTYPE_MXFP4; }
template <int QT> constexpr bool is_q23() { return QT == QTYPE_Q2_K || QT == QTYPE_Q3_K; }     // 2- / 3-bit quants, a scale per 16 weights

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {     // selector bit 3 of a nibble: replicate the byte's sign bit
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// 16-bit pair times 16-bit pair (one rounding per element; exact for the FP4 value x block scale products it is used for).
template <typename T> __device__ __forceinline__ uint32_t mul_pair(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t mul_pair<__half>(uint32_t a, uint32_t b) {
  const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t mul_pair<__nv_bfloat16>(uint32_t a, uint32_t b) {
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <typename T> __device__ __forceinline__ uint32_t splat_pair(float f);
template <> __device__ __forceinline__ uint32_t splat_pair<__half>(float f) {
  const __half2 v = __float2half2_rn(f);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t splat_pair<__nv_bfloat16>(float f) {
  const __nv_bfloat162 v = __float2bfloat162_rn(f);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Eight FP4 (e2m1) codes of one 32-bit word -> their exact values as 16-bit MMA operand pairs: lo01 / lo23 = the low nibbles of
// bytes (0, 1) / (2, 3), hi01 / hi23 = the high nibbles.  Magnitudes come from byte look-up tables held in two registers
// (prmt with the codes as selector), the sign bit is OR-ed in.  No offset, no rounding: every e2m1 value is a 16-bit float.
template <typename T>
__device__ __forceinline__ void fp4x8_operands(uint32_t w, uint32_t& lo01, uint32_t& lo23, uint32_t& hi01, uint32_t& hi23) {
  const uint32_t m = w & 0x77777777u, w4 = w << 4;
  // sign of [b0.lo, b0.hi, b1.lo, b1.hi] and of [b2.lo, b2.hi, b3.lo, b3.hi] on bit 7 of a byte each
  const uint32_t sa = prmt(w4, w, 0xD9C8u) & 0x80808080u, sb = prmt(w4, w, 0xFBEAu) & 0x80808080u;
  if constexpr (std::is_same<T, __half>::value) {
    // 0, .5, 1, 1.5, 2, 3, 4, 6 as fp16: high bytes 00 38 3C 3E 40 42 44 46, low bytes zero
    const uint32_t ha = prmt(0x3E3C3800u, 0x46444240u, m) | sa, hb = prmt(0x3E3C3800u, 0x46444240u, m >> 16) | sb;
    lo01 = prmt(ha, 0u, 0x2404u); hi01 = prmt(ha, 0u, 0x3414u);
    lo23 = prmt(hb, 0u, 0x2404u); hi23 = prmt(hb, 0u, 0x3414u);
  } else {
    // as bf16: 0000 3F00 3F80 3FC0 4000 4040 4080 40C0
    const uint32_t ha = prmt(0x3F3F3F00u, 0x40404040u, m) | sa, hb = prmt(0x3F3F3F00u, 0x40404040u, m >> 16) | sb;
    const uint32_t la = prmt(0xC0800000u, 0xC0804000u, m), lb = prmt(0xC0800000u, 0xC0804000u, m >> 16);
    lo01 = prmt(la, ha, 0x6240u); hi01 = prmt(la, ha, 0x7351u);
    lo23 = prmt(lb, hb, 0x6240u); hi23 = prmt(lb, hb, 0x7351u);
  }
}

constexpr int kGroupWarps = kKC;
constexpr int kMaxSlices = 4;
constexpr int kBarBytes = 256;                  // mbarrier area in front of the ring (up to 32 barriers)

template <int MXC, int NCW> struct RedBuf {
  float red[NCW][kRows][MXC];    // per consumer warp: sum_j ds * S' for (row, activation column)
  float xt[NCW][kRows][MXC];     // per consumer warp: sum_j dm * X (integer path, types with mins)
};

template <int QT, int MXC, int NG, int D, bool RAG> constexpr size_t smem_fixed_bytes() {
  return kBarBytes /* barriers */ + size_t(D) * kRows * stage_pitch<QT, RAG>() + 2 * sizeof(RedBuf<MXC, NG * kGroupWarps>);
}
// Integer path: per super-block and activation row the digit planes, a scale, and (types with mins) the sub-block sums.
template <int QT, int MXC> constexpr size_t smem_planes_bytes(int chunks) {
  return !int_path<QT, MXC>() ? 0 : size_t(MXC) * chunks * kKC * (planes::kSbBytes + sizeof(float) * (1 + (planes::has_mins<QT>() ? (planes::sub16<QT>() ? 16 : 8) : 0)));
}

// The line of units a launch deals to its CTAs: K in `slices` slices of `len` chunks (the first one may be shorter), slice-major, then
// tiles, then the chunks of the slice.  With one slice a CTA walks whole rows of weights.
struct Line {
  int tiles, nchunks, len, slices;
  __host__ __device__ int units() const { return tiles * nchunks; }
  __host__ __device__ int first_len() const { return nchunks - (slices - 1) * len; }
  __host__ __device__ int first_chunk(int slice) const { return slice == 0 ? 0 : first_len() + (slice - 1) * len; }
};
struct Place {                       // one unit of the line: (slice, tile, chunk inside the slice)
  int slice, tile, c, here;          // here: chunks of this slice
  __device__ __forceinline__ Place(const Line& l, int u) {
    slice = 0;
    here = l.first_len();
    for (int units = here * l.tiles; u >= units; units = here * l.tiles) {      // at most kMaxSlices steps
      u -= units;
      ++slice;
      here = l.len;
    }
    tile = u / here;
    c = u - tile * here;
  }
  __device__ __forceinline__ int chunk(const Line& l) const { return l.first_chunk(slice) + c; }
  __device__ __forceinline__ int vt(const Line& l) const { return slice * l.tiles + tile; }      // tile of the line: one slice of a row tile
  __device__ __forceinline__ void back(const Line& l) {        // the unit before
    if (--c >= 0) return;
    if (--tile < 0) { --slice; here = slice == 0 ? l.first_len() : l.len; tile = l.tiles - 1; }
    c = here - 1;
  }
};

// MXC: activation rows covered (power of two >= m, <= 8).  NG: groups of 8 consumer warps.  D: ring slots (D % NG == 0).
// Threads: NG * 8 consumer warps, then the producer warp, then the epilogue warp.
// PROBE: bandwidth probe - the bytes move through the ring exactly as usual, the consumers skip the arithmetic (the
// output is all zeros); it measures what the data path alone sustains for a shape.
template <int QT, typename T, int MXC, int NG, int D, bool PROBE, bool RAG>
__global__ void __launch_bounds__((NG * kGroupWarps + 2) * 32, NG == 1 ? 2 : 1)
gemv_stream_kernel(const T* __restrict__ x, const uint8_t* __restrict__ w, const T* __restrict__ bias, T* __restrict__ y,
                       int m, int n, int k, int* status, uint64_t* partial, uint64_t* slice_words, const Line line, const PeerOut peers,
                       const __grid_constant__ CUtensorMap w_map) {
  using MT = MmaType<T>;
  constexpr int NCW = NG * kGroupWarps;
  constexpr int MC = MXC == 1 ? 1 : 2;             // accumulator columns a lane keeps
  constexpr bool kInt = int_path<QT, MXC>();       // one or two rows: byte operands against digit planes (gemv_int_planes.cuh)
  static_assert(kInt || (!RAG && QT != QTYPE_Q8_0 && !std::is_same<T, float>::value), "the 16-bit operand path needs 16-byte rows and 16-bit activations");
  constexpr int kSbBytes = Geom<QT>::kSbBytes, kPitch = stage_pitch<QT, RAG>(), kStageBytes = kRows * kPitch;
  constexpr bool kB32 = is_blk32<QT>() && !kInt;            // Q4_0 / MXFP4: one scale per 32 weights, two MMAs per block
  constexpr bool kNv = QT == QTYPE_NVFP4;          // a ue4m3 scale per 16 weights, multiplied into the operand (exact)
  constexpr bool kQ23 = is_q23<QT>() && !kInt;              // Q2_K / Q3_K: one MMA per 16-weight sub-block, offsets folded against 16-wide activation sums
  constexpr bool kMinTerm = QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q4_0 || kQ23;   // these fold their mins / offsets against activation sums; Q6_K and the FP4 types have none
  constexpr bool kQ5 = QT == QTYPE_Q5_K;           // Q4_K arithmetic plus the fifth bit of every quant
  // From three activation rows on, the types with folded offsets take the per-sub-block activation sums from the tensor cores (an MMA
  // of the same activation fragment against an all-ones operand).
  constexpr bool kOnes = kMinTerm && !kInt;
  constexpr bool kNeedK = kOnes && (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K || QT == QTYPE_Q2_K);   // types with a min besides the operand offset
  constexpr int kQsOff = kQ5 ? 48 : 16;            // where the nibbles start inside a block
  static_assert(!kInt || NG == 1, "the digit planes belong to one group of consumer warps");
  static_assert(D % NG == 0 && D >= 2 * NG, "every group needs its own ring slots, at least two");
  static_assert(MXC == 1 || MXC == 2 || MXC == 4 || MXC == 8, "MXC");
  using Red = RedBuf<MXC, NCW>;

  extern __shared__ __align__(128) uint8_t smem_dyn[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_dyn);               // full[D], empty[D], red_full[2], red_empty[2]
  uint8_t* sW = smem_dyn + kBarBytes;                                         // D x kStageBytes
  Red* sRed = reinterpret_cast<Red*>(sW + size_t(D) * kStageBytes);      // [2]
  const int nsb = (k + 255) >> 8;
  // integer path: digit planes [MXC][plane_sbs] of the slice at hand, then scales and sums alike
  constexpr int sums_per_sb = planes::sub16<QT>() ? 16 : 8;
  const int plane_sbs = line.len * kKC;
  uint8_t* sPlanes = reinterpret_cast<uint8_t*>(sRed + 2);
  float* sXs = reinterpret_cast<float*>(sPlanes + size_t(MXC) * plane_sbs * planes::kSbBytes);
  float* sX = sXs + MXC * plane_sbs;
  __shared__ __align__(16) float sS[NCW][kRows][planes::sub16<QT>() ? planes::kScalePitch : 8];   // d * sc per row, sub-block (warp-private scratch)
  __shared__ __align__(16) float sK[kNeedK ? NCW : 1][kNeedK ? kRows : 1][QT == QTYPE_Q2_K ? kQ6ScalePitch : 8];   // kOnes: MAGIC * d * sc + dmin * min (Q2_K: dmin * min) per row, sub-block
  constexpr int kTileWords = kRows * MXC, kBatch = MXC >= 4 ? 1 : 128 / kTileWords;      // tiles whose slices the epilogue warp adds at a time
  __shared__ float sOut[kTileWords * kBatch];                            // epilogue warp scratch
  __shared__ int s_abort;
  static_assert((2 * D + 4) * 8 <= kBarBytes, "barrier area");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nchunks = line.nchunks;
  // this CTA's units [u0, u1) of the line; walked from u1 - 1 down
  const int share = line.units() / int(gridDim.x), extra = line.units() - share * int(gridDim.x);
  const int u0 = int(blockIdx.x) * share + min(int(blockIdx.x), extra), u1 = u0 + share + (int(blockIdx.x) < extra ? 1 : 0);
  const int nunits = u1 - u0;
  const Place first(line, u1 - 1), last(line, u0);
  const int t_hi = first.vt(line), ntiles = t_hi - last.vt(line) + 1;      // tiles of the line touched, from t_hi down
  // a tile cut between two CTAs: the lower-numbered CTA walks it first and leaves a partial, the next one adds it and stores
  const bool first_cut = first.c != first.here - 1, last_cut = last.c != 0;
  const int other = int(blockIdx.x) - 1;                                   // the CTA whose partial this one adds
  const int64_t row_bytes = RAG ? int64_t(k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes : int64_t(nsb) * kSbBytes;
  volatile int* abort_flag = &s_abort;

  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * uint32_t(s); };
  auto empty = [&](int s) { return bar0 + 8u * uint32_t(D + s); };
  auto red_full = [&](int b) { return bar0 + 8u * uint32_t(2 * D + b); };
  auto red_empty = [&](int b) { return bar0 + 8u * uint32_t(2 * D + 2 + b); };

  if (tid == 0) {
    for (int s = 0; s < D; ++s) {
      mbar_init(full(s), 1);                    // the producer's arrive.expect_tx; the bytes complete the phase
      mbar_init(empty(s), kGroupWarps);         // one elected arrive per consumer warp of the slot's group
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(red_full(b), NCW);
      mbar_init(red_empty(b), 1);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

  if (warp == NCW) {
    // ------------------------------------------------------------------ producer: weights are constants, no dependency wait
    bool ok = true;
    int issued = 0;
    Place at = first;
    if (tiled_copy<QT, RAG>() && lane == 0) asm volatile("prefetch.tensormap [%0];\n" ::"l"(&w_map) : "memory");
    const uint32_t sW_u32 = smem_u32(sW);
    for (int u = 0; u < nunits; ++u) {
      const int slot = u % D, it = u / D;
      if (it > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty(slot), uint32_t(it - 1) & 1u, abort_flag, status, ST_STREAM_EMPTY) ? 1 : 0) != 0;
        if (!ok) break;
      }
      const int chunk = at.chunk(line), tile = at.tile;
      const int sbs = min(kKC, nsb - chunk * kKC);
      const int rows_valid = min(kRows, n - tile * kRows);
      if constexpr (RAG) {
        // the 16-byte aligned window around this row's piece (up to 15 bytes on either side: never beyond the 16-byte granule of the
        // first and the last byte of the weight)
        const uint8_t* src = w + int64_t(tile * kRows + min(lane, rows_valid - 1)) * row_bytes + int64_t(chunk) * (kKC * kSbBytes);
        const uint32_t phase = uint32_t(reinterpret_cast<uintptr_t>(src)) & 15u;
        const uint32_t piece = uint32_t(min(int64_t(kKC * kSbBytes), row_bytes - int64_t(chunk) * (kKC * kSbBytes)));
        const uint32_t bytes = lane < rows_valid ? (phase + piece + 15u) & ~15u : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_arrive_expect_tx(full(slot), total);
        __syncwarp();
        if (lane < rows_valid) bulk_load(sW_u32 + uint32_t(slot) * kStageBytes + uint32_t(lane) * kPitch, src - phase, bytes, full(slot));
      } else {
       if (tiled_copy<QT, RAG>() && u >= D) {
        // one box of 16 rows x kPitch bytes (the next chunk's first bytes pad the row; past the weight's end: zeros)
        if (lane == 0) {
          mbar_arrive_expect_tx(full(slot), uint32_t(kStageBytes));
          tma_load_2d(sW_u32 + uint32_t(slot) * kStageBytes, &w_map, full(slot), chunk * (kKC * kSbBytes / 8), tile * kRows);
        }
        __syncwarp();
       } else {
        const uint32_t bytes_row = uint32_t(sbs) * kSbBytes;
        if (lane == 0) mbar_arrive_expect_tx(full(slot), uint32_t(rows_valid) * bytes_row);
        __syncwarp();
        if (lane < rows_valid)
          bulk_load(sW_u32 + uint32_t(slot) * kStageBytes + uint32_t(lane) * kPitch,
                    w + int64_t(tile * kRows + lane) * row_bytes + int64_t(chunk) * (kKC * kSbBytes), bytes_row, full(slot));
       }
      }
      issued = u + 1;
      at.back(line);
    }
    if (!ok && lane == 0)       // aborting: the copies still in flight must land before this CTA's shared memory goes away
      for (int v = max(0, issued - D); v < issued; ++v) mbar_wait_plain(full(v % D), uint32_t(v / D) & 1u);
    return;
  }

  // Everything below reads activations / writes outputs that a preceding kernel in the stream may still be producing.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");

  if (warp == NCW + 1) {
    // ------------------------------------------------------------------ epilogue warp
    __shared__ float sPart[kRows * 8];      // the neighbouring CTA's partial sums of the cut tile, fetched as soon as they exist
    bool have_partial = !last_cut;
    // The neighbour's partial sums arrive as 64-bit words {value, 1}: a word is its own flag, so there is no fence and no separate
    // flag to poll (a fenced store, a flag and a second load cost 3 us per launch when every CTA ends on a cut tile).  Fetches
    // them if they are all there (blocking = keep polling, bounded); all lanes return the same answer.
    constexpr int kWords = (kRows * MXC + 31) / 32;
    auto fetch_partial = [&](bool blocking) -> bool {
      uint64_t* theirs = partial + size_t(other) * (kRows * 8);
      uint64_t word[kWords];
      uint64_t start = 0;
      for (uint32_t i = 0; i < kSpinLimit; ++i) {
        bool there = true;
#pragma unroll
        for (int q = 0; q < kWords; ++q) {
          word[q] = 1ull << 32;
          if (lane + 32 * q < kRows * MXC) word[q] = ld_relaxed_gpu(theirs + lane + 32 * q);
          there = there && (word[q] >> 32) != 0;
        }
        if (__all_sync(0xffffffffu, there ? 1 : 0)) {
#pragma unroll
          for (int q = 0; q < kWords; ++q)
            if (lane + 32 * q < kRows * MXC) {
              sPart[lane + 32 * q] = __uint_as_float(uint32_t(word[q]));
              st_relaxed_gpu(theirs + lane + 32 * q, 0);            // emptied by its only reader: nothing to clear between launches
            }
          __syncwarp();
          return true;
        }
        if (!blocking) return false;
        if ((i & 63u) == 0u) {
          const uint64_t now = globaltimer_ns();
          if (i == 0) start = now;
          if (__any_sync(0xffffffffu, (*abort_flag || now - start > kWaitLimitNs) ? 1 : 0)) break;
        }
      }
      if (lane == 0) { *abort_flag = 1; atomicCAS(status, 0, ST_STREAM_PARTIAL); }
      return false;
    };
    auto store_tile = [&](int tile, const float* sOut) {
      for (int idx = lane; idx < kRows * MXC; idx += 32) {
        const int r = idx & (kRows - 1), c = idx >> 4;
        const int row = tile * kRows + r;
        if (row >= n || c >= m) continue;
        float v = sOut[idx];
        int64_t at = int64_t(c) * n + row;
        if (peers.act != ACT_NONE) {
          // gated pair: rows r < 8 of the tile belong to the first matrix, r + 8 to the second; output has n / 2 columns
          if (r >= 8) continue;
          float u = sOut[idx + 8];
          if (bias != nullptr) {           // interleaved like the rows: bias0 of the gate row, bias1 of its up row
            v += MT::to_float(bias[row]);
            u += MT::to_float(bias[row + 8]);
          }
          v = gate_activation(v, peers.act) * u;
          at = int64_t(c) * (n >> 1) + (tile * 8 + r);
        } else if (bias != nullptr) {
          v += MT::to_float(bias[row]);
        }
        const T out = MT::from_float(v);
        y[at] = out;
#pragma unroll
        for (int pi = 0; pi < 8; ++pi)
          if (pi < peers.count) static_cast<T*>(peers.ptr[pi])[at] = out;
      }
    };
    // Sums over the slices of `count` tiles from `tile` on -> sOut, all loads in flight together; the words are emptied.  Bounded
    // like every wait.
    auto gather_slices = [&](int tile, int count) -> bool {
      constexpr int kPer = (kTileWords * kBatch + 31) / 32;
      uint64_t word[kMaxSlices][kPer];
      const uint64_t start = globaltimer_ns();
      auto at = [&](int sl, int q) -> uint64_t* {
        const int i = lane + 32 * q, ti = i / kTileWords;
        return slice_words + (size_t(tile + ti) * line.slices + sl) * kTileWords + (i - ti * kTileWords);
      };
      for (uint32_t i = 0; i < kSpinLimit; ++i) {
        bool there = true;
#pragma unroll
        for (int sl = 0; sl < kMaxSlices; ++sl)
#pragma unroll
          for (int q = 0; q < kPer; ++q) {
            word[sl][q] = 1ull << 32;
            if (sl < line.slices && lane + 32 * q < count * kTileWords) word[sl][q] = ld_relaxed_gpu(at(sl, q));
            there = there && (word[sl][q] >> 32) != 0;
          }
        if (__all_sync(0xffffffffu, there ? 1 : 0)) {
#pragma unroll
          for (int q = 0; q < kPer; ++q)
            if (lane + 32 * q < count * kTileWords) {
              float sum = 0.f;
#pragma unroll
              for (int sl = 0; sl < kMaxSlices; ++sl)
                if (sl < line.slices) {
                  sum += __uint_as_float(uint32_t(word[sl][q]));
                  st_relaxed_gpu(at(sl, q), 0);
                }
              sOut[lane + 32 * q] = sum;
            }
          __syncwarp();
          return true;
        }
        if ((i & 63u) == 63u && __any_sync(0xffffffffu, (*abort_flag || globaltimer_ns() - start > kWaitLimitNs) ? 1 : 0)) break;
      }
      if (lane == 0) { *abort_flag = 1; atomicCAS(status, 0, ST_STREAM_PARTIAL); }
      return false;
    };
    for (int tl = 0; tl < ntiles; ++tl) {
      const int buf = tl & 1;
      if (!have_partial) have_partial = fetch_partial(false);      // off the critical path: the neighbour wrote it at its start
      if (!(__all_sync(0xffffffffu, mbar_wait(red_full(buf), uint32_t(tl >> 1) & 1u, abort_flag, status, ST_STREAM_RED_FULL) ? 1 : 0))) break;
      const Red& rb = sRed[buf];
      for (int idx = lane; idx < kRows * MXC; idx += 32) {
        const int r = idx & (kRows - 1), c = idx >> 4;
        float v = 0.f, xs = 0.f;
#pragma unroll
        for (int wv = 0; wv < NCW; ++wv) {
          v += rb.red[wv][r][c];
          if constexpr (kInt && planes::has_mins<QT>()) xs += rb.xt[wv][r][c];
        }
        sOut[idx] = v - xs;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(red_empty(buf));
      const int vt = t_hi - tl, slice = line.slices == 1 ? 0 : vt / line.tiles, tile = vt - slice * line.tiles;
      if (tl == 0 && first_cut) {
        // the rest of this tile belongs to the neighbouring CTA, which reaches it last: leave the partial sums
        uint64_t* mine = partial + size_t(blockIdx.x) * (kRows * 8);
        for (int idx = lane; idx < kRows * MXC; idx += 32) st_relaxed_gpu(mine + idx, (1ull << 32) | __float_as_uint(sOut[idx]));
        __syncwarp();                         // sOut is rewritten for the next tile
        continue;
      }
      if (tl == ntiles - 1 && last_cut) {
        // the other chunks of this tile were computed by the neighbouring CTA at the start of its walk
        if (!have_partial) have_partial = fetch_partial(true);
        if (!have_partial) break;
        for (int idx = lane; idx < kRows * MXC; idx += 32) sOut[idx] += sPart[idx];
        __syncwarp();
      }
      if (line.slices > 1) {                // one slice of the tile's K: leave the sums for the CTA that has the last slice
        uint64_t* slot = slice_words + (size_t(tile) * line.slices + slice) * (kRows * MXC);
        for (int idx = lane; idx < kRows * MXC; idx += 32) st_relaxed_gpu(slot + idx, (1ull << 32) | __float_as_uint(sOut[idx]));
      } else {
        store_tile(tile, sOut);
      }
      __syncwarp();                         // sOut is rewritten for the next tile
    }
    // The tiles whose last slice was this CTA's: add the slices in order (they belong to lower-numbered CTAs) and store.
    if (line.slices > 1) {
      const int done_hi = first_cut ? t_hi - 1 : t_hi, done_lo = max(t_hi - ntiles + 1, (line.slices - 1) * line.tiles);
      for (int vt = done_lo; vt <= done_hi; vt += kBatch) {
        const int tile = vt - (line.slices - 1) * line.tiles, count = min(kBatch, done_hi - vt + 1);
        if (!gather_slices(tile, count)) break;
        for (int i = 0; i < count; ++i) store_tile(tile + i, sOut + i * kTileWords);
        __syncwarp();
      }
    }
    return;
  }

  // -------------------------------------------------------------------- consumer warps
  const int cw = warp, grp = cw / kGroupWarps, wq = cw % kGroupWarps;
  const int g = lane >> 2, t = lane & 3;
  const int srow = lane >> 1, shalf = lane & 1;   // scale-decode role of this lane

  if constexpr (kInt) {
    // A warp meets the super-blocks wq, wq + 8, ... of every tile, so it makes the digit planes of exactly those, each when it first
    // meets it: nothing is shared between warps and no barrier stands between the activations and the first weights.
    for (int sb = line.first_chunk(first.slice) * kKC + wq; sb < min(nsb, line.first_chunk(first.slice + 1) * kKC); sb += kKC)
#pragma unroll
      for (int c = 0; c < MXC; ++c)
        if (sb * 256 + 8 * lane < k) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(x + int64_t(c) * k + sb * 256 + 8 * lane));
    uint32_t made = 0;                          // chunks of the slice at hand whose planes exist (32 of them do not fit into shared memory)
    int slice = first.slice;
    float ires[2] = {0.f, 0.f}, xt[MXC];
#pragma unroll
    for (int c = 0; c < MXC; ++c) xt[c] = 0.f;
    int slot = 0, left = nunits;
    uint32_t parity = 0;
    Place at = first;
    for (int tl = 0; tl < ntiles; ++tl) {
      const int here = min(left, at.c + 1), row_tile = at.tile;       // units of this tile
      left -= here;
      if (at.slice != slice) { slice = at.slice; made = 0; }
      for (int i = 0; i < here; ++i, at.back(line)) {
        const int sb = at.chunk(line) * kKC + wq, psb = at.c * kKC + wq;
        if (!PROBE && sb < nsb && !((made >> at.c) & 1u)) {
          made |= 1u << at.c;
#pragma unroll
          for (int c = 0; c < MXC; ++c)
            planes::make<QT, T>(x + int64_t(c) * k + sb * 256, k - sb * 256, lane, sPlanes + size_t(c * plane_sbs + psb) * planes::kSbBytes,
                                sXs + c * plane_sbs + psb, sX + (c * plane_sbs + psb) * sums_per_sb);
          __syncwarp();
        }
        if (!__all_sync(0xffffffffu, mbar_wait(full(slot), parity, abort_flag, status, ST_STREAM_FULL) ? 1 : 0)) return;
        if (!PROBE && sb < nsb) {
          const uint8_t* st = sW + slot * kStageBytes + wq * kSbBytes;
          const uint8_t *bs = st + srow * kPitch, *b0 = st + g * kPitch, *b1 = st + (g + 8) * kPitch;
          if constexpr (RAG) {
            const uintptr_t piece = reinterpret_cast<uintptr_t>(w) + uintptr_t(int64_t(at.chunk(line)) * (kKC * kSbBytes));
            const int row0 = row_tile * kRows;
            auto phase = [&](int r) { return int((piece + uintptr_t(int64_t(min(row0 + r, n - 1)) * row_bytes)) & 15); };
            bs += phase(srow); b0 += phase(g); b1 += phase(g + 8);
          }
          const uint8_t* xp = sPlanes + psb * planes::kSbBytes;
          const int blocks = RAG ? min(8, (k - sb * 256) / QTraits<QT>::kBlock) : 8;
          constexpr bool kTwoByteBlocks = QT == QTYPE_Q6_K || QT == QTYPE_Q3_K;      // odd super-blocks of a stage start 2 bytes off a word boundary
          float scale;
          if (!RAG && kTwoByteBlocks && (wq & 1))
            scale = planes::superblock<QT, MXC, true, false>(bs, b0, b1, sS[cw], xp, plane_sbs * planes::kSbBytes, sXs + psb, plane_sbs, sX + psb * sums_per_sb,
                                                             plane_sbs * sums_per_sb, blocks, lane, ires, xt);
          else
            scale = planes::superblock<QT, MXC, false, RAG>(bs, b0, b1, sS[cw], xp, plane_sbs * planes::kSbBytes, sXs + psb, plane_sbs, sX + psb * sums_per_sb,
                                                            plane_sbs * sums_per_sb, blocks, lane, ires, xt);
          if (__builtin_expect(__any_sync(0xffffffffu, scale == 0.f), 0)) {
            const float2 rest = planes::plain<QT, T, MXC>(b0, b1, x + int64_t(MXC == 2 ? t >> 1 : 0) * k + sb * 256, min(256, k - sb * 256), scale == 0.f, t);
            ires[0] += rest.x;
            ires[1] += rest.y;
          }
        }
        __syncwarp();                            // every lane is done with the stage (and with sS)
        if (lane == 0) mbar_arrive(empty(slot));
        if (++slot == D) { slot = 0; parity ^= 1u; }
      }
      // hand the tile's sums to the epilogue warp
      const int buf = tl & 1;
      if (tl >= 2 && !__all_sync(0xffffffffu, mbar_wait(red_empty(buf), uint32_t((tl >> 1) - 1) & 1u, abort_flag, status, ST_STREAM_RED_EMPTY) ? 1 : 0)) return;
      Red& rb = sRed[buf];
      planes::join<QT, MXC>(ires);
      if ((t & 1) == 0 && (t >> 1) < MXC) {
        rb.red[cw][g][t >> 1] = ires[0];
        rb.red[cw][g + 8][t >> 1] = ires[1];
      }
      ires[0] = ires[1] = 0.f;
      if constexpr (planes::has_mins<QT>()) {
#pragma unroll
        for (int c = 0; c < MXC; ++c) {
          const float both = xt[c] + __shfl_xor_sync(0xffffffffu, xt[c], 1);
          if (shalf == 0) rb.xt[cw][srow][c] = both;
          xt[c] = 0.f;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(red_full(buf));
    }
    return;
  }
  if constexpr (!kInt) {
  float res[1][4] = {{0.f, 0.f, 0.f, 0.f}};
  float zero4[4];
  opaque_zero4(zero4);
  const T* xbase = x + int64_t(min(g, m - 1)) * k;   // rows >= m read a clamped (valid) row; their columns are never stored
  const T* xrow = xbase + 8 * t;

  bool ok = true;
  int cur_tile = 0;                             // tile (local index) the accumulators belong to
  auto flush = [&](int tl) {
    const int buf = tl & 1;
    if (tl >= 2) ok = __all_sync(0xffffffffu, mbar_wait(red_empty(buf), uint32_t((tl >> 1) - 1) & 1u, abort_flag, status, ST_STREAM_RED_EMPTY) ? 1 : 0) != 0;
    if (!ok) return;
    Red& rb = sRed[buf];
    if (2 * t < MXC) {
      rb.red[cw][g][2 * t] = res[0][0];
      rb.red[cw][g + 8][2 * t] = res[0][2];
      if (MC == 2) {
        rb.red[cw][g][2 * t + 1] = res[0][1];
        rb.red[cw][g + 8][2 * t + 1] = res[0][3];
      }
    }
    res[0][0] = res[0][1] = res[0][2] = res[0][3] = 0.f;
    __syncwarp();
    if (lane == 0) mbar_arrive(red_full(buf));
  };

  // local unit u is unit u1 - 1 - u of the line: its chunk counts down, its local tile index up
  int tl = 0, chunk = first.c - grp;            // one slice: the chunk inside the slice is the chunk
  while (chunk < 0 && tl < ntiles) { chunk += nchunks; ++tl; }
  for (int u = grp; u < nunits && ok; u += NG) {
    while (cur_tile < tl && ok) { flush(cur_tile); ++cur_tile; }
    if (!ok) break;
    const int slot = u % D;
    ok = __all_sync(0xffffffffu, mbar_wait(full(slot), uint32_t(u / D) & 1u, abort_flag, status, ST_STREAM_FULL) ? 1 : 0) != 0;
    if (!ok) break;
    const int sb = chunk * kKC + wq;
    if (!PROBE && sb < nsb && kB32) {
      if constexpr (kB32) {
        constexpr int BB = QT == QTYPE_Q4_0 ? 18 : 17, QOFF = BB - 16;       // block bytes, where its 16 nibble bytes start
        const uint8_t* st = sW + size_t(slot) * kStageBytes + wq * kSbBytes;
        {  // lane pair (srow, shalf): the scales of blocks 4*shalf .. +3 of row srow -> shared memory; Q4_0's offset folded against X
          const uint8_t* sp = st + srow * kPitch + 4 * shalf * BB;
          float4 dsv;
          float* dsf = reinterpret_cast<float*>(&dsv);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if constexpr (QT == QTYPE_Q4_0) dsf[i] = half_bits_to_float(*reinterpret_cast<const uint16_t*>(sp + BB * i));
            else dsf[i] = __fmul_rn(e8m0_half(sp[BB * i]), 2.f);             // 2^(e - 127): the operands are the e2m1 values themselves
          }
          *reinterpret_cast<float4*>(&sS[cw][srow][4 * shalf]) = dsv;
        }
        __syncwarp();
        const float4 dsa0 = *reinterpret_cast<const float4*>(&sS[cw][g][0]);
        const float4 dsa1 = *reinterpret_cast<const float4*>(&sS[cw][g][4]);
        const float4 dsb0 = *reinterpret_cast<const float4*>(&sS[cw][g + 8][0]);
        const float4 dsb1 = *reinterpret_cast<const float4*>(&sS[cw][g + 8][4]);
        const float ds_a[8] = {dsa0.x, dsa0.y, dsa0.z, dsa0.w, dsa1.x, dsa1.y, dsa1.z, dsa1.w};
        const float ds_b[8] = {dsb0.x, dsb0.y, dsb0.z, dsb0.w, dsb1.x, dsb1.y, dsb1.z, dsb1.w};
        // Byte j of a block holds weight j (low nibble) and weight 16 + j (high nibble).  Lane t takes bytes 4t .. 4t+3 of rows g
        // and g + 8: its low nibbles are weights 4t .. 4t+3 (first MMA of the block: K slots 2t, 2t+1 and 2t+8, 2t+9), its high
        // nibbles weights 16 + 4t .. (second MMA); the activations follow the same order (two 8-byte loads per block).
        const uint8_t* r0 = st + g * kPitch + 4 * t;
        const uint8_t* r1 = r0 + 8 * kPitch;
        const T* xs = xbase + 4 * t + sb * 256;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const int o = BB * b + QOFF, oa = o & ~3, sh = 8 * (o & 3);         // constants after unrolling; blocks are 1- / 2-byte aligned
          uint32_t w0 = *reinterpret_cast<const uint32_t*>(r0 + oa), w1 = *reinterpret_cast<const uint32_t*>(r1 + oa);
          if (sh != 0) {
            w0 = __funnelshift_r(w0, *reinterpret_cast<const uint32_t*>(r0 + oa + 4), sh);
            w1 = __funnelshift_r(w1, *reinterpret_cast<const uint32_t*>(r1 + oa + 4), sh);
          }
          uint32_t a_lo[4], a_hi[4];
          if constexpr (QT == QTYPE_Q4_0) {
            const uint32_t l0 = w0 & 0x0f0f0f0fu, h0 = (w0 >> 4) & 0x0f0f0f0fu, l1 = w1 & 0x0f0f0f0fu, h1 = (w1 >> 4) & 0x0f0f0f0fu;
            a_lo[0] = MT::fix(__byte_perm(l0, MT::kMagicBytes, 0x4140)); a_lo[1] = MT::fix(__byte_perm(l1, MT::kMagicBytes, 0x4140));
            a_lo[2] = MT::fix(__byte_perm(l0, MT::kMagicBytes, 0x4342)); a_lo[3] = MT::fix(__byte_perm(l1, MT::kMagicBytes, 0x4342));
            a_hi[0] = MT::fix(__byte_perm(h0, MT::kMagicBytes, 0x4140)); a_hi[1] = MT::fix(__byte_perm(h1, MT::kMagicBytes, 0x4140));
            a_hi[2] = MT::fix(__byte_perm(h0, MT::kMagicBytes, 0x4342)); a_hi[3] = MT::fix(__byte_perm(h1, MT::kMagicBytes, 0x4342));
          } else {
            fp4x8_operands<T>(w0, a_lo[0], a_lo[2], a_hi[0], a_hi[2]);
            fp4x8_operands<T>(w1, a_lo[1], a_lo[3], a_hi[1], a_hi[3]);
          }
          const uint2 xa = __ldg(reinterpret_cast<const uint2*>(xs + 32 * b));
          const uint2 xb = __ldg(reinterpret_cast<const uint2*>(xs + 32 * b + 16));
          float acc[4];
          MT::mma_c(acc, a_lo, xa.x, xa.y, zero4);
          MT::mma(acc, a_hi, xb.x, xb.y);
          if constexpr (kOnes) {               // Q4_0: sum of (MAGIC + q) x  ->  sum of (q - 8) x with the block's activation sums
            const uint32_t ones[4] = {MT::kOnePair, MT::kOnePair, MT::kOnePair, MT::kOnePair};
            float sx[4];
            MT::mma_c(sx, ones, xa.x, xa.y, zero4);
            MT::mma(sx, ones, xb.x, xb.y);
            constexpr float kOff = MT::kMagic + 8.f;
            acc[0] = fmaf(-kOff, sx[0], acc[0]);
            acc[2] = fmaf(-kOff, sx[0], acc[2]);
            if (MC == 2) {
              acc[1] = fmaf(-kOff, sx[1], acc[1]);
              acc[3] = fmaf(-kOff, sx[1], acc[3]);
            }
          }
          res[0][0] = fmaf(ds_a[b], acc[0], res[0][0]);
          res[0][2] = fmaf(ds_b[b], acc[2], res[0][2]);
          if (MC == 2) {
            res[0][1] = fmaf(ds_a[b], acc[1], res[0][1]);
            res[0][3] = fmaf(ds_b[b], acc[3], res[0][3]);
          }
        }
      }
    } else if (!PROBE && sb < nsb && kQ23) {
      if constexpr (kQ23) {
        // Q2_K: scales[16] (4-bit scale, 4-bit min per 16 weights), qs[64], d, dmin.  Q3_K: hmask[32], qs[64], scales[12] (6-bit), d.
        // Weight 128*hb + 32*j + l is bits 2j, 2j+1 of qs[32*hb + l] (Q3_K: plus bit 4*hb + j of hmask[l] as a third bit, less 4);
        // sub-block (hb, j, h16) = its weights l = 16*h16 .. +15, scale index 8*hb + 2*j + h16.  One MMA per sub-block.
        constexpr int kQs = QT == QTYPE_Q2_K ? 16 : 32;
        const uint8_t* st = sW + size_t(slot) * kStageBytes + wq * kSbBytes;
        {  // lane pair (srow, shalf): the eight sub-block scales of half-block shalf of row srow
          const uint8_t* blk = st + srow * kPitch;
          float dsf[8], dmv[8];                // d * scale; Q2_K: dmin * min
          if constexpr (QT == QTYPE_Q2_K) {
            const float d = half_at(blk + 80), dmin = half_at(blk + 82);
            const uint32_t* scp = reinterpret_cast<const uint32_t*>(blk + 8 * shalf);   // blocks (84 B) are word aligned, not more
            const uint32_t sc0 = scp[0], sc1 = scp[1];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint32_t b = ((i < 4 ? sc0 : sc1) >> (8 * (i & 3))) & 0xffu;
              dsf[i] = d * float(b & 0x0fu);
              dmv[i] = dmin * float(b >> 4);
            }
          } else {
            const float d = half_at(blk + 108);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              dsf[i] = d * float(q3k_scale(blk + 96, 8 * shalf + i) - 32);
              dmv[i] = 0.f;
            }
          }
          *reinterpret_cast<float4*>(&sS[cw][srow][8 * shalf]) = make_float4(dsf[0], dsf[1], dsf[2], dsf[3]);
          *reinterpret_cast<float4*>(&sS[cw][srow][8 * shalf + 4]) = make_float4(dsf[4], dsf[5], dsf[6], dsf[7]);
          if constexpr (kNeedK) {                 // Q2_K: dmin * min, applied to the sums from the tensor cores below
            *reinterpret_cast<float4*>(&sK[cw][srow][8 * shalf]) = make_float4(dmv[0], dmv[1], dmv[2], dmv[3]);
            *reinterpret_cast<float4*>(&sK[cw][srow][8 * shalf + 4]) = make_float4(dmv[4], dmv[5], dmv[6], dmv[7]);
          }
        }
        __syncwarp();
        // Lane t takes bytes 4t .. 4t+3 of every 16-byte run of rows g and g + 8: four weights of each of the four sub-blocks
        // (j = 0..3) that share those bytes; K slots 2t, 2t+1 and 2t+8, 2t+9 carry them, the activations follow the same order.
        // Q3_K blocks (110 B) sit 2 bytes off a word boundary in every odd super-block: two aligned loads and a funnel shift.
        const uint32_t sh = (QT == QTYPE_Q3_K) ? 16u * uint32_t(wq & 1) : 0u;
        auto word = [&](const uint8_t* p) -> uint32_t {      // 4 bytes at p, p being `sh / 8` bytes past a word boundary
          if constexpr (QT == QTYPE_Q3_K) {
            const uint32_t* a = reinterpret_cast<const uint32_t*>(p - (sh >> 3));
            return __funnelshift_r(a[0], a[1], sh);
          } else {
            return *reinterpret_cast<const uint32_t*>(p);
          }
        };
        const uint8_t* r0 = st + g * kPitch + 4 * t;
        const uint8_t* r1 = r0 + 8 * kPitch;
        const T* xs = xbase + 4 * t + sb * 256;
#pragma unroll
        for (int h16 = 0; h16 < 2; ++h16) {
          uint32_t hm0 = 0, hm1 = 0;
          if constexpr (QT == QTYPE_Q3_K) { hm0 = word(r0 + 16 * h16); hm1 = word(r1 + 16 * h16); }
#pragma unroll
          for (int hb = 0; hb < 2; ++hb) {
            const uint32_t w0 = word(r0 + kQs + 32 * hb + 16 * h16), w1 = word(r1 + kQs + 32 * hb + 16 * h16);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t n0 = (w0 >> (2 * j)) & 0x03030303u, n1 = (w1 >> (2 * j)) & 0x03030303u;
              if constexpr (QT == QTYPE_Q3_K) {
                n0 |= ((hm0 >> (4 * hb + j)) & 0x01010101u) << 2;
                n1 |= ((hm1 >> (4 * hb + j)) & 0x01010101u) << 2;
              }
              const uint32_t a[4] = {MT::fix(__byte_perm(n0, MT::kMagicBytes, 0x4140)), MT::fix(__byte_perm(n1, MT::kMagicBytes, 0x4140)),
                                     MT::fix(__byte_perm(n0, MT::kMagicBytes, 0x4342)), MT::fix(__byte_perm(n1, MT::kMagicBytes, 0x4342))};
              const uint2 xa = __ldg(reinterpret_cast<const uint2*>(xs + 128 * hb + 32 * j + 16 * h16));
              float acc[4];
              MT::mma_c(acc, a, xa.x, xa.y, zero4);
              const int idx = 8 * hb + 2 * j + h16;
              const float da = sS[cw][g][idx], db = sS[cw][g + 8][idx];      // 16 scales per row: read where used, not held in registers
              if constexpr (kOnes) {             // the operand offset (and Q2_K's min) against the sub-block's activation sums
                const uint32_t ones[4] = {MT::kOnePair, MT::kOnePair, MT::kOnePair, MT::kOnePair};
                float sx[4];
                MT::mma_c(sx, ones, xa.x, xa.y, zero4);
                constexpr float kOff = MT::kMagic + (QT == QTYPE_Q3_K ? 4.f : 0.f);
                acc[0] = fmaf(-kOff, sx[0], acc[0]);
                acc[2] = fmaf(-kOff, sx[0], acc[2]);
                if (MC == 2) {
                  acc[1] = fmaf(-kOff, sx[1], acc[1]);
                  acc[3] = fmaf(-kOff, sx[1], acc[3]);
                }
                if constexpr (QT == QTYPE_Q2_K) {
                  const float ma = sK[cw][g][idx], mb = sK[cw][g + 8][idx];
                  res[0][0] = fmaf(-ma, sx[0], res[0][0]);
                  res[0][2] = fmaf(-mb, sx[0], res[0][2]);
                  if (MC == 2) {
                    res[0][1] = fmaf(-ma, sx[1], res[0][1]);
                    res[0][3] = fmaf(-mb, sx[1], res[0][3]);
                  }
                }
              }
              res[0][0] = fmaf(da, acc[0], res[0][0]);
              res[0][2] = fmaf(db, acc[2], res[0][2]);
              if (MC == 2) {
                res[0][1] = fmaf(da, acc[1], res[0][1]);
                res[0][3] = fmaf(db, acc[3], res[0][3]);
              }
            }
          }
        }
      }
    } else if (!PROBE && sb < nsb && kNv) {
      if constexpr (kNv) {
        // Four blocks of 64 weights (four ue4m3 scales, 32 bytes of nibbles).  Lane t owns sub-block t of every block for rows g
        // and g + 8: 8 bytes whose byte i holds weights i (low nibble) and 8 + i (high nibble).  Value x scale is exact in either
        // 16-bit type (2 + 4 significant bits), so the operand is the dequantized weight itself and nothing is applied after
        // the MMA; the four MMAs of a block take weights 4j .. 4j+3 of every sub-block (K slots 2t, 2t+1, 2t+8, 2t+9), the
        // activations follow the same order: 16 consecutive values per lane and block.
        const uint8_t* st = sW + size_t(slot) * kStageBytes + wq * kSbBytes;
        const uint8_t* r0 = st + g * kPitch;
        const uint8_t* r1 = r0 + 8 * kPitch;
        const T* xs = xbase + sb * 256 + 16 * t;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint32_t s0 = splat_pair<T>(__fmul_rn(ue4m3_half(r0[36 * b + t]), 2.f));
          const uint32_t s1 = splat_pair<T>(__fmul_rn(ue4m3_half(r1[36 * b + t]), 2.f));
          uint32_t a[4][4];           // [MMA j][fragment register]
#pragma unroll
          for (int i = 0; i < 2; ++i) {   // word i: low nibbles -> MMA i, high nibbles -> MMA 2 + i
            const uint32_t w0 = *reinterpret_cast<const uint32_t*>(r0 + 36 * b + 4 + 8 * t + 4 * i);
            const uint32_t w1 = *reinterpret_cast<const uint32_t*>(r1 + 36 * b + 4 + 8 * t + 4 * i);
            fp4x8_operands<T>(w0, a[i][0], a[i][2], a[2 + i][0], a[2 + i][2]);
            fp4x8_operands<T>(w1, a[i][1], a[i][3], a[2 + i][1], a[2 + i][3]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            a[j][0] = mul_pair<T>(a[j][0], s0); a[j][2] = mul_pair<T>(a[j][2], s0);
            a[j][1] = mul_pair<T>(a[j][1], s1); a[j][3] = mul_pair<T>(a[j][3], s1);
          }
          const uint4 xa = __ldg(reinterpret_cast<const uint4*>(xs + 64 * b));
          const uint4 xb = __ldg(reinterpret_cast<const uint4*>(xs + 64 * b + 8));
          float acc[4];
          MT::mma_c(acc, a[0], xa.x, xa.y, zero4);
          MT::mma(acc, a[1], xa.z, xa.w);
          MT::mma(acc, a[2], xb.x, xb.y);
          MT::mma(acc, a[3], xb.z, xb.w);
          res[0][0] += acc[0];
          res[0][2] += acc[2];
          if (MC == 2) {
            res[0][1] += acc[1];
            res[0][3] += acc[3];
          }
        }
      }
    } else if (!PROBE && sb < nsb && QT == QTYPE_Q6_K) {
      if constexpr (QT == QTYPE_Q6_K && !kInt) {
        // row pitch and stage size are multiples of 4, so a block's phase against a word boundary is that of wq * 210
        const uint8_t* st = sW + size_t(slot) * kStageBytes + wq * kSbBytes;
        const T* const xr[1] = {xbase + 4 * t};                // this lane's four K positions of every 16-wide sub-block
        if (wq & 1)
          q6k_superblock<T, 1, MC, Q6_ODD>(st + srow * kPitch, st + g * kPitch, st + (g + 8) * kPitch, sS[cw], xr, sb, lane, res);
        else
          q6k_superblock<T, 1, MC, Q6_ALIGNED>(st + srow * kPitch, st + g * kPitch, st + (g + 8) * kPitch, sS[cw], xr, sb, lane, res);
      }
    } else if (!PROBE && sb < nsb && !kB32 && !kNv && !kQ23) {
     if constexpr (QT == QTYPE_Q4_K || QT == QTYPE_Q5_K) if constexpr (!kInt) {
      const uint8_t* st = sW + size_t(slot) * kStageBytes + wq * kSbBytes;
      {  // lane pair (srow, shalf): 4 sub-block scales -> ds to shared memory, min/MAGIC term folded against X
        const uint4 hdr = *reinterpret_cast<const uint4*>(st + srow * kPitch);
        const float d = half_bits_to_float(uint16_t(hdr.x & 0xffffu));
        const float dmin = half_bits_to_float(uint16_t(hdr.x >> 16));
        // sub-blocks 0..3 keep their 6-bit fields in place; 4..7 are split across two bytes
        const uint32_t sc_lo = hdr.y & 0x3f3f3f3fu, mn_lo = hdr.z & 0x3f3f3f3fu;
        const uint32_t sc_hi = (hdr.w & 0x0f0f0f0fu) | (((hdr.y >> 6) & 0x03030303u) << 4);
        const uint32_t mn_hi = ((hdr.w >> 4) & 0x0f0f0f0fu) | (((hdr.z >> 6) & 0x03030303u) << 4);
        const uint32_t scb = shalf ? sc_hi : sc_lo, mnb = shalf ? mn_hi : mn_lo;
        float4 dsv;
        float kk[4];
        float* dsf = reinterpret_cast<float*>(&dsv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dsf[i] = d * byte_to_float(scb, i);
          kk[i] = fmaf(MT::kMagic, dsf[i], dmin * byte_to_float(mnb, i));
        }
        *reinterpret_cast<float4*>(&sS[cw][srow][4 * shalf]) = dsv;
        if constexpr (kOnes) *reinterpret_cast<float4*>(&sK[cw][srow][4 * shalf]) = make_float4(kk[0], kk[1], kk[2], kk[3]);
      }
      __syncwarp();
      const float4 dsa0 = *reinterpret_cast<const float4*>(&sS[cw][g][0]);
      const float4 dsa1 = *reinterpret_cast<const float4*>(&sS[cw][g][4]);
      const float4 dsb0 = *reinterpret_cast<const float4*>(&sS[cw][g + 8][0]);
      const float4 dsb1 = *reinterpret_cast<const float4*>(&sS[cw][g + 8][4]);
      const float ds_a[8] = {dsa0.x, dsa0.y, dsa0.z, dsa0.w, dsa1.x, dsa1.y, dsa1.z, dsa1.w};
      const float ds_b[8] = {dsb0.x, dsb0.y, dsb0.z, dsb0.w, dsb1.x, dsb1.y, dsb1.z, dsb1.w};
      const uint8_t* q0p = st + g * kPitch + kQsOff + 8 * t;
      const uint8_t* q1p = q0p + 8 * kPitch;
      const T* xs = xrow + sb * 256;
      // Q5_K: bit 2G+h of qh byte l is the fifth bit of weight l of sub-block 2G+h; this lane's eight l are bytes 8t .. 8t+7
      uint2 qh0 = make_uint2(0u, 0u), qh1 = make_uint2(0u, 0u);
      if constexpr (kQ5) {
        qh0 = *reinterpret_cast<const uint2*>(st + g * kPitch + 16 + 8 * t);
        qh1 = *reinterpret_cast<const uint2*>(st + (g + 8) * kPitch + 16 + 8 * t);
      }
#pragma unroll
      for (int G = 0; G < 4; ++G) {
        const uint2 q0 = *reinterpret_cast<const uint2*>(q0p + 32 * G);
        const uint2 q1 = *reinterpret_cast<const uint2*>(q1p + 32 * G);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t n0x = (h ? q0.x >> 4 : q0.x) & 0x0f0f0f0fu, n0y = (h ? q0.y >> 4 : q0.y) & 0x0f0f0f0fu;
          uint32_t n1x = (h ? q1.x >> 4 : q1.x) & 0x0f0f0f0fu, n1y = (h ? q1.y >> 4 : q1.y) & 0x0f0f0f0fu;
          if constexpr (kQ5) {               // q = nibble + 16 * bit: still an exact 128 + q operand (q <= 31)
            constexpr uint32_t kBit = 0x01010101u;
            n0x |= ((qh0.x >> (2 * G + h)) & kBit) * 16u;
            n0y |= ((qh0.y >> (2 * G + h)) & kBit) * 16u;
            n1x |= ((qh1.x >> (2 * G + h)) & kBit) * 16u;
            n1y |= ((qh1.y >> (2 * G + h)) & kBit) * 16u;
          }
          const uint32_t a_lo[4] = {MT::fix(__byte_perm(n0x, MT::kMagicBytes, 0x4140)), MT::fix(__byte_perm(n1x, MT::kMagicBytes, 0x4140)),
                                    MT::fix(__byte_perm(n0x, MT::kMagicBytes, 0x4342)), MT::fix(__byte_perm(n1x, MT::kMagicBytes, 0x4342))};
          const uint32_t a_hi[4] = {MT::fix(__byte_perm(n0y, MT::kMagicBytes, 0x4140)), MT::fix(__byte_perm(n1y, MT::kMagicBytes, 0x4140)),
                                    MT::fix(__byte_perm(n0y, MT::kMagicBytes, 0x4342)), MT::fix(__byte_perm(n1y, MT::kMagicBytes, 0x4342))};
          // rows >= m read a clamped (valid) row; their accumulator columns are never stored
          const uint4 xb = __ldg(reinterpret_cast<const uint4*>(xs + 64 * G + 32 * h));
          float acc[4];
          MT::mma_c(acc, a_lo, xb.x, xb.y, zero4);
          MT::mma(acc, a_hi, xb.z, xb.w);
          const float dsr0 = ds_a[2 * G + h], dsr1 = ds_b[2 * G + h];
          res[0][0] = fmaf(dsr0, acc[0], res[0][0]);
          res[0][2] = fmaf(dsr1, acc[2], res[0][2]);
          if (MC == 2) {
            res[0][1] = fmaf(dsr0, acc[1], res[0][1]);
            res[0][3] = fmaf(dsr1, acc[3], res[0][3]);
          }
          if constexpr (kOnes) {
            // the sub-block's activation sums of columns 2t, 2t+1 (the same in every row of the tile), then the folded offsets
            const uint32_t ones[4] = {MT::kOnePair, MT::kOnePair, MT::kOnePair, MT::kOnePair};
            float sx[4];
            MT::mma_c(sx, ones, xb.x, xb.y, zero4);
            MT::mma(sx, ones, xb.z, xb.w);
            const float kk0 = sK[cw][g][2 * G + h], kk1 = sK[cw][g + 8][2 * G + h];
            res[0][0] = fmaf(-kk0, sx[0], res[0][0]);
            res[0][2] = fmaf(-kk1, sx[0], res[0][2]);
            if (MC == 2) {
              res[0][1] = fmaf(-kk0, sx[1], res[0][1]);
              res[0][3] = fmaf(-kk1, sx[1], res[0][3]);
            }
          }
        }
      }
     }
    }
    __syncwarp();                              // every lane is done with the stage (and with sS)
    if (lane == 0) mbar_arrive(empty(slot));
    chunk -= NG;
    while (chunk < 0) { chunk += nchunks; ++tl; }
  }
  // the tiles this warp has not flushed yet (all of them contribute to every tile's reduction, zeros included)
  while (cur_tile < ntiles && ok) { flush(cur_tile); ++cur_tile; }
  }
}

// ---------------------------------------------------------------------------------------- host side
using Scratch = StreamScratch;
int stream_scratch(cudaStream_t stream, bool slices, Scratch* out);             // gemv_stream.cu: one set per (device, stream)
int sm_count();                                                 // of the current device

// Dynamic shared memory a launch may take beside its static arrays (scales of every consumer warp): one or two CTAs per SM.
template <int QT, int MXC, int NG> constexpr size_t smem_limit(int ctas_per_sm) {
  const size_t fixed = size_t(NG * kGroupWarps) * kRows * (planes::sub16<QT>() ? planes::kScalePitch : 8) * sizeof(float) *
                           (MXC <= 2 || QT == QTYPE_Q6_K || QT == QTYPE_Q3_K ? 1 : 2) + 2048;
  return (ctas_per_sm == 2 ? size_t(227) * 1024 / 2 : size_t(227) * 1024) - fixed;
}
template <int QT, int MXC, int NG, int D, bool RAG = false> bool fits(int chunks, int ctas_per_sm) {      // chunks: of a slice
  return smem_fixed_bytes<QT, MXC, NG, D, RAG>() + smem_planes_bytes<QT, MXC>(chunks) <= smem_limit<QT, MXC, NG>(ctas_per_sm);
}

template <int QT, typename T, int MXC, int NG, int D, bool PROBE = false, bool RAG = false>
static int launch_cfg(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, int ctas_per_sm, const PeerOut& peers,
                          cudaStream_t s, int slice_chunks = 0) {     // 0: one slice
  Line line;
  line.tiles = (n + kRows - 1) / kRows;
  line.nchunks = ((k + 255) / 256 + kKC - 1) / kKC;
  line.len = slice_chunks > 0 ? min(slice_chunks, line.nchunks) : line.nchunks;
  line.slices = (line.nchunks + line.len - 1) / line.len;
  if (int64_t(line.tiles) * line.nchunks > 0x3fffffff) return RC_RANGE;
  if (!fits<QT, MXC, NG, D, RAG>(line.len, 1)) return RC_RANGE;
  const size_t smem = smem_fixed_bytes<QT, MXC, NG, D, RAG>() + smem_planes_bytes<QT, MXC>(line.len);
  int* status = stream_status_ptr();
  if (status == nullptr) return RC_LAUNCH;
  auto kern = gemv_stream_kernel<QT, T, MXC, NG, D, PROBE, RAG>;
  static SmemOptIn granted;
  if (!smem_opt_in(kern, smem, granted)) return RC_LAUNCH;
  // a CTA owns at least as many units as a tile of the line has, so that a tile is cut between two CTAs at most
  const int ctas = min(min(line.units() / line.len, sm_count() * (ctas_per_sm < 1 ? 1 : ctas_per_sm)), kStreamMaxCtas);
  Scratch sc;
  if (int rc = stream_scratch(s, line.slices > 1, &sc)) return rc;
  CUtensorMap w_map = {};
  if constexpr (tiled_copy<QT, RAG>()) {
    EncodeTiledFn enc = encode_tiled();
    if (enc == nullptr) return RC_LAUNCH;
    const cuuint64_t row_bytes = cuuint64_t(k / 256) * Geom<QT>::kSbBytes;
    const cuuint64_t dims[2] = {row_bytes / 8, cuuint64_t(n)}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {cuuint32_t(stage_pitch<QT, RAG>() / 8), cuuint32_t(kRows)}, estr[2] = {1, 1};
    if (enc(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void*>(b), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return RC_LAUNCH;
  }
  const cudaError_t err = gemv_launch(kern, ctas, 1, (NG * kGroupWarps + 2) * 32, smem, s, static_cast<const T*>(a),
                                      static_cast<const uint8_t*>(b), static_cast<const T*>(bias), static_cast<T*>(c), m, n, k, status,
                                      sc.partial, sc.slice_words, line, peers, w_map);
  return err == cudaSuccess ? RC_OK : RC_LAUNCH;
}

// Ring depths of the integer path, by the size of a stage (16 rows x 8 super-blocks): 13.3 - 19 KB, 23 / 26 KB, 35 KB.
template <int QT> constexpr int int_depth() { return QT == QTYPE_Q8_0 ? 2 : (QT == QTYPE_Q6_K || QT == QTYPE_Q5_K) ? 3 : 4; }

// The integer path for M = MXC rows, 8 consumer warps per CTA, two CTAs per SM.
//   One slice where the digit planes of all of K (4 K bytes per row and CTA) fit beside a ring of two stages and there is a row tile
//   for every SM ([1024 x 14336] Q4_K, M = 2: 7.9 us in slices, 12.8 us on the tile kernel).  Else K is cut into up
//   to four slices of at least two chunks (4096 weights): a CTA then makes the planes of its slice only and uses them for several
//   tiles; the slices of a tile meet through global memory.  Q4_K [8192 x 28672], M = 1: 33.0 us in four slices, 43.0 us with one
//   CTA per SM and all planes, 38.9 us with 16-bit operands.
template <int QT, typename T, int MXC, bool RAG>
static int launch_int(const void* a, const void* b, const void* bias, void* c, int n, int k, const PeerOut& peers, cudaStream_t s) {
  constexpr int D = int_depth<QT>();
  const int nchunks = ((k + 255) / 256 + kKC - 1) / kKC, tiles = (n + kRows - 1) / kRows;
  int len = nchunks;
  if (nchunks >= 4 && (tiles <= sm_count() || !fits<QT, MXC, 1, 2, RAG>(nchunks, 2))) {
    const int slices = min(kMaxSlices, nchunks / 2);
    len = (nchunks + slices - 1) / slices;
    if (size_t(tiles) * ((nchunks + len - 1) / len) * (kRows * MXC * sizeof(uint64_t)) > kStreamSliceBytes) len = nchunks;
  }
  if (fits<QT, MXC, 1, D, RAG>(len, 2)) return launch_cfg<QT, T, MXC, 1, D, false, RAG>(a, b, bias, c, MXC, n, k, 2, peers, s, len);
  if constexpr (D > 3)
    if (fits<QT, MXC, 1, 3, RAG>(len, 2)) return launch_cfg<QT, T, MXC, 1, 3, false, RAG>(a, b, bias, c, MXC, n, k, 2, peers, s, len);
  if constexpr (D > 2)
    if (fits<QT, MXC, 1, 2, RAG>(len, 2)) return launch_cfg<QT, T, MXC, 1, 2, false, RAG>(a, b, bias, c, MXC, n, k, 2, peers, s, len);
  return launch_cfg<QT, T, MXC, 1, D, false, RAG>(a, b, bias, c, MXC, n, k, 1, peers, s, len);
}

}  // namespace stream
}  // namespace b200gguf
