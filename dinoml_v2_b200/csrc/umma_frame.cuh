// The frame that the tcgen05 GEMMs share (umma_gemm.cuh, umma_split.cuh): weights as the UMMA A operand from tensor memory, activations by
// TMA, accumulators in tensor memory, stream-K or K slices in a cluster, bounded waits.
//
// Swap-AB: the weight tile is the UMMA "A" operand (128 rows per CTA = UMMA M), the activation tile is "B" (bn rows = UMMA N, 16..256), so
// D[n, m] lives in TMEM as 128 lanes x bn fp32 columns and one CTA reuses every dequantized weight tile across bn activation rows.  The
// weight operand is fed from TENSOR MEMORY (tcgen05.mma with A in TMEM): a 128 x 64 tile of 16-bit values is 128 lanes x 32 columns, a
// ring of such slots sits behind the accumulator columns, so the dequantized weights never touch shared memory.  Roles of a CTA:
//   * PW producer warps unpack (the kernels' own part) and run the epilogue;
//   * warp PW: TMA (SWIZZLE_128B, no multicast) of the activation tiles; rows past M are zero-filled by the tensor map;
//   * warp PW + 1: MMA issue;
//   * warp PW + 2: TMA of the packed weight bytes into a ring of their own.
// A hand-over unit is HS K stages of 64 weights (the slots in TMEM paired with activation tiles in shared memory): one full / empty
// barrier pair, one wait and one commit per unit, because barrier handling on the issuing warp takes about 300 cycles whatever it hands over.
//
// Three sizes of it:
//   * PW = 8, two CTAs per SM (half of the registers, shared memory and tensor memory each), up to 128 activation rows: the producers are
//     the bound there, and while one CTA waits for its barriers, its copies or its epilogue the other one unpacks; the next launch's
//     CTAs start beside the last ones of this launch;
//   * PW = 16, one CTA per SM: tiles whose rings do not fit into half an SM;
//   * PW = 16 in pairs (cta_group::2), from 129 activation rows on: the two CTAs unpack 128 weight rows each and hold half of the activation
//     tile each, which halves the bytes an SM fetches per MMA and makes room for a stage ring of two super-blocks.
//
// Every mbarrier wait is bounded: after kSpinLimit polls the waiter records a code in a device status
// word, raises a CTA-wide abort flag and every role falls through to the common teardown (outstanding
// TMA copies are waited for, TMEM is freed).  Nothing traps or spins forever.
#pragma once
#include <type_traits>

#include "gemv_mma_common.cuh"
#include "scratch_sets.h"
#include "tensor_map.cuh"

namespace b200gguf {

int check_gemm_args(const void* a, const void* b, const void* c, int qtype, int dtype, int m, int n, int k);

namespace umma {

constexpr int kRowsW = 128;            // weight rows per CTA (UMMA M)
constexpr int kBK = 64;                // K per pipeline stage (one 128-byte swizzle atom of 16-bit values)
constexpr int kStagesPerSb = 4;         // 256 weights / kBK
constexpr int kWSlotCols = kBK / 2;     // 64 16-bit values per lane = 32 columns
constexpr int kSmemBudget = 227 * 1024, kSmemHalf = 113 * 1024;      // of a CTA alone on its SM, of two
constexpr uint32_t kSpinLimit = 1u << 24;   // try_wait polls before a wait gives up (a launch may stand behind a long one)

enum : int { ST_OK = 0, ST_EMPTY_TIMEOUT = 1, ST_FULL_TIMEOUT = 2, ST_ACC_TIMEOUT = 3, ST_PEER_TIMEOUT = 4 };
constexpr uint32_t kFlagSpinLimit = 1u << 23;   // polls (100 ns apart) of another CTA's partial-tile flag

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (after flagging) if the phase never completes or the CTA is aborting.
// The non-blocking test comes first: on the MMA-issuing warp most waits find their phase already complete, and
// there test_wait measured ~90 cycles less than a try_wait that succeeds at once.
// There is no sleep back-off: try_wait itself suspends the thread for a hardware-defined slice.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (mbar_test_wait(bar, parity)) return true;
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicCAS(status, 0, code);
  return false;
}
// A shared-memory address of this CTA as that of the same place in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_address(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
__device__ __forceinline__ void ld_cluster4(uint32_t address, float (&v)[4]) {
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(address) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t address) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(address) : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}\n" : "=r"(pred));
  return pred != 0;
}
// Bounded wait with no flagging, for teardown paths.
__device__ __forceinline__ void mbar_wait_plain(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return;
    if (i > 64) __nanosleep(40);
  }
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Tensor memory and MMAs of one CTA, or of a pair of CTAs whose even one issues.  `to`: CTAs of the pair whose barrier is arrived at.
template <bool PAIR> __device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t columns) {
  if (PAIR) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
}
template <bool PAIR> __device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t columns) {
  if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(columns) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(columns) : "memory");
}
template <bool PAIR> __device__ __forceinline__ void umma_commit(uint32_t bar, uint16_t to) {
  if (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar), "h"(to) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// Activation tile; in a pair the bytes may count on the even CTA's barrier.
template <bool PAIR> __device__ __forceinline__ void tma_load_x(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if (PAIR)
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(dst), "l"(map),
                 "r"(bar), "r"(c0), "r"(c1) : "memory");
  else
    tma_load_2d(dst, map, bar, c0, c1);
}
// K-major, SWIZZLE_128B shared-memory matrix descriptor: rows of 128 B, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  return uint64_t((addr & 0x3ffffu) >> 4) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(2) << 61);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
               "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// A operand from tensor memory, B from shared memory.
template <bool PAIR> __device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  if (PAIR)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d), "r"(tmem_a),
                 "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d), "r"(tmem_a),
                 "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

// 16-bit pair arithmetic used to turn quants into MMA operand values.
template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  static constexpr uint32_t kMagicBytes = 0x43434343u;   // 0x43qq = 128 + q
  static constexpr float kMagic = 128.f;
  static constexpr uint32_t kFormat = 1;                  // UMMA F16F32Format::BF16
  static constexpr int kFp4MagPos = 6;                    // FP4 codes: exponent / mantissa bits land on bits 6..8
  static constexpr float kFp4Up = 0x1p120f, kFp4Rest = 0x1p6f;   // bits = e2m1 * 2^-126; * kFp4Up is a normal number
  static constexpr CUtensorMapDataType kTmaType = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  using V = __nv_bfloat162;
  static __device__ __forceinline__ V splat(float f) { return __float2bfloat162_rn(f); }
  static __device__ __forceinline__ V pack(float lo, float hi) { return __floats2bfloat162_rn(lo, hi); }
  static __device__ __forceinline__ __nv_bfloat16 cvt(float f) { return __float2bfloat16_rn(f); }
  static __device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
};
template <> struct Pair<__half> {
  static constexpr uint32_t kMagicBytes = 0x64646464u;   // 0x64qq = 1024 + q
  static constexpr float kMagic = 1024.f;
  static constexpr uint32_t kFormat = 0;                  // UMMA F16F32Format::F16
  static constexpr int kFp4MagPos = 9;                    // bits 9..11
  static constexpr float kFp4Up = 0x1p14f, kFp4Rest = 1.f;       // bits = e2m1 * 2^-14
  static constexpr CUtensorMapDataType kTmaType = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  using V = __half2;
  static __device__ __forceinline__ V splat(float f) { return __float2half2_rn(f); }
  static __device__ __forceinline__ V pack(float lo, float hi) { return __floats2half2_rn(lo, hi); }
  static __device__ __forceinline__ __half cvt(float f) { return __float2half_rn(f); }
  static __device__ __forceinline__ float up(__half v) { return __half2float(v); }
};
template <typename V> __device__ __forceinline__ V as_pair(uint32_t r) { return *reinterpret_cast<V*>(&r); }
template <typename V> __device__ __forceinline__ uint32_t as_u32(V v) { return *reinterpret_cast<uint32_t*>(&v); }
struct Params {
  const void* bias;       // [n] or null
  void* out;              // [m, n] in the activation dtype
  float* partial;         // one fp32 tile [bn][128] per CTA (stream-K partial sums)
  int* flags;             // one word per CTA: 1 = that CTA's partial tile is complete in `partial`
  int* status;            // device status word
  int m, n, k;
  int m_tiles;            // activation tiles per weight panel
  int bn;                 // activation rows of a tile: a multiple of 16 (pairs: 32), at most BM (the UMMA N of this launch)
  int slices;             // > 1: K of every tile is cut across a cluster of so many CTAs
  int shared;             // two teams of producers: 1 = both work on every super-block, 0 = on every other one each
  long long units;        // output tiles x super-blocks
  PeerOut peers;          // extra destinations of the output (SCATTER kernels only)
};

// Stream-K work split.  The work of the launch is a line of units (tile t, super-block sb), tile-major; worker c of G (a CTA, or a pair)
// owns the contiguous range [start(c), start(c+1)), so every SM gets the same amount of tensor-core work whatever the tile
// count.  A worker walks its range from the HIGHEST tile down; the segment that holds the end of a tile is therefore the
// last thing it does, and the other pieces of that tile belong to lower-numbered workers that computed them first.
// Those store an fp32 partial tile and raise a flag; the one with the end of the tile adds the partials in
// order to its own accumulator, applies bias and stores (deterministic summation order).  Dependencies only point to
// lower-numbered CTAs, which are dispatched first, and every flag wait is bounded.
__device__ __forceinline__ long long unit_start(int c, long long units, int workers) { return (static_cast<long long>(c) * units) / workers; }
__device__ __forceinline__ int unit_owner(long long u, long long units, int workers) { return int(((u + 1) * workers - 1) / units); }

struct Walk {
  long long u0, u1;
  int nsb;
  __device__ __forceinline__ int tile_hi() const { return int((u1 - 1) / nsb); }
  __device__ __forceinline__ int tile_lo() const { return int(u0 / nsb); }
  __device__ __forceinline__ void segment(int t, int& sb_b, int& sb_e) const {
    const long long base = static_cast<long long>(t) * nsb;
    sb_b = int((u0 > base ? u0 : base) - base);
    sb_e = int((u1 < base + nsb ? u1 : base + nsb) - base);
  }
};

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) { asm volatile("st.release.gpu.global.s32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory"); }

// Launch of `workers` CTAs, clusters of `slices` CTAs (along y) or pairs (along x), with programmatic stream serialization.
template <class S, typename Kernel, typename... Args>
inline cudaError_t launch_frame(Kernel kern, int workers, int slices, cudaStream_t s, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S::PAIR ? 2 * workers : workers, slices);
  cfg.blockDim = dim3(S::kThreads);
  cfg.dynamicSmemBytes = S::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = S::PAIR ? 2 : 1;
  attr[1].val.clusterDim.y = unsigned(slices);
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = S::PAIR || slices > 1 ? 2 : 1;
  if ((S::PAIR ? 2 : 1) * slices > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return cudaErrorInvalidConfiguration;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// A CTA of the frame.
//   T: activation type; BM: most activation rows of a tile; PW: producer warps, 16 (one CTA per SM) or 8 (two);
//   PAIR: two CTAs (256 weight rows) work as one, the even one issues their MMAs;
//   TERMS: 16-bit numbers per weight; HS: K stages of a hand-over unit; NB: units in the stage ring;
//   NRAW, RAW_BYTES: ring of packed bytes; RAW_ARRIVE: producer warps that read one of its slots; FILL: producer warps that fill a unit.
template <typename T_, int BM_, int PW_, bool PAIR_, int TERMS_, int HS_, int NB_, int NRAW_, int RAW_BYTES_, int RAW_ARRIVE_, int FILL_, bool SLICED_ = true>
struct Shape {
  using T = T_;
  static constexpr int BM = BM_, PW = PW_, TERMS = TERMS_, HS = HS_, NB = NB_, NRAW = NRAW_, RAW_BYTES = RAW_BYTES_, RAW_ARRIVE = RAW_ARRIVE_, FILL = FILL_;
  static constexpr bool PAIR = PAIR_, SLICED = SLICED_;           // SLICED: K of a tile may be cut across a cluster
  static constexpr int NS = NB * HS;                             // stages in the ring
  static constexpr int kJobs = 16 / PW, kTeams = PW / 8;         // CTAs per SM; teams of eight producer warps
  static constexpr int kUnits = kStagesPerSb / HS;               // hand-over units per super-block
  static constexpr int kXTile = (PAIR ? BM / 2 : BM) * kBK * 2;  // this CTA's activation bytes of a stage
  static constexpr int kThreads = PW * 32 + 96, kCtasPerSm = kJobs;
  static constexpr uint32_t kTmemCols = 512 / kJobs;
  static constexpr int kBars = 2 * NB + 2 * NRAW + 4;
  static constexpr int kRings = NS * kXTile + NRAW * RAW_BYTES;   // bytes of both rings
  static constexpr size_t kSmem = 1024 + size_t(NS) * kXTile + size_t(NRAW) * RAW_BYTES + kBars * 8 + 16;
  static_assert(NRAW >= 2 && NB >= 2 && BM + NS * TERMS * kWSlotCols <= int(kTmemCols), "rings");
  static_assert(kSmem <= size_t(kJobs == 2 ? kSmemHalf : kSmemBudget), "shared memory");
  static_assert(!SLICED || BM * kRowsW * 4 <= kRings, "the sums of a slice go where activations and packed bytes were");
};

template <class S> struct Cta {
  using T = typename S::T;
  const Params& p;
  uint8_t *xtiles, *raw;
  uint32_t bar0, tmem_base;
  volatile int* abort_flag;
  int tid, warp, lane, rank, lead, worker, workers, nsb, tile_hi, tile_lo;
  Walk walk;
  bool has_work, dep_waited = false;
  uint32_t epi_phase = 0;

  // Barriers: full[NB], empty[NB], rawfull[NRAW], rawfree[NRAW], accumulator full, accumulator free, drain, epilogue.  A unit is "full"
  // when its producer warps (FILL, 8 if teams share) have written the weight tiles AND the activation tiles' bytes have landed (one barrier, one
  // wait for the MMA warp); it is "empty" when the MMAs that read it have completed (one tcgen05.commit, watched by
  // producers and TMA).  In a pair the even CTA's `full` and `accumulator free` count both CTAs.
  __device__ __forceinline__ uint32_t full(int u) const { return bar0 + 8u * u; }
  __device__ __forceinline__ uint32_t empty(int u) const { return bar0 + 8u * (S::NB + u); }
  __device__ __forceinline__ uint32_t rawfull(int s) const { return bar0 + 8u * (2 * S::NB + s); }
  __device__ __forceinline__ uint32_t rawfree(int s) const { return bar0 + 8u * (2 * S::NB + S::NRAW + s); }
  __device__ __forceinline__ uint32_t accbar() const { return bar0 + 8u * (2 * S::NB + 2 * S::NRAW); }
  __device__ __forceinline__ uint32_t accfree() const { return accbar() + 8u; }
  __device__ __forceinline__ uint32_t drainbar() const { return accbar() + 16u; }
  __device__ __forceinline__ uint32_t epibar() const { return accbar() + 24u; }

  __device__ __forceinline__ Cta(const Params& params, uint8_t* smem_raw) : p(params) {
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    xtiles = smem;                                              // NS x [activation rows][128 B]
    raw = xtiles + S::NS * S::kXTile;                           // NRAW x packed bytes
    uint64_t* bars = reinterpret_cast<uint64_t*>(raw + S::NRAW * S::RAW_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + S::kBars);
    abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    bar0 = smem_u32(bars);
    tid = threadIdx.x; warp = tid >> 5; lane = tid & 31;
    rank = S::PAIR ? int(blockIdx.x & 1u) : 0;
    lead = S::PAIR ? 2 * int(blockIdx.y) : 0;                   // cluster rank of the CTA that issues this pair's MMAs
    worker = S::PAIR ? int(blockIdx.x >> 1) : int(blockIdx.x);
    workers = S::PAIR ? int(gridDim.x >> 1) : int(gridDim.x);
    nsb = (p.k + 255) >> 8;
    walk.nsb = nsb;
    if (S::SLICED && p.slices > 1) {                            // one tile, one slice of its K
      const long long base = static_cast<long long>(worker) * nsb;
      walk.u0 = base + int(blockIdx.y) * nsb / p.slices;
      walk.u1 = base + (int(blockIdx.y) + 1) * nsb / p.slices;
    } else {
      walk.u0 = unit_start(worker, p.units, workers);
      walk.u1 = unit_start(worker + 1, p.units, workers);
    }
    has_work = walk.u1 > walk.u0;
    tile_hi = has_work ? walk.tile_hi() : -1;
    tile_lo = has_work ? walk.tile_lo() : 0;
    if (tid == 0) {
      for (int s = 0; s < S::NB; ++s) {
        mbar_init(full(s), (S::PAIR ? 2 : 1) * (p.shared ? 8 : S::FILL) + 1);             // the producer warps that fill it + the TMA lane's arrive.expect_tx
        mbar_init(empty(s), 1);
      }
      for (int s = 0; s < S::NRAW; ++s) {
        mbar_init(rawfull(s), 1);
        mbar_init(rawfree(s), p.shared ? S::PW : S::RAW_ARRIVE);
      }
      mbar_init(accbar(), 1);
      mbar_init(accfree(), S::PAIR ? 2 * S::PW : S::PW);
      mbar_init(drainbar(), 1);
      mbar_init(epibar(), S::PW);
      *abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncwarp();
    if (warp == S::PW + 1) tmem_alloc<S::PAIR>(smem_u32(tmem_slot), S::kTmemCols);
    tcgen05_fence_before();
    if constexpr (S::PAIR) cluster_barrier(); else __syncthreads();
    tcgen05_fence_after();
    tmem_base = *tmem_slot;
    // Programmatic dependent launch.  The next kernel in the stream may begin once every CTA of this grid is past this
    // point; its CTAs take over an SM as soon as one of ours exits (or stand beside ours: PW = 8).  In the other direction, the packed
    // weights are constants: the weight TMA, the unpack and the tcgen05.st of this grid run ahead of `griddepcontrol.wait`, which only
    // the activation TMA warp (before its first load) and the producers (before their first epilogue: outputs, partial
    // tiles and flags are shared with the preceding launch) execute.
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  }

  __device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, int code) const {      // by a converged warp, one answer for all lanes
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.status, code) ? 1 : 0) != 0;
  }
  __device__ __forceinline__ void arrive_lead(uint32_t bar) const {      // on the barrier of the CTA that issues the MMAs
    if constexpr (S::PAIR) mbar_arrive_cluster(cluster_address(bar, uint32_t(lead))); else mbar_arrive(bar);
  }
  // Barrier over the producer warps on an mbarrier, so that it is bounded like every other wait (a plain bar.sync
  // would hang the warps that reached it if another warp had given up).
  __device__ __forceinline__ bool producer_sync() {
    __syncwarp();
    int ok = 1;
    if (lane == 0) {
      mbar_arrive(epibar());
      ok = mbar_wait(epibar(), epi_phase & 1u, abort_flag, p.status, ST_ACC_TIMEOUT) ? 1 : 0;
    }
    ++epi_phase;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
  }
  __device__ __forceinline__ void wait_dependency() {
    if (!dep_waited) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    dep_waited = true;
  }
  // Position in a ring.  A warp waits for every lap of the slots it uses (a parity says nothing about the lap before), so the warps of a
  // half of the super-block share no slot with the others: NB is a multiple of 2 where there are two groups of eight.
  struct Ring {
    int at;
    uint32_t phase;                   // of the `full` barrier; `empty` is waited for at the other one (true at once on the first lap)
    __device__ __forceinline__ void step(int by, int depth) { at += by; if (at >= depth) { at -= depth; phase ^= 1u; } }
  };

  // ------------------------------------------------------------------ activation TMA
  // The three control warps stay converged: every lane runs the loop and polls the barriers, one elected lane issues
  // the asynchronous instructions.  Inside a divergent `if (lane == 0)` region the compiler cannot keep descriptors,
  // coordinates and barrier addresses in uniform registers, and each tcgen05.mma / bulk copy then costs tens of cycles
  // of register shuffling on the one thread the whole pipeline waits for.  (One warp for both kinds of loads would leave the producers more
  // registers, and was slower: [28672 x 8192] Q4_K, M = 16, 39.3 -> 41.2 us, one CTA per SM 43.2 -> 51.1.)
  __device__ __forceinline__ void load_activations(const CUtensorMap* x_map) const {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");     // the activations may be the preceding kernel's output
    Ring u{0, 0u};
    const uint32_t bytes = uint32_t(p.bn) * (kBK * 2) * S::HS, x0 = smem_u32(xtiles);
    bool ok = true;
    for (int t = tile_hi; t >= tile_lo && ok; --t) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const int m0 = (t % p.m_tiles) * p.bn + (S::PAIR ? rank * (tile_rows(t) >> 1) : 0);
      for (int st = sb_b * kStagesPerSb; st < sb_e * kStagesPerSb && ok; st += S::HS) {
        if (!wait(empty(u.at), u.phase ^ 1u, ST_EMPTY_TIMEOUT)) { ok = false; break; }
        if (elect_one()) {
          if (!S::PAIR || rank == 0) mbar_arrive_expect_tx(full(u.at), bytes);      // both CTAs' bytes
          const uint32_t bar = S::PAIR ? cluster_address(full(u.at), uint32_t(lead)) : full(u.at);
#pragma unroll
          for (int i = 0; i < S::HS; ++i)
            tma_load_x<S::PAIR>(x0 + uint32_t((u.at * S::HS + i) * S::kXTile), x_map, bar, (st + i) * kBK, m0);
        }
        __syncwarp();
        u.step(1, S::NB);
      }
    }
    // Aborting: activation copies may still be writing shared memory, and their barrier also counts producer
    // arrivals that will never come, so it cannot be waited on.  A copy of this size lands within microseconds; give
    // the last ones a millisecond before the CTA may exit.
    if (*abort_flag)
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }

  // ------------------------------------------------------------------ MMA issue
  __device__ __forceinline__ void issue_mmas() const {
    if (S::PAIR && rank != 0) return;
    constexpr uint32_t kFormat = Pair<T>::kFormat;
    const uint32_t idesc0 = (1u << 4) | (kFormat << 7) | (kFormat << 10) | (uint32_t((S::PAIR ? 2 : 1) * kRowsW >> 4) << 24);
    const uint64_t db0 = smem_desc_sw128(smem_u32(xtiles));
    const uint16_t both = uint16_t(3u << lead);                  // the CTAs of the pair
    Ring u{0, 0u};
    int segi = 0;
    bool ok = true;
    for (int t = tile_hi; t >= tile_lo && ok; --t, ++segi) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      if (segi > 0) {                        // the previous segment's accumulator has been read out
        ok = wait(accfree(), uint32_t(segi - 1) & 1u, ST_ACC_TIMEOUT);
        if (!ok) break;
        tcgen05_fence_after();
      }
      uint32_t accumulate = 0;
      const uint32_t idesc = idesc0 | (uint32_t(tile_rows(t) >> 3) << 17);
      auto unit = [&](int at) -> bool {                           // one wait, 4 HS TERMS MMAs, one commit per unit
        if (!wait(full(at), u.phase, ST_FULL_TIMEOUT)) return false;
        tcgen05_fence_after();
        if (elect_one()) {
          const uint32_t a0 = tmem_base + uint32_t(S::BM + at * (S::HS * S::TERMS * kWSlotCols));
          const uint64_t d0 = db0 + uint64_t(uint32_t(at * (S::HS * S::kXTile)) >> 4);
#pragma unroll
          for (int i = 0; i < S::HS; ++i)
#pragma unroll
            for (int tm = 0; tm < S::TERMS; ++tm)
#pragma unroll
              for (int kk = 0; kk < kBK / 16; ++kk) {     // 16 K values = 8 TMEM columns of A, 32 bytes of each B row
                umma_f16_ts<S::PAIR>(tmem_base, a0 + uint32_t((i * S::TERMS + tm) * kWSlotCols + 8 * kk), d0 + uint64_t((i * S::kXTile) >> 4) + uint64_t(2 * kk),
                                     idesc, accumulate);
                accumulate = 1;
              }
          umma_commit<S::PAIR>(empty(at), both);
        }
        accumulate = 1;
        __syncwarp();
        return true;
      };
      if constexpr (S::NB == S::kUnits) {                         // a ring of one super-block: every address is a constant
        for (int sb = sb_b; sb < sb_e && ok; ++sb) {
#pragma unroll
          for (int i = 0; i < S::kUnits; ++i)
            if (ok) ok = unit(i);
          u.phase ^= 1u;
        }
      } else {
        for (int h = (sb_e - sb_b) * S::kUnits; h > 0 && ok; --h) {
          ok = unit(u.at);
          u.step(1, S::NB);
        }
      }
      if (ok && elect_one()) umma_commit<S::PAIR>(accbar(), both);
      __syncwarp();
    }
    if (!ok && has_work && elect_one()) {   // aborting: let every MMA already issued finish before TMEM is freed
      umma_commit<S::PAIR>(drainbar(), uint16_t(1u << lead));
      mbar_wait_plain(drainbar(), 0);
    }
    __syncwarp();
  }

  // ------------------------------------------------------------------ packed weights
  // load(slot address, barrier, super-block, weight row): called by the converged warp once the slot is free.
  template <typename Load>
  __device__ __forceinline__ void load_weights(Load load) const {
    Ring r{0, 0u};
    int issued = 0;
    bool ok = true;
    for (int t = tile_hi; t >= tile_lo && ok; --t) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const int n0 = row0(t);
      for (int sb = sb_b; sb < sb_e && ok; ++sb) {
        if (!wait(rawfree(r.at), r.phase ^ 1u, ST_EMPTY_TIMEOUT)) { ok = false; break; }
        load(smem_u32(raw) + uint32_t(r.at * S::RAW_BYTES), rawfull(r.at), sb, n0);
        __syncwarp();
        ++issued;
        r.step(1, S::NRAW);
      }
    }
    if (*abort_flag) {
      for (int i = max(0, issued - S::NRAW); i < issued; ++i) mbar_wait_plain(rawfull(i % S::NRAW), uint32_t(i / S::NRAW) & 1u);
    }
  }
  // Activation rows of tile t that the MMAs multiply: the last tile of a panel has fewer where its rows end before it does (M = 333: 192 and 160 rows).
  __device__ __forceinline__ int tile_rows(int t) const {
    if (!S::PAIR) return p.bn;
    return min(p.bn, (p.m - (t % p.m_tiles) * p.bn + 31) & ~31);
  }
  __device__ __forceinline__ int row0(int t) const { return ((t / p.m_tiles) * (S::PAIR ? 2 : 1) + rank) * kRowsW; }      // of this CTA's part of tile t

  // ------------------------------------------------------------------ epilogue
  // Of one segment (tile t, super-blocks [sb_b, sb_e), the segi-th of this CTA), by the producer warps.  false = a wait gave up.  GATED:
  // p.peers.act may ask for a gated output; SCATTER: p.peers may name further destinations.  seen(v): called with every finished sum.
  template <bool GATED, bool SCATTER, typename Seen>
  __device__ __forceinline__ bool epilogue(int t, int sb_b, int sb_e, int segi, Seen seen_sum) {
    using P = Pair<T>;
    wait_dependency();
    {
      int ok = 1;
      if (lane == 0) ok = mbar_wait(accbar(), uint32_t(segi) & 1u, abort_flag, p.status, ST_ACC_TIMEOUT) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) return false;
    }
    tcgen05_fence_after();
    constexpr int kWide = S::PAIR ? 2 : 1, kGroups = S::PW / 4;
    const int row = 32 * (warp & 3) + lane;
    const int n_row = row0(t) + row, m0 = (t % p.m_tiles) * p.bn;
    const bool whole = sb_b == 0 && sb_e == nsb;
    const bool finishes = sb_e == nsb;            // this CTA stores the tile (after adding the others' partial sums)
    int peer0 = worker;                           // first worker with a piece of this tile; peers are peer0 .. worker-1
    if (finishes && !whole) {
      peer0 = unit_owner(static_cast<long long>(t) * nsb, p.units, workers);
      for (int peer = peer0 + tid; peer < worker; peer += S::PW * 32) {      // one tile of a very long K has more pieces than eight warps have threads
        bool seen = false;
        for (uint32_t i = 0; i < kFlagSpinLimit && !seen; ++i) {
          seen = ld_acquire(p.flags + peer * kWide + rank) != 0;
          if (!seen) __nanosleep(100);
        }
        if (!seen) { *abort_flag = 1; atomicCAS(p.status, 0, ST_PEER_TIMEOUT); }
      }
      if (!producer_sync()) return false;
    }
    const float bias_v = (finishes && p.bias != nullptr && n_row < p.n) ? P::up(static_cast<const T*>(p.bias)[n_row]) : 0.f;
    const size_t tile_floats = size_t(p.bn) * kRowsW;
    // The warps that share a lane quarter split the tile's bn columns: evenly where that is at most 16 each, above that in
    // rounds of 16 taken in turn (32 per round, or uneven splits, spill registers that the unpack loop needs).
    constexpr int CH = 16, kRound = kGroups * CH;
    const int per = min(CH, p.bn / kGroups);
    for (int col = (warp >> 2) * per; col < p.bn; col += kRound) {
      uint32_t r[CH];
      tmem_ld16(tmem_base + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(col), r);
      tmem_ld_wait();
      if (!finishes) {
        float* dst = p.partial + size_t(worker * kWide + rank) * tile_floats + size_t(col) * kRowsW + row;     // tile-local [bn][128]
#pragma unroll
        for (int j = 0; j < CH; ++j)
          if (j < per) dst[j * kRowsW] = __uint_as_float(r[j]);
      } else {
        for (int peer = peer0; peer < worker; ++peer) {
          const float* src = p.partial + size_t(peer * kWide + rank) * tile_floats + size_t(col) * kRowsW + row;
          float v[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) v[j] = j < per ? __ldcg(src + j * kRowsW) : 0.f;
#pragma unroll
          for (int j = 0; j < CH; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + v[j]);
        }
        if (GATED && p.peers.act != ACT_NONE) {
          // gated pair: within every 16 weight rows the first 8 belong to the first matrix, the next 8 to the second;
          // lane l and lane l ^ 8 hold the two halves, the output has n / 2 columns
          // Of every two columns the gate lane finishes the even one and its partner the odd one: one exchange and one
          // activation per lane and pair (the activations were a third of an M = 512 launch with half of the lanes idle).
          const int out_row = ((n_row >> 4) << 3) + (n_row & 7);
          const int64_t n_out = p.n >> 1;
          const int odd = (lane >> 3) & 1;
          auto gated_columns = [&](auto act) {
#pragma unroll
            for (int j = 0; j < CH; j += 2) {
              const float even_v = __uint_as_float(r[j]) + bias_v, odd_v = __uint_as_float(r[j + 1]) + bias_v;   // bias interleaved like the rows (0 without one)
              const float got = __shfl_xor_sync(0xffffffffu, odd ? even_v : odd_v, 8);
              const float gate = odd ? got : even_v, up = odd ? odd_v : got;
              const int mcol = m0 + col + j + odd;
              if (n_row < p.n && mcol < p.m && j < per) store<SCATTER>(int64_t(mcol) * n_out + out_row, P::cvt(gate_activation(gate, decltype(act)::value) * up));
            }
          };
          if (p.peers.act == ACT_SILU) gated_columns(std::integral_constant<int, ACT_SILU>{});
          else gated_columns(std::integral_constant<int, ACT_FAST_GELU>{});
        } else if (n_row < p.n) {
#pragma unroll
          for (int j = 0; j < CH; ++j)
            if (j < per) {
              seen_sum(__uint_as_float(r[j]));
              if (m0 + col + j < p.m) store<SCATTER>(int64_t(m0 + col + j) * p.n + n_row, P::cvt(__uint_as_float(r[j]) + bias_v));
            }
        }
      }
    }
    if (!finishes) {
      // every producer thread's partial sums happen before the barrier; the release below is cumulative over them
      if (!producer_sync()) return false;
      if (tid == 0) { __threadfence(); st_release(p.flags + worker * kWide + rank, 1); }
    } else if (!whole) {
      if (!producer_sync()) return false;    // every thread has read the peers' tiles
      for (int peer = peer0 + tid; peer < worker; peer += S::PW * 32) p.flags[peer * kWide + rank] = 0;   // leave the flags clear for the next launch
    }
    tcgen05_fence_before();
    __syncwarp();
    if (lane == 0) arrive_lead(accfree());           // the accumulator columns may be overwritten
    return true;
  }
  template <bool SCATTER> __device__ __forceinline__ void store(int64_t at, T v) const {
    static_cast<T*>(p.out)[at] = v;
    if (SCATTER) {
#pragma unroll
      for (int pi = 0; pi < 8; ++pi)
        if (pi < p.peers.count) static_cast<T*>(p.peers.ptr[pi])[at] = v;
    }
  }

  // Sliced tiles: every CTA of the cluster leaves its sums where its activations were, and finishes an equal share of the tile's columns
  // from all of them, in slice order.  The producer warps' part ...
  __device__ __forceinline__ bool leave_slice() {
    wait_dependency();
    int ok = 1;
    if (lane == 0) ok = mbar_wait(accbar(), 0u, abort_flag, p.status, ST_ACC_TIMEOUT) ? 1 : 0;
    if (__shfl_sync(0xffffffffu, ok, 0) == 0) return false;
    tcgen05_fence_after();
    constexpr int kGroups = S::PW / 4, CH = 16;
    const int per = min(CH, p.bn / kGroups);
    float* sums = reinterpret_cast<float*>(xtiles) + 32 * (warp & 3) + lane;      // [bn][128]
    for (int col = (warp >> 2) * per; col < p.bn; col += kGroups * CH) {
      uint32_t r[CH];
      tmem_ld16(tmem_base + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(col), r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < CH; ++j)
        if (j < per) sums[(col + j) * kRowsW] = __uint_as_float(r[j]);
    }
    return true;
  }
  // ... and that of all threads of the cluster: four rows of a column at a time, so that few trips to the other CTAs' memory follow one
  // another (a row at a time: [4096 x 4096], M = 64, 10.2 us instead of 9.2; several columns at a time spill registers; sums pushed to the CTA that
  // finishes them, by remote stores and a barrier or by st.async: [1024 x 4096], M = 16, 5.0 -> 5.8, [4096 x 4096], M = 512, 21.1 -> 22.7 and 24.7).
  template <bool GATED, bool SCATTER, typename Seen>
  __device__ __forceinline__ void join_slices(Seen seen_sum) {
    using P = Pair<T>;
    __syncwarp();
    cluster_barrier();
    if (warp < S::PW) {
      const int me = blockIdx.y, t = worker, n0 = row0(t), m0 = (t % p.m_tiles) * p.bn;
      const int c0 = me * p.bn / p.slices, c1 = min((me + 1) * p.bn / p.slices, p.m - m0);
      const uint32_t sums = smem_u32(xtiles);
      auto total = [&](int col, int row, float (&sum)[4]) {
        const uint32_t at = sums + uint32_t(col * kRowsW + row) * 4u;
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[i] = 0.f;
        for (int s0 = 0; s0 < p.slices; s0 += 4) {
          float v[4][4];
#pragma unroll
          for (int s = 0; s < 4; ++s)
            if (s0 + s < p.slices) ld_cluster4(cluster_address(at, uint32_t(S::PAIR ? 2 * (s0 + s) + rank : s0 + s)), v[s]);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            if (s0 + s < p.slices) {
#pragma unroll
              for (int i = 0; i < 4; ++i) sum[i] += v[s][i];
            }
        }
        if (p.bias != nullptr) {
          const T* bias = static_cast<const T*>(p.bias) + n0 + row;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n0 + row + i < p.n) sum[i] += P::up(bias[i]);
        }
      };
      if (GATED && p.peers.act != ACT_NONE) {
        for (int i = c0 * 16 + tid; i < c1 * 16; i += S::PW * 32) {
          const int col = i >> 4, pr = 4 * (i & 15), row = ((pr >> 3) << 4) | (pr & 7);
          if (n0 + row >= p.n) continue;
          float gate[4], up[4];
          total(col, row, gate);
          total(col, row + 8, up);
#pragma unroll
          for (int j = 0; j < 4; ++j) gate[j] = gate_activation(gate[j], p.peers.act) * up[j];
          store4<SCATTER>(int64_t(m0 + col) * (p.n >> 1) + (n0 >> 1) + pr, gate, 4);      // n is a multiple of 16
        }
      } else {
        for (int i = c0 * (kRowsW / 4) + tid; i < c1 * (kRowsW / 4); i += S::PW * 32) {
          const int col = i / (kRowsW / 4), row = 4 * (i % (kRowsW / 4));
          if (n0 + row >= p.n) continue;
          float v[4];
          total(col, row, v);
#pragma unroll
          for (int j = 0; j < 4; ++j) seen_sum(v[j]);
          store4<SCATTER>(int64_t(m0 + col) * p.n + n0 + row, v, p.n - n0 - row);
        }
      }
    }
    __syncwarp();
    cluster_barrier();                       // no CTA leaves while another one reads its sums
  }
  // Up to four consecutive results, at once where the place allows it.
  template <bool SCATTER> __device__ __forceinline__ void store4(int64_t at, const float (&v)[4], int count) const {
    using P = Pair<T>;
    T* dst = static_cast<T*>(p.out) + at;
    if (!SCATTER && count >= 4 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(as_u32<typename P::V>(P::pack(v[0], v[1])), as_u32<typename P::V>(P::pack(v[2], v[3])));
      return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < count) store<SCATTER>(at + j, P::cvt(v[j]));
  }

  // f(weight row, first activation row, how many) for the results that this thread has stored.
  template <typename F> __device__ __forceinline__ void for_stored(F f) const {
    if (warp >= S::PW) return;
    const int row = 32 * (warp & 3) + lane;
    if (S::SLICED && p.slices > 1) {
      const int me = blockIdx.y, n0 = row0(worker), m0 = (worker % p.m_tiles) * p.bn;
      const int c0 = me * p.bn / p.slices, c1 = min((me + 1) * p.bn / p.slices, p.m - m0);
      for (int i = c0 * (kRowsW / 4) + tid; i < c1 * (kRowsW / 4); i += S::PW * 32)
        for (int r = n0 + 4 * (i % (kRowsW / 4)), j = 0; j < 4 && r + j < p.n; ++j) f(r + j, m0 + i / (kRowsW / 4), 1);
      return;
    }
    constexpr int kGroups = S::PW / 4;
    const int per = min(16, p.bn / kGroups);
    for (int t = tile_hi; t >= tile_lo; --t) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const int n_row = row0(t) + row, m0 = (t % p.m_tiles) * p.bn;
      if (sb_e != nsb || n_row >= p.n) continue;
      for (int col = (warp >> 2) * per; col < min(p.bn, p.m - m0); col += kGroups * 16) f(n_row, m0 + col, min(per, p.m - m0 - col));
    }
  }

  __device__ __forceinline__ void finish() const {
    __syncwarp();
    tcgen05_fence_before();
    if constexpr (S::PAIR) cluster_barrier(); else __syncthreads();     // a pair's MMAs and commits reach into both CTAs
    if (warp == S::PW + 1) {
      tcgen05_fence_after();
      tmem_dealloc<S::PAIR>(tmem_base, S::kTmemCols);
    }
  }
};

}  // namespace umma
}  // namespace b200gguf
