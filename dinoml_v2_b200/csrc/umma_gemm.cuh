// Fused GGUF prefill GEMM ("umma" variant) on tcgen05 tensor cores with TMEM accumulators, M >= 9.
//
// C[M,N] = A[M,K] * dequant(W[N,K])^T (+ bias), float16 / bfloat16; all nine weight types (Q8_0, Q4_0, Q2_K .. Q6_K, MXFP4, NVFP4)
// (the kernel template lives in this header; umma_gemm_<type>.cu instantiates it per weight type).
// Tensor-core bound for M >= 512 (Q6_K 4096x14336: 1248 FLOP per weight byte at M = 512).
//
// The frame is umma_frame.cuh's.  Packed bytes: a 2-D byte tensor map over the weight, one box (Q8_0: two) of 128 rows x the 16-byte aligned
// window around a 256-weight super-block; no thread spends issue slots on the copy.  The producers copy their own words to registers,
// release the ring slot, then unpack with 32-bit logic + packed bf16x2/f16x2 math: thread (row = 32*(warp%4)+lane, half = (warp%8)/4)
// unpacks the 128 weights of its half of the super-block, one K stage after the other, and writes them to its TMEM lane; then
// tcgen05.wait::st + mbarrier arrive.  Sixteen warps are two teams of eight that take turns, or, where a worker has few super-blocks, share each: team
// = half, and a thread unpacks one K stage.  The warps only meet at mbarriers, never at a CTA barrier.
// The packed-weight tensor map needs weight rows that are multiples of 16 bytes: any K % 256 == 0 for the types whose 256
// weights take a multiple of 16 bytes, K % 512 == 0 for MXFP4 (136 bytes), K % 1024 == 0 for Q2_K (84), K % 2048 == 0 for
// Q6_K (210) and Q3_K (110).  Other
// shapes are served by the other variants.
//
// The reference has no counterpart kernel: its CUDA path dequantizes the whole weight to a dense
// scratch and calls an Sm80 mma.sync CUTLASS GEMM (src/dinoml/lowering/ops/gemm.py:729-749,
// kernels/cuda/src/cutlass_gemm.cu:56-89); the tile-level dequantize-then-MMA idea follows its
// prototype WMMA kernels (kernels/rocm/src/ck_gguf_q8_gemm.hip:1209-1618).
#pragma once
#include "umma_unpack.cuh"

namespace b200gguf {
namespace umma {

// Rings of a tile height: a hand-over unit is half a super-block, two stages.  kFits: whether they fit, with two CTAs on an SM (PW = 8) a ring of
// two packed super-blocks beside the stage ring that half of the tensor memory holds.  Q8_0 (272 bytes) has no room for them there.
template <int QT, int BM, int PW> struct Geo {
  static constexpr bool kPair = BM == 256;
  static constexpr int kPart = kRowsW * RawGeom<QT>::kPitch * RawGeom<QT>::kBoxes;
  static constexpr int NB = PW == 8 ? (256 - BM) / (2 * kWSlotCols) : 4;
  static constexpr int kUnit = 2 * (kPair ? BM / 2 : BM) * kBK * 2, kRest = 1024 + 512;
  static constexpr int kFit = ((PW == 8 ? kSmemHalf : kSmemBudget) - kRest - NB * kUnit) / kPart;
  static constexpr bool kFits = kFit >= 2 && !(kPair && PW == 8);
  static constexpr int kEach = PW / 8;                      // slots of a lap's turn: a slot belongs to the same team on every lap
  static constexpr int kSlots = kFit < 6 ? kFit : 6, NRAW = !kFits ? 2 : PW == 8 ? kSlots : kSlots / kEach * kEach;
  template <typename T> using Of = Shape<T, BM, PW, kPair, 1, 2, NB, NRAW, kPart, 8, 4>;
};
// Producer warps of a launch.  Up to 64 activation rows the producers are the bound, and two CTAs of eight on an SM pay ([28672 x 8192]
// Q4_K, M = 16: 39 us against 43), but for Q8_0: with one and a half super-blocks in the ring of half an SM it was 5 - 17 % slower than sixteen warps with
// four in theirs ([28672 x 4096], M = 16: 40.7 us against 35.3; [8192 x 28672] 70.1 against 55.8; [14336 x 4096], M = 128 31.0 against 24.9).  Above that the stage ring of half an SM is short, and they pay only for weights of more than half as many
// tiles as SMs, which K slices of whole SMs cannot serve, and a short K ([11008 x 4096], M = 100: 17.1 us against 19.0; [5760 x 4096] 13.2
// against 13.0).
template <int QT> constexpr bool eight_fit(int bm) { return bm == 64 ? Geo<QT, 64, 8>::kFits : bm == 128 && Geo<QT, 128, 8>::kFits; }

// SCATTER: finished tiles are also stored to the extra destinations in p.peers (other GPUs' gather buffers).
template <int QT, typename T, int BM, bool SCATTER, int PW>
__global__ void __launch_bounds__(Geo<QT, BM, PW>::template Of<T>::kThreads, Geo<QT, BM, PW>::template Of<T>::kCtasPerSm)
gemm_umma_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ Params p) {
  using S = typename Geo<QT, BM, PW>::template Of<T>;
  constexpr int kPitch = RawGeom<QT>::kPitch, kBoxes = RawGeom<QT>::kBoxes, kBlockBytes = RawGeom<QT>::kSuper, kBox = kRowsW * kPitch;
  extern __shared__ uint8_t smem_raw[];
  Cta<S> cta(p, smem_raw);
  const int warp = cta.warp, lane = cta.lane;

  if (warp < PW) {
    // ------------------------------------------------------------------ producers
    // Eight warps unpack a super-block, thread (row, half) half of a row.  Sixteen are two teams.  Each team takes every other super-block, or,
    // where a worker has few of them, both take every one: team (half), thread (row, stage) then.
    const int row = 32 * (warp & 3) + lane, sub = (warp >> 2) & 1, team = warp >> 3;
    const bool shared = S::kTeams > 1 && p.shared;
    const int half = shared ? team : sub;
    const uint32_t tmem_lane = cta.tmem_base + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(BM);   // this warp's lanes, first A column
    bool alive = true;
    int segi = 0;                                               // segments done by this CTA so far
    int pend_t = -1, pend_b = 0, pend_e = 0;                    // segment whose epilogue has not run yet
    const int stride = shared ? 1 : S::kTeams;                  // this warp's super-blocks: every stride-th
    int turn = shared ? 0 : team;                               // super-blocks until its next one
    typename Cta<S>::Ring raw{0, 0u}, unit{0, 0u};
    raw.step(turn, S::NRAW);
    unit.step(turn * 2 + half, S::NB);
    for (int t = cta.tile_hi; t >= cta.tile_lo && alive; --t, ++segi) {
      int sb_b, sb_e;
      cta.walk.segment(t, sb_b, sb_e);
      for (int sb = sb_b; sb < sb_e; ++sb) {
        if (S::kTeams > 1 && turn-- > 0) continue;
        turn = stride - 1;
        if (!cta.wait(cta.rawfull(raw.at), raw.phase, ST_FULL_TIMEOUT)) { alive = false; break; }
        const int slot = raw.at;
        const uint8_t* rowbase = cta.raw + slot * S::RAW_BYTES + (kBoxes == 2 ? half * kBox : 0) + row * kPitch;
        using H = Half<QT, T>;
        H w;
        auto words_read = [&]() {                               // every lane holds its words: the ring slot may be refilled
          __syncwarp();
          if (lane == 0) mbar_arrive(cta.rawfree(slot));
        };
        const uint32_t slots = tmem_lane + uint32_t(unit.at * (2 * kWSlotCols));
        uint32_t o[16];
        auto slot_free = [&]() -> bool {
          if (!cta.wait(cta.empty(unit.at), unit.phase ^ 1u, ST_EMPTY_TIMEOUT)) return false;
          tcgen05_fence_after();
          return true;
        };
        // groups 2 stage, 2 stage + 1; the first one is unpacked before its slot is waited for
        auto unpack = [&](int stage, bool wait_first) -> bool {
          w.group(2 * stage, o);
          if (wait_first && !slot_free()) return false;
          tmem_st16(slots + uint32_t(stage * kWSlotCols), o);
          w.group(2 * stage + 1, o);
          tmem_st16(slots + uint32_t(stage * kWSlotCols + 16), o);
          return true;
        };
        if (shared) {
          w.load(rowbase, sb, half, H::kLoads == 2 ? sub : 0);
          words_read();
          alive = sub == 0 ? unpack(0, true) : unpack(1, true);
        } else {
          w.load(rowbase, sb, half, 0);
          if constexpr (H::kLoads == 1) words_read();
          alive = unpack(0, true);
          if constexpr (H::kLoads == 2) {
            w.load(rowbase, sb, half, 1);
            words_read();
          }
          if (alive) unpack(1, false);
        }
        if (!alive) break;
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) cta.arrive_lead(cta.full(unit.at));
        raw.step(stride, S::NRAW);
        unit.step(2 * stride, S::NB);
        // The previous segment's epilogue runs only now, after the first super-block of this segment has been unpacked (the ring holds it):
        // the MMA warp finds its next weight tiles ready the moment the accumulator is handed back.
        if (pend_t >= 0) {
          if (!cta.template epilogue<true, SCATTER>(pend_t, pend_b, pend_e, segi - 1, [](float) {})) { alive = false; break; }
          pend_t = -1;
        }
      }
      if (!alive) break;
      if (S::kTeams > 1 && pend_t >= 0) {                       // a segment without a super-block for this warp
        if (!cta.template epilogue<true, SCATTER>(pend_t, pend_b, pend_e, segi - 1, [](float) {})) { alive = false; break; }
      }
      pend_t = t; pend_b = sb_b; pend_e = sb_e;
    }
    if (alive && pend_t >= 0) {
      if (S::SLICED && p.slices > 1) cta.leave_slice();
      else cta.template epilogue<true, SCATTER>(pend_t, pend_b, pend_e, segi - 1, [](float) {});
    }
  } else if (warp == PW) {
    cta.load_activations(&x_map);
  } else if (warp == PW + 1) {
    cta.issue_mmas();
  } else {
    cta.load_weights([&](uint32_t slot, uint32_t bar, int sb, int n0) {
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, uint32_t(S::RAW_BYTES));
        // x coordinate = block start rounded down to 16 bytes; rows past N and bytes past the row end read as zero.  The second box of Q8_0:
        // blocks 4..7 start 8 bytes in
        tma_load_2d(slot, &w_map, bar, (sb * kBlockBytes) & ~15, n0);
        if (kBoxes == 2) tma_load_2d(slot + uint32_t(kBox), &w_map, bar, sb * kBlockBytes + 128, n0);
      }
    });
  }
  if (S::SLICED && p.slices > 1) cta.template join_slices<true, SCATTER>([](float) {});
  cta.finish();
}

// ---------------------------------------------------------------------------------------- host side
constexpr int kMaxCtas = kUmmaMaxCtas;

// Tile shape and grid of one problem.
struct Plan {
  int bm, bn, m_tiles;        // bm: the kernel instantiation (slot sizes), bn: activation rows of a tile
  int workers, slices;        // stream-K workers (CTAs, or pairs of them); with slices > 1 one worker per tile, a cluster of so many CTAs
  int ctas_per_sm;            // 2: eight producer warps per CTA, 1: sixteen
  bool shared;                // few super-blocks per worker: all producers work on the same one
  long long units;
  size_t workspace_bytes;     // fp32 partial tiles, one per CTA; 0 when every worker's range ends on a tile boundary
};

// Where a launch finds its partial-tile workspace, flags and status word.
struct Scratch { float* workspace; int* flags; int* status; };

template <int QT, typename T, int BM, int PW>
int launch(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, const Plan& pl, Scratch sc,
                  const PeerOut& peers, cudaStream_t s) {
  using S = typename Geo<QT, BM, PW>::template Of<T>;
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) return RC_LAUNCH;
  const cuuint32_t estr[2] = {1, 1};
  CUtensorMap x_map, w_map;
  {   // activations [m, k], 16-bit: box = one K stage x bn rows (pairs: half of them), 128-byte swizzle (the MMA's B operand layout)
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(m)};
    const cuuint64_t strides[1] = {cuuint64_t(k) * 2};
    const cuuint32_t box[2] = {cuuint32_t(kBK), cuuint32_t(S::PAIR ? pl.bn / 2 : pl.bn)};
    if (enc(&x_map, Pair<T>::kTmaType, 2, const_cast<void*>(a), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return RC_LAUNCH;
  }
  {   // packed weight as bytes [n, row_bytes]: box = the aligned window around one block x 128 rows, no swizzle
    const cuuint64_t row_bytes = cuuint64_t(k / 256) * RawGeom<QT>::kSuper;
    const cuuint64_t dims[2] = {row_bytes, cuuint64_t(n)};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {cuuint32_t(RawGeom<QT>::kPitch), cuuint32_t(kRowsW)};
    if (enc(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(b), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return RC_LAUNCH;
  }
  const bool scatter = peers.count > 0;
  auto kern = scatter ? gemm_umma_kernel<QT, T, BM, true, PW> : gemm_umma_kernel<QT, T, BM, false, PW>;
  static SmemOptIn granted[2];
  if (!smem_opt_in(kern, S::kSmem, granted[scatter])) return RC_LAUNCH;
  Params p;
  p.bias = bias;
  p.out = c;
  p.partial = sc.workspace;
  p.flags = sc.flags;
  p.status = sc.status;
  p.m = m; p.n = n; p.k = k;
  p.m_tiles = pl.m_tiles;
  p.bn = pl.bn;
  p.slices = pl.slices;
  p.shared = S::kTeams > 1 && pl.shared ? 1 : 0;
  p.units = pl.units;
  p.peers = peers;
  // programmatic stream serialization: see the griddepcontrol notes in the kernel
  return launch_frame<S>(kern, pl.workers, pl.slices, s, x_map, w_map, p) == cudaSuccess ? RC_OK : RC_LAUNCH;
}

constexpr bool eight_fit(int qtype, int bm) {
  switch (qtype) {
    case QTYPE_Q4_K: return eight_fit<QTYPE_Q4_K>(bm);
    case QTYPE_Q5_K: return eight_fit<QTYPE_Q5_K>(bm);
    case QTYPE_Q6_K: return eight_fit<QTYPE_Q6_K>(bm);
    case QTYPE_Q8_0: return eight_fit<QTYPE_Q8_0>(bm);
    case QTYPE_Q4_0: return eight_fit<QTYPE_Q4_0>(bm);
    case QTYPE_MXFP4: return eight_fit<QTYPE_MXFP4>(bm);
    case QTYPE_NVFP4: return eight_fit<QTYPE_NVFP4>(bm);
    case QTYPE_Q2_K: return eight_fit<QTYPE_Q2_K>(bm);
    case QTYPE_Q3_K: return eight_fit<QTYPE_Q3_K>(bm);
    default: return false;
  }
}

// Every instantiation of one weight type: the activation dtype, the tile height and the number of producer warps are picked at run time.  One
// translation unit per weight type calls this (umma_gemm_<type>.cu), so the types compile in parallel.
template <int QT, typename T>
int launch_dtype(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, const Plan& pl, Scratch sc, const PeerOut& peers,
                 cudaStream_t s) {
  if (pl.bm == 64) return launch<QT, T, 64, Geo<QT, 64, 8>::kFits ? 8 : 16>(a, b, bias, c, m, n, k, pl, sc, peers, s);
  if (pl.bm == 256) return launch<QT, T, 256, 16>(a, b, bias, c, m, n, k, pl, sc, peers, s);
  if constexpr (Geo<QT, 128, 8>::kFits)
    if (pl.ctas_per_sm == 2) return launch<QT, T, 128, 8>(a, b, bias, c, m, n, k, pl, sc, peers, s);
  return launch<QT, T, 128, 16>(a, b, bias, c, m, n, k, pl, sc, peers, s);
}
template <int QT>
int launch_qtype(int dtype, const void* a, const void* b, const void* bias, void* c, int m, int n, int k, const Plan& pl, Scratch sc,
                 const PeerOut& peers, cudaStream_t s) {
  return dtype == DINO_BF16 ? launch_dtype<QT, __nv_bfloat16>(a, b, bias, c, m, n, k, pl, sc, peers, s)
                            : launch_dtype<QT, __half>(a, b, bias, c, m, n, k, pl, sc, peers, s);
}

// One function per weight type, each defined in its own translation unit.
#define B200_UMMA_LAUNCH_ARGS                                                                                                   \
  int dtype, const void *a, const void *b, const void *bias, void *c, int m, int n, int k, const Plan &pl, Scratch sc,          \
      const PeerOut &peers, cudaStream_t s
int launch_q4_k(B200_UMMA_LAUNCH_ARGS);
int launch_q5_k(B200_UMMA_LAUNCH_ARGS);
int launch_q6_k(B200_UMMA_LAUNCH_ARGS);
int launch_q8_0(B200_UMMA_LAUNCH_ARGS);
int launch_q4_0(B200_UMMA_LAUNCH_ARGS);
int launch_mxfp4(B200_UMMA_LAUNCH_ARGS);
int launch_nvfp4(B200_UMMA_LAUNCH_ARGS);
int launch_q2_k(B200_UMMA_LAUNCH_ARGS);
int launch_q3_k(B200_UMMA_LAUNCH_ARGS);

}  // namespace umma
}  // namespace b200gguf
