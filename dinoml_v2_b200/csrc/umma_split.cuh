// Fused GGUF GEMM on tcgen05 tensor cores for 16-bit activations and weight rows that are not multiples of 16 bytes (Q6_K with K =
// 11008, 32-weight blocks with K = 2880), above the sizes where mma.sync is the quicker (gemm_exact.cuh): C[M,N] = A[M,K] *
// dequant(W[N,K])^T (+ bias).
//
// Same frame as umma_gemm.cuh (weights as the UMMA A operand from tensor memory, activations by TMA, stream-K, bounded waits); what differs:
//   * no weight is cut to 16 bits: a dequantized weight (fp32) is the sum of TERMS 16-bit numbers - three bfloat16 (24 bits), or two
//     float16 (22 bits, below the rounding of an fp32 sum over K; never finer than float16's own subnormals), fewer where they hold it
//     exactly - in TERMS operand slots per stage, one MMA each against the same activation tile.  (Not for float32 activations: the tensor cores' own accumulation leaves
//     6e-6 on a sum, thirty times what mma.sync with fp32 scaling does.)
//   * R = 16 / gcd(16, row bytes) consecutive rows together are a multiple of 16 bytes: the tensor map's rows are groups of R weight
//     rows, and R boxes per super-block fetch the rows of one residue each, at that residue's 16-byte aligned window.  (One bulk
//     copy per row was measured first: 128 copies of 224 bytes take 6.5 us, whatever the arithmetic; used for the last tile alone it
//     still took NVFP4 [5230 x 2880], M = 24, from 14 to 21 us.)  A last group that is not full has a map of its own, as wide as the
//     rows it has, so that nothing beyond the weight is read;
//   * K may be any multiple of the block (the tail of the last super-block counts as zero);
//   * a result that is not finite is computed again weight by weight: two or three parts of a weight make Inf - Inf of an
//     infinite activation, and a weight or its scale (times 32) may be beyond float16.
// Tensor memory holds the accumulator and a ring of stages, TERMS slots each: up to 256 activation rows (in pairs) with a ring of at least a
// super-block for one or two terms, of two stages for three.
#pragma once
#include "gemm_exact.cuh"
#include "gemv_stream_common.cuh"
#include "umma_gemm.cuh"

namespace b200gguf {
namespace umma {

// Terms that hold a weight exactly, or to 22 bits: an FP4 code times its scale has at most six significant bits, a Q4_0 quant times
// its scale fifteen.
template <int QT, typename T> constexpr int split_terms() {
  return QT == QTYPE_MXFP4 || QT == QTYPE_NVFP4 ? 1 : QT == QTYPE_Q4_0 || std::is_same<T, __half>::value ? 2 : 3;
}
// Whether a scale may be one that the type of the operands does not hold.
template <int QT, typename T> constexpr bool split_checks_scale() { return QT == QTYPE_MXFP4 && std::is_same<T, __half>::value; }
// Types whose stages share packed bytes.
template <int QT> constexpr bool shares_bytes() { return QT == QTYPE_Q6_K || QT == QTYPE_Q2_K || QT == QTYPE_Q3_K; }
// Rings of a tile height.  A hand-over unit is half a super-block with one term, a K stage with more.  Two CTAs share an SM up to 64 activation
// rows with one or two terms (128 with one); three terms would leave each of them two stages, and the words of types that share bytes between
// stages do not fit beside two terms.  What a producer thread takes of a super-block:
//   kHalf: eight producer warps, (row, half), the two stages of half a super-block one after the other;
//   kRun: sixteen, types that share bytes, (row, half, run): 16 weights of every 32 of a half;
//   kStage: sixteen, the others, (row, half, stage);
//   else (three terms beside 256 columns of sums) the ring is shorter than a super-block: eight warps take one stage of both halves each.
template <int QT, typename T, int BM> struct SplitGeo {
  static constexpr int kTerms = split_terms<QT, T>(), HS = kTerms == 1 ? 2 : 1;
  static constexpr bool kPair = BM == 256;
  static constexpr int PW = !kPair && kTerms * BM <= 128 && !shares_bytes<QT>() ? 8 : 16;
  static constexpr int kPart = kRowsW * exact::raw_pitch<QT>(), kUnit = HS * (kPair ? BM / 2 : BM) * kBK * 2, kRest = 1024 + 512;
  static constexpr int kColumns = (PW == 8 ? 256 : 512) - BM, kMost = kColumns / (HS * kTerms * kWSlotCols), kDeep = HS == 1 && PW == 16 ? 4 : 6, NB = kMost < kDeep ? kMost : kDeep;
  static constexpr int kFit = ((PW == 8 ? kSmemHalf : kSmemBudget) - kRest - NB * kUnit) / kPart, NRAW = kFit < 4 ? kFit : 4;
  static constexpr bool kHalf = PW == 8, kLong = NB >= kStagesPerSb / HS, kRun = !kHalf && kLong && shares_bytes<QT>(), kStage = !kHalf && kLong && !kRun;
  using Of = Shape<T, BM, PW, kPair, kTerms, HS, NB, NRAW, kPart, PW, kHalf || (kStage && HS == 1) ? 4 : 8, BM * kRowsW * 4 <= NB * kUnit + NRAW * kPart>;
};

// Group i of a unit -> its dequantized weights as TERMS 16-bit numbers each (term[.][..]).
template <int QT, typename O, int TERMS, int NJ>
__device__ __forceinline__ void split16(const exact::Unit<QT, NJ>& unit, int i, float scale, float mn, uint32_t (&term)[TERMS][8]) {
  constexpr int kOff = exact::byte_offset<QT>();
  if constexpr (TERMS == 1) {
    // FP4: byte - 12 = 2 e2m1, times half the scale; both factors and the product are exact in bfloat16, and in float16 for the scales that
    // it holds (0x43qq is 128 + q as bfloat16; as float16 0x50qq is 32 + q / 32, which leaves the scale 32 times larger, away from the
    // subnormals).  A ue4m3 scale is always one of them; an e8m0 scale is from 2^-23 to 2^11.  A group with another one becomes NaN,
    // unless its weights are all zero, and the results of the row are computed again.
    using V = typename Pair<O>::V;
    constexpr bool kHalf = std::is_same<O, __half>::value;
    const V s1 = Pair<O>::splat(kHalf ? 32.f * scale : scale), off = Pair<O>::splat(kHalf ? 32.f + float(kOff) / 32.f : 128.f + float(kOff));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = unit.bytes(i, k);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t magic = __byte_perm(w, kHalf ? 0x50505050u : 0x43434343u, e == 0 ? 0x4140 : 0x4342);
        term[0][2 * k + e] = as_u32<V>(__hmul2(__hsub2(as_pair<V>(magic), off), s1));
      }
    }
    if constexpr (split_checks_scale<QT, O>()) {
      if (__builtin_expect(scale != 0.f && !(scale >= 0x1p-24f && scale <= 0x1p10f), 0)) {
        const uint32_t fill = ((unit.w[i][0] | unit.w[i][1] | unit.w[i][2] | unit.w[i][3]) >> (4 * unit.u)) & 0x07070707u ? 0x7fff7fffu : 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) term[0][k] = fill;
      }
    }
  } else if constexpr (TERMS == 2 && std::is_same<O, __half>::value && !exact::has_mins<QT>()) {
    // float16, packed: with r = (byte - offset) / 32 (0x50qq is 32 + q / 32) and 32 scale = s1 + s2, hi = fl(r s1), and
    // lo = fl(r s2 + (r s1 - hi)) with the parenthesis exact: three instructions per pair
    const float s32 = 32.f * scale;
    const __half h1 = __float2half_rn(s32);
    const __half2 s1 = __half2half2(h1), s2 = __float2half2_rn(s32 - __half2float(h1)), off = __float2half2_rn(32.f + float(kOff) / 32.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = unit.bytes(i, k);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t magic = __byte_perm(w, 0x50505050u, e == 0 ? 0x4140 : 0x4342);
        const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&magic), off);
        const __half2 hi = __hmul2_rn(r, s1), lo = __hfma2(r, s2, __hfma2(r, s1, __hneg2(hi)));
        term[0][2 * k + e] = *reinterpret_cast<const uint32_t*>(&hi);
        term[1][2 * k + e] = *reinterpret_cast<const uint32_t*>(&lo);
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = unit.bytes(i, k);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float lo = byte_to_float(w, 2 * e), hi = byte_to_float(w, 2 * e + 1);
        if constexpr (kOff != 0) { lo -= float(kOff); hi -= float(kOff); }
        if constexpr (exact::has_mins<QT>()) { lo = fmaf(scale, lo, -mn); hi = fmaf(scale, hi, -mn); }
        else { lo *= scale; hi *= scale; }
#pragma unroll
        for (int tm = 0; tm < TERMS; ++tm) {
          const uint32_t pr = exact::pack<O>(lo, hi);
          term[tm][2 * k + e] = pr;
          if (tm + 1 < TERMS) {
            const float2 back = MmaType<O>::pair_to_float2(pr);
            lo -= back.x;
            hi -= back.y;
          }
        }
      }
    }
  }
}

template <int QT, typename T, int BM>
__global__ void __launch_bounds__(SplitGeo<QT, T, BM>::Of::kThreads, SplitGeo<QT, T, BM>::Of::kCtasPerSm)
gemm_split_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap w_tail_map,
                  const T* __restrict__ x, const uint8_t* __restrict__ w, int residues, const __grid_constant__ Params p) {
  using G = SplitGeo<QT, T, BM>;
  using S = typename G::Of;
  constexpr int PW = S::PW, TERMS = S::TERMS, HS = S::HS, kPitch = exact::raw_pitch<QT>(), kSbBytes = exact::sb_bytes<QT>();
  constexpr bool kRedo = TERMS > 1 || split_checks_scale<QT, T>();
  extern __shared__ uint8_t smem_raw[];
  Cta<S> cta(p, smem_raw);
  const int warp = cta.warp, lane = cta.lane;
  const int64_t row_bytes = int64_t(p.k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes;
  const int rows_per_box = kRowsW / residues;
  float check = 0.f;                              // NaN once one of this thread's results is not finite
  auto seen = [&](float v) { if constexpr (kRedo) check = fmaf(0.f, v, check); };

  if (warp < PW) {
    // ------------------------------------------------------------------ producers
    const int row = 32 * (warp & 3) + lane, sub = (warp >> 2) & 1, team = warp >> 3;
    const uint32_t tmem_a = cta.tmem_base + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(BM);
    const int my_row = ((row & (residues - 1)) * rows_per_box + row / residues) * kPitch;      // in a raw slot: by residue
    bool alive = true;
    int segi = 0, pend_t = -1, pend_b = 0, pend_e = 0;
    // A warp's units are at most NB apart (a wait for a slot could otherwise take the lap before for the one it means), and before the
    // epilogue of the segment before it stores none that only the MMAs after that epilogue set free.
    constexpr bool kHalf = G::kHalf, kStage = G::kStage, kRun = G::kRun;
    constexpr int kStep = kRun || (kHalf && HS == 1) ? 3 : kStage ? S::kUnits : 2;      // from the warp's last unit of a super-block (else: half) to its next one
    static_assert(kStep <= S::NB, "laps");
    const int half = kHalf ? sub : team, stage = kHalf ? 0 : sub;
    typename Cta<S>::Ring raw{0, 0u}, unit{0, 0u};
    unit.step(kHalf || kRun ? half * (2 / HS) : kStage ? (HS == 2 ? half : 2 * half + stage) : team, S::NB);
    static_assert(!kRun || HS == 1, "types that share bytes have two terms at least");
    using Words = exact::Unit<QT, kRun ? 4 : 2>;                       // of a 16-weight run of the stage's two 32-weight groups, or of the half's four
    auto epilogue_before = [&](bool first_sb) -> bool {
      if (!first_sb || pend_t < 0) return true;
      const int t = pend_t;
      pend_t = -1;
      return cta.template epilogue<false, false>(t, pend_b, pend_e, segi - 1, seen);
    };
    // A ring of one super-block, which a warp's next lap of is its next super-block: its slots are the same in all of them.
    constexpr bool kFixed = S::NB == kStagesPerSb && HS == 1 && (kRun || kStage);
    auto slot = [&](int st) { return !kFixed ? unit.at : kRun ? 2 * half + st : 2 * half + stage; };
    auto slot_free = [&](int st) -> bool {
      if (!cta.wait(cta.empty(slot(st)), unit.phase ^ 1u, ST_EMPTY_TIMEOUT)) return false;
      tcgen05_fence_after();
      return true;
    };
    auto signal = [&](int st, int by) {
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) cta.arrive_lead(cta.full(slot(st)));
      if (!kFixed) unit.step(by, S::NB);
      else if (!kRun || st == 1) unit.phase ^= 1u;
    };
    // 16 weights (run u of the 32-weight group j of half hb) to the unit's stage `st`
    auto unpack = [&](const Words& w, int i, int at, uint32_t (&out)[TERMS][8]) {
      const bool in = at < p.k;                                        // else past the end of the row
      split16<QT, T, TERMS>(w, i, in ? w.scale[i] : 0.f, in ? w.mn[i] : 0.f, out);
    };
    auto put = [&](int at, int st, int column, const uint32_t (&out)[TERMS][8]) {       // stage st of the unit in slot `at`
#pragma unroll
      for (int tm = 0; tm < TERMS; ++tm) tmem_st8(tmem_a + uint32_t(((at * HS + st) * TERMS + tm) * kWSlotCols + column), out[tm]);
    };
    for (int t = cta.tile_hi; t >= cta.tile_lo && alive; --t, ++segi) {
      int sb_b, sb_e;
      cta.walk.segment(t, sb_b, sb_e);
      const uint8_t* wrow = w + int64_t(min(cta.row0(t) + row, p.n - 1)) * row_bytes;
      for (int sb = sb_b; sb < sb_e && alive; ++sb) {
        if (!cta.wait(cta.rawfull(raw.at), raw.phase, ST_FULL_TIMEOUT)) { alive = false; break; }
        const uint8_t* block = cta.raw + raw.at * S::RAW_BYTES + my_row + (reinterpret_cast<uintptr_t>(wrow + int64_t(sb) * kSbBytes) & 15);
        auto words_read = [&]() {                                      // every lane holds its words: the ring slot may be refilled
          __syncwarp();
          if (lane == 0) mbar_arrive(cta.rawfree(raw.at));
          raw.step(1, S::NRAW);
        };
        if constexpr (kRun) {
          Words words;
          words.load(block, half, 0, sub);
          words_read();
#pragma unroll
          for (int st = 0; st < 2; ++st) {
            constexpr int kEarly = TERMS == 2 ? 2 : 1;                 // groups unpacked before their slot is waited for (three terms of two spill)
            uint32_t out[kEarly][TERMS][8];
            auto group = [&](int i) { unpack(words, 2 * st + i, sb * 256 + 128 * half + 64 * st + 32 * i + 16 * sub, out[i % kEarly]); };
#pragma unroll
            for (int i = 0; i < kEarly; ++i) group(i);
            if (!slot_free(st)) { alive = false; break; }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (i >= kEarly) group(i);
              put(slot(st), 0, 16 * i + 8 * sub, out[i % kEarly]);
            }
            signal(st, st == 0 ? 1 : kStep);
          }
          // not between the stages, where the words would have to outlive it; the ring holds a whole super-block
          if (alive) alive = epilogue_before(sb == sb_b);
        } else if constexpr (kHalf || kStage) {
          Words words[2];
#pragma unroll
          for (int st = 0; st < (kHalf ? 2 : 1); ++st) {
            const int mine = kHalf ? st : stage;                       // stage of the half
            words[0].load(block, half, 2 * mine, 0);
            words[1].load(block, half, 2 * mine, 1);
            if (!kHalf || st == 1) words_read();
#pragma unroll
            for (int piece = 0; piece < 4; ++piece) {
              const int i = piece >> 1, u = piece & 1;
              uint32_t out[TERMS][8];
              unpack(words[u], i, sb * 256 + 128 * half + 64 * mine + 32 * i + 16 * u, out);
              if (piece == 0 && (HS == 1 || st == 0) && !slot_free(st)) { alive = false; break; }
              put(slot(st), HS == 2 ? mine : 0, 16 * i + 8 * u, out);
            }
            if (!alive) break;
            if (HS == 1 || !kHalf || st == 1) {
              signal(st, kHalf && HS == 1 && st == 0 ? 1 : kStep);
              if (st == 0 || HS == 2) alive = epilogue_before(sb == sb_b);
            }
            if (!alive) break;
          }
        } else {
          // sixteen warps, a ring of two stages: team i takes stage i of either half, thread (row, run) 32 weights of it
#pragma unroll 1
          for (int hb = 0; hb < 2 && alive; ++hb) {
            Words words;
            words.load(block, hb, 2 * team, sub);
            if (hb == 1) words_read();
            if (!slot_free(hb)) { alive = false; break; }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t out[TERMS][8];
              unpack(words, i, sb * 256 + 128 * hb + 64 * team + 32 * i + 16 * sub, out);
              put(slot(hb), 0, 16 * i + 8 * sub, out);
            }
            signal(hb, kStep);
            if (hb == 0) alive = epilogue_before(sb == sb_b);
          }
        }
      }
      if (!alive) break;
      pend_t = t; pend_b = sb_b; pend_e = sb_e;
    }
    if (alive && pend_t >= 0) {
      if (S::SLICED && p.slices > 1) cta.leave_slice();
      else cta.template epilogue<false, false>(pend_t, pend_b, pend_e, segi - 1, seen);
    }
  } else if (warp == PW) {
    cta.load_activations(&x_map);
  } else if (warp == PW + 1) {
    cta.issue_mmas();
  } else {
    cta.load_weights([&](uint32_t slot, uint32_t bar, int sb, int n0) {
      // lane r < residues: the box of the rows r, r + residues, ... (16-bit elements: Q8_0 windows are wider than 256 bytes).  In a tile
      // that reaches past the full groups the residues which the last group still has take its map; what a map does not hold is zero.
      if (lane == 0) mbar_arrive_expect_tx(bar, uint32_t(S::RAW_BYTES));
      __syncwarp();
      if (lane < residues) {
        const bool tail = n0 + kRowsW > p.n && (lane < p.n % residues || p.n < residues);
        tma_load_2d(slot + uint32_t(lane * rows_per_box * kPitch), tail ? &w_tail_map : &w_map, bar,
                    int(((int64_t(lane) * row_bytes + int64_t(sb) * kSbBytes) & ~int64_t(15)) >> 1), n0 / residues);
      }
    });
  }
  if (S::SLICED && p.slices > 1) cta.template join_slices<false, false>(seen);
  if (kRedo && check != 0.f) {                    // at the end, where nothing else is held: inside the epilogue it cost 2 - 5 % of a launch
    T* y = static_cast<T*>(p.out);
    cta.for_stored([&](int n_row, int m_row, int rows) {
      const float bias_v = p.bias != nullptr ? MmaType<T>::to_float(static_cast<const T*>(p.bias)[n_row]) : 0.f;
      redo<QT, T, false>(y + int64_t(m_row) * p.n + n_row, p.n, x + int64_t(m_row) * p.k, p.k, w + int64_t(n_row) * row_bytes, bias_v, rows, p.k);
    });
  }
  cta.finish();
}

template <int QT, typename T, int BM>
int launch_split(const void* x, const void* w, const void* bias, void* c, int m, int n, int k, const Plan& pl, Scratch sc, cudaStream_t s) {
  using S = typename SplitGeo<QT, T, BM>::Of;
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) return RC_LAUNCH;
  const cuuint32_t estr[2] = {1, 1};
  CUtensorMap x_map, w_map, w_tail_map;
  {
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(m)};
    const cuuint64_t strides[1] = {cuuint64_t(k) * 2};
    const cuuint32_t box[2] = {cuuint32_t(kBK), cuuint32_t(S::PAIR ? pl.bn / 2 : pl.bn)};
    if (enc(&x_map, Pair<T>::kTmaType, 2, const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return RC_LAUNCH;
  }
  // Groups of `residues` weight rows as the maps' rows: the full groups, and all groups at the width of the last one (whose odd byte, if
  // any, is rounded up to an element).  A weight with fewer rows than a group has only the second.
  const int64_t row_bytes = int64_t(k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes;
  int residues = 1;
  while ((row_bytes * residues) & 15) residues *= 2;
  const int64_t group = row_bytes * residues, rest = n % residues ? (n % residues) * row_bytes : group;
  auto encode_rows = [&](CUtensorMap* map, int64_t width, int64_t rows) {
    const cuuint64_t dims[2] = {cuuint64_t((width + 1) / 2), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(group)};
    const cuuint32_t box[2] = {cuuint32_t(exact::raw_pitch<QT>() / 2), cuuint32_t(kRowsW / residues)};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  const int64_t groups = (int64_t(n) + residues - 1) / residues;
  if (!encode_rows(&w_tail_map, rest, groups) || !encode_rows(&w_map, n < residues ? rest : group, n < residues ? 1 : n / residues)) return RC_LAUNCH;
  auto kern = gemm_split_kernel<QT, T, BM>;
  static SmemOptIn granted;
  if (!smem_opt_in(kern, S::kSmem, granted)) return RC_LAUNCH;
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
  p.shared = 0;
  p.units = pl.units;
  p.peers = no_peers();
  return launch_frame<S>(kern, pl.workers, pl.slices, s, x_map, w_map, w_tail_map, static_cast<const T*>(x),
                     static_cast<const uint8_t*>(w), residues, p) == cudaSuccess ? RC_OK : RC_LAUNCH;
}

}  // namespace umma
}  // namespace b200gguf
