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
// Tensor memory holds the accumulator and TERMS slots for four stages, so a tile has up to 256 activation rows with one or two terms and
// 128 with three.
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
template <int QT, typename T> constexpr int split_bm() { return split_terms<QT, T>() < 3 ? 256 : 128; }
template <int QT> constexpr int split_raw_slots() { return exact::sb_bytes<QT>() > 240 ? 2 : 3; }
template <int QT, typename T> constexpr size_t split_smem() {
  return 1024 + size_t(kStagesPerSb) * split_bm<QT, T>() * kBK * 2 + size_t(split_raw_slots<QT>()) * kRowsW * exact::raw_pitch<QT>() + 512;
}

// Group i of a unit -> its dequantized weights as TERMS 16-bit numbers each (term[.][q][..]).
template <int QT, typename O, int TERMS>
__device__ __forceinline__ void split16(const exact::Unit<QT, 4>& unit, int i, float scale, float mn, uint32_t (&term)[TERMS][2][8], int q) {
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
        term[0][q][2 * k + e] = as_u32<V>(__hmul2(__hsub2(as_pair<V>(magic), off), s1));
      }
    }
    if constexpr (split_checks_scale<QT, O>()) {
      if (__builtin_expect(scale != 0.f && !(scale >= 0x1p-24f && scale <= 0x1p10f), 0)) {
        const uint32_t fill = ((unit.w[i][0] | unit.w[i][1] | unit.w[i][2] | unit.w[i][3]) >> (4 * unit.u)) & 0x07070707u ? 0x7fff7fffu : 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) term[0][q][k] = fill;
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
        term[0][q][2 * k + e] = *reinterpret_cast<const uint32_t*>(&hi);
        term[1][q][2 * k + e] = *reinterpret_cast<const uint32_t*>(&lo);
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
          term[tm][q][2 * k + e] = pr;
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

template <int QT, typename T>
__global__ void __launch_bounds__(kThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap w_tail_map,
                  const T* __restrict__ x, const uint8_t* __restrict__ w, int residues, const Params p) {
  using P = Pair<T>;
  constexpr int BM = split_bm<QT, T>(), TERMS = split_terms<QT, T>(), NSR = split_raw_slots<QT>(), NS = kStagesPerSb;
  constexpr int kXTile = BM * kBK * 2, kPitch = exact::raw_pitch<QT>(), kRawBytes = kRowsW * kPitch, kSbBytes = exact::sb_bytes<QT>();
  constexpr uint32_t kTmemCols = 512;
  constexpr bool kRedo = TERMS > 1 || split_checks_scale<QT, T>();
  static_assert(BM + NS * TERMS * kWSlotCols <= 512, "tensor memory");
  const uint32_t idesc = (1u << 4) | (P::kFormat << 7) | (P::kFormat << 10) | (uint32_t(p.bn >> 3) << 17) | (uint32_t(kRowsW >> 4) << 24);
  const uint32_t x_bytes = uint32_t(p.bn) * (kBK * 2);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* xtiles = smem;                                              // NS x [BM][128 B]
  uint8_t* raw = xtiles + NS * kXTile;                                 // NSR x [residue][128 / residues][kPitch]
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw + NSR * kRawBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NS + 2 * NSR + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (NS + s); };
  auto rawfull = [&](int s) { return bar0 + 8u * (2 * NS + s); };
  auto rawfree = [&](int s) { return bar0 + 8u * (2 * NS + NSR + s); };
  const uint32_t accbar = bar0 + 8u * (2 * NS + 2 * NSR), accfree = accbar + 8u, drainbar = accbar + 16u, epibar = accbar + 24u;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = blockIdx.x, ctas = gridDim.x;
  const int nsb = (p.k + 255) >> 8;
  const int64_t row_bytes = int64_t(p.k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes;
  const int rows_per_box = kRowsW / residues;
  auto row_offset = [&](int r) { return ((r & (residues - 1)) * rows_per_box + r / residues) * kPitch; };    // of tile row r in a raw slot
  Walk walk;
  walk.u0 = unit_start(cta, p.units, ctas);
  walk.u1 = unit_start(cta + 1, p.units, ctas);
  walk.nsb = nsb;
  const bool has_work = walk.u1 > walk.u0;
  const int tile_hi = has_work ? walk.tile_hi() : -1, tile_lo = has_work ? walk.tile_lo() : 0;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(full(s), kGroupThreads / 32 + 1);      // the 8 producer warps of the stage + the TMA lane's arrive.expect_tx
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < NSR; ++s) {
      mbar_init(rawfull(s), 1);
      mbar_init(rawfree(s), kProducerThreads / 32);
    }
    mbar_init(accbar, 1);
    mbar_init(accfree, kProducerThreads / 32);
    mbar_init(drainbar, 1);
    mbar_init(epibar, kProducerThreads / 32);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

  if (warp < 16) {
    // ------------------------------------------------------------------ producers (roles as in gemm_umma_kernel)
    const int grp = warp >> 3, row = 32 * (warp & 3) + lane, lhalf = (warp >> 2) & 1;
    const uint32_t lanes = uint32_t(32 * (warp & 3)) << 16, tmem_a = tmem_base + lanes + uint32_t(BM);
    const int my_row = row_offset(row);
    bool alive = true;
    int it = 0, segi = 0;
    uint32_t epi_phase = 0;
    auto warp_poll = [&](uint32_t bar, uint32_t parity, int code) -> bool {      // one lane polls, the warp follows
      int ok = 1;
      if (lane == 0) ok = mbar_wait(bar, parity, abort_flag, p.status, code) ? 1 : 0;
      return __shfl_sync(0xffffffffu, ok, 0) != 0;
    };
    auto producer_sync = [&]() -> bool {
      __syncwarp();
      if (lane == 0) mbar_arrive(epibar);
      return warp_poll(epibar, epi_phase++ & 1u, ST_ACC_TIMEOUT);
    };
    bool dep_waited = false;
    float check = 0.f;                              // NaN once one of this thread's results is not finite
    auto epilogue = [&](int t, int sb_b, int sb_e, int segi) -> bool {
      if (!dep_waited) {
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        dep_waited = true;
      }
      if (!warp_poll(accbar, uint32_t(segi) & 1u, ST_ACC_TIMEOUT)) return false;
      tcgen05_fence_after();
      const int n_row = (t / p.m_tiles) * kRowsW + row, m0 = (t % p.m_tiles) * p.bn;
      const bool finishes = sb_e == nsb, whole = finishes && sb_b == 0;
      int peer0 = cta;                              // first CTA with a piece of this tile; peers are peer0 .. cta-1
      if (finishes && !whole) {
        peer0 = unit_owner(static_cast<long long>(t) * nsb, p.units, ctas);
        if (tid < cta - peer0) {
          bool seen = false;
          for (uint32_t i = 0; i < kFlagSpinLimit && !seen; ++i) {
            seen = ld_acquire(p.flags + peer0 + tid) != 0;
            if (!seen) __nanosleep(100);
          }
          if (!seen) { *abort_flag = 1; atomicCAS(p.status, 0, ST_PEER_TIMEOUT); }
        }
        if (!producer_sync()) return false;
      }
      const float bias_v = (finishes && p.bias != nullptr && n_row < p.n) ? MmaType<T>::to_float(static_cast<const T*>(p.bias)[n_row]) : 0.f;
      for (int col = (warp >> 2) * 16; col < p.bn; col += 64) {
        uint32_t r[16];
        tmem_ld16(tmem_base + lanes + uint32_t(col), r);
        tmem_ld_wait();
        if (!finishes) {
          float* dst = p.partial + (static_cast<size_t>(cta) * BM + col) * kRowsW + row;     // tile-local [BM][128]
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[j * kRowsW] = __uint_as_float(r[j]);
        } else {
          for (int peer = peer0; peer < cta; ++peer) {
            const float* src = p.partial + (static_cast<size_t>(peer) * BM + col) * kRowsW + row;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __ldcg(src + j * kRowsW);
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + v[j]);
          }
          if (n_row < p.n) {
            T* dst = static_cast<T*>(p.out) + int64_t(m0 + col) * p.n + n_row;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if constexpr (kRedo) check = fmaf(0.f, __uint_as_float(r[j]), check);
              if (m0 + col + j < p.m) dst[int64_t(j) * p.n] = MmaType<T>::from_float(__uint_as_float(r[j]) + bias_v);
            }
          }
        }
      }
      if (!finishes) {
        if (!producer_sync()) return false;
        if (tid == 0) { __threadfence(); st_release(p.flags + cta, 1); }
      } else if (!whole) {
        if (!producer_sync()) return false;
        if (tid < cta - peer0) p.flags[peer0 + tid] = 0;
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree);
      return true;
    };
    int pend_t = -1, pend_b = 0, pend_e = 0;
    for (int t = tile_hi; t >= tile_lo && alive; --t, ++segi) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const uint8_t* wrow = w + int64_t(min((t / p.m_tiles) * kRowsW + row, p.n - 1)) * row_bytes;
      for (int sb = sb_b; sb < sb_e && alive; ++sb, ++it) {
        const int rslot = it % NSR;
        if (!warp_poll(rawfull(rslot), uint32_t(it / NSR) & 1u, ST_FULL_TIMEOUT)) { alive = false; break; }
        const uint8_t* block = raw + rslot * kRawBytes + my_row + (reinterpret_cast<uintptr_t>(wrow + int64_t(sb) * kSbBytes) & 15);
        exact::Unit<QT, 4> unit;               // K values 16 lhalf .. and 32 + 16 lhalf .. of this thread's two 64-wide stages
        unit.load(block, grp, 0, lhalf);
        __syncwarp();
        if (lane == 0) mbar_arrive(rawfree(rslot));              // every lane holds its words: the ring slot may be refilled
#pragma unroll
        for (int ls = 0; ls < 2; ++ls) {
          const int slot = 2 * grp + ls;
          uint32_t term[TERMS][2][8];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const bool in = sb * 256 + 128 * grp + 64 * ls + 32 * q + 16 * lhalf < p.k;      // else past the end of the row
            split16<QT, T, TERMS>(unit, 2 * ls + q, in ? unit.scale[2 * ls + q] : 0.f, in ? unit.mn[2 * ls + q] : 0.f, term, q);
          }
          if (it > 0) {
            if (!warp_poll(empty(slot), uint32_t(it - 1) & 1u, ST_EMPTY_TIMEOUT)) { alive = false; break; }
            tcgen05_fence_after();
          }
#pragma unroll
          for (int tm = 0; tm < TERMS; ++tm) {
            const uint32_t tile = tmem_a + uint32_t((slot * TERMS + tm) * kWSlotCols);
            tmem_st8(tile + 8 * lhalf, term[tm][0]);
            tmem_st8(tile + 16 + 8 * lhalf, term[tm][1]);
          }
          tmem_st_wait();
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(full(slot));
        }
        if (!alive) break;
        // the previous segment's epilogue, once the first super-block of this one is unpacked
        if (sb == sb_b && pend_t >= 0) {
          if (!epilogue(pend_t, pend_b, pend_e, segi - 1)) { alive = false; break; }
          pend_t = -1;
        }
      }
      if (!alive) break;
      pend_t = t; pend_b = sb_b; pend_e = sb_e;
    }
    if (alive && pend_t >= 0) epilogue(pend_t, pend_b, pend_e, segi - 1);
    if (kRedo && check != 0.f)                      // at the end, where nothing else is held: inside the epilogue it cost 2 - 5 % of a launch
      for (int t = tile_hi; t >= tile_lo; --t) {
        int sb_b, sb_e;
        walk.segment(t, sb_b, sb_e);
        const int n_row = (t / p.m_tiles) * kRowsW + row, m0 = (t % p.m_tiles) * p.bn;
        if (sb_e != nsb || n_row >= p.n) continue;
        const float bias_v = p.bias != nullptr ? MmaType<T>::to_float(static_cast<const T*>(p.bias)[n_row]) : 0.f;
        for (int col = (warp >> 2) * 16; col < min(p.bn, p.m - m0); col += 64)
          redo<QT, T, false>(static_cast<T*>(p.out) + int64_t(m0 + col) * p.n + n_row, p.n, x + int64_t(m0 + col) * p.k, p.k, w + int64_t(n_row) * row_bytes,
                             bias_v, min(16, p.m - m0 - col), p.k);
      }
  } else if (warp == 16) {
    // ------------------------------------------------------------------ activation TMA
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    int it = 0;
    bool ok = true;
    for (int t = tile_hi; t >= tile_lo && ok; --t) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const int m0 = (t % p.m_tiles) * p.bn;
      for (int sb = sb_b; sb < sb_e && ok; ++sb, ++it)
        for (int slot = 0; slot < NS; ++slot) {
          if (it > 0 && !warp_wait(empty(slot), uint32_t(it - 1) & 1u, abort_flag, p.status, ST_EMPTY_TIMEOUT)) { ok = false; break; }
          if (elect_one()) {
            mbar_arrive_expect_tx(full(slot), x_bytes);
            tma_load_2d(smem_u32(xtiles + slot * kXTile), &x_map, full(slot), sb * 256 + slot * kBK, m0);
          }
          __syncwarp();
        }
    }
    // aborting: the copies in flight land within microseconds; their barrier also counts producers that will not come
    if (*abort_flag)
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  } else if (warp == 18) {
    // ------------------------------------------------------------------ packed weights
    int it = 0;
    bool ok = true;
    for (int t = tile_hi; t >= tile_lo && ok; --t) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      const int n0 = (t / p.m_tiles) * kRowsW;
      for (int sb = sb_b; sb < sb_e; ++sb, ++it) {
        const int slot = it % NSR, use = it / NSR;
        if (use > 0 && !warp_wait(rawfree(slot), uint32_t(use - 1) & 1u, abort_flag, p.status, ST_EMPTY_TIMEOUT)) { ok = false; break; }
        const int64_t at = int64_t(sb) * kSbBytes;
        // lane r < residues: the box of the rows r, r + residues, ... (16-bit elements: Q8_0 windows are wider than 256 bytes).  In a tile
        // that reaches past the full groups the residues which the last group still has take its map; what a map does not hold is zero.
        if (lane == 0) mbar_arrive_expect_tx(rawfull(slot), uint32_t(kRawBytes));
        __syncwarp();
        if (lane < residues) {
          const bool tail = n0 + kRowsW > p.n && (lane < p.n % residues || p.n < residues);
          tma_load_2d(smem_u32(raw + slot * kRawBytes + lane * rows_per_box * kPitch), tail ? &w_tail_map : &w_map, rawfull(slot),
                      int(((int64_t(lane) * row_bytes + at) & ~int64_t(15)) >> 1), n0 / residues);
        }
      }
    }
    if (*abort_flag) {
      for (int i = max(0, it - NSR); i < it; ++i) mbar_wait_plain(rawfull(i % NSR), uint32_t(i / NSR) & 1u);
    }
  } else {
    // ------------------------------------------------------------------ MMA issue
    bool ok = true;
    const uint64_t db0 = smem_desc_sw128(smem_u32(xtiles));
    int it = 0, segi = 0;
    for (int t = tile_hi; t >= tile_lo && ok; --t, ++segi) {
      int sb_b, sb_e;
      walk.segment(t, sb_b, sb_e);
      if (segi > 0) {
        ok = warp_wait(accfree, uint32_t(segi - 1) & 1u, abort_flag, p.status, ST_ACC_TIMEOUT);
        if (!ok) break;
        tcgen05_fence_after();
      }
      for (int sb = sb_b; sb < sb_e && ok; ++sb, ++it) {
#pragma unroll
        for (int slot = 0; slot < NS; ++slot) {
          ok = warp_wait(full(slot), uint32_t(it) & 1u, abort_flag, p.status, ST_FULL_TIMEOUT);
          if (!ok) break;
          tcgen05_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int tm = 0; tm < TERMS; ++tm)
#pragma unroll
              for (int kk = 0; kk < kBK / 16; ++kk)
                umma_f16_ts(tmem_base, tmem_base + uint32_t(BM + (slot * TERMS + tm) * kWSlotCols + 8 * kk), db0 + uint64_t((slot * kXTile) >> 4) + uint64_t(2 * kk),
                            idesc, (sb > sb_b || slot > 0 || tm > 0 || kk > 0) ? 1u : 0u);
            umma_commit(empty(slot));
          }
          __syncwarp();
        }
      }
      if (ok && elect_one()) umma_commit(accbar);
      __syncwarp();
    }
    if (!ok && has_work && elect_one()) {   // aborting: let every MMA already issued finish before TMEM is freed
      umma_commit(drainbar);
      mbar_wait_plain(drainbar, 0);
    }
    __syncwarp();
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 17) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

template <int QT, typename T>
int launch_split(const void* x, const void* w, const void* bias, void* c, int m, int n, int k, const Plan& pl, Scratch sc, cudaStream_t s) {
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) return RC_LAUNCH;
  const cuuint32_t estr[2] = {1, 1};
  CUtensorMap x_map, w_map, w_tail_map;
  {
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(m)};
    const cuuint64_t strides[1] = {cuuint64_t(k) * 2};
    const cuuint32_t box[2] = {cuuint32_t(kBK), cuuint32_t(pl.bn)};
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
  auto kern = gemm_split_kernel<QT, T>;
  constexpr size_t smem = split_smem<QT, T>();
  static_assert(smem <= size_t(kSmemBudget), "shared-memory rings exceed the per-CTA limit");
  static SmemOptIn granted;
  if (!smem_opt_in(kern, smem, granted)) return RC_LAUNCH;
  Params p;
  p.bias = bias;
  p.out = c;
  p.partial = sc.workspace;
  p.flags = sc.flags;
  p.status = sc.status;
  p.m = m; p.n = n; p.k = k;
  p.m_tiles = pl.m_tiles;
  p.bn = pl.bn;
  p.units = pl.units;
  p.peers = no_peers();
  return gemv_launch(kern, pl.ctas, 1, kThreads, smem, s, x_map, w_map, w_tail_map, static_cast<const T*>(x),
                     static_cast<const uint8_t*>(w), residues, p) == cudaSuccess ? RC_OK : RC_LAUNCH;
}

}  // namespace umma
}  // namespace b200gguf
