// Entry and instantiations of the tcgen05 GEMM with split operands (umma_split.cuh).
#include "umma_split.cuh"

namespace b200gguf {
namespace umma {

Plan split_plan(int m, int n, int k, int bm, int ctas_per_sm, bool sliced, int terms, float* cost);                             // umma_gemm.cu
int split_state(size_t workspace_bytes, cudaStream_t stream, Scratch* sc);

template <int QT, typename T, int BM>
static Plan plan_bm(int m, int n, int k, float* cost = nullptr) {
  using G = SplitGeo<QT, T, BM>;
  return split_plan(m, n, k, BM, G::Of::kCtasPerSm, G::Of::SLICED, G::kTerms, cost);
}
template <int QT, typename T, int BM>
static int run_bm(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  const Plan pl = plan_bm<QT, T, BM>(m, n, k);
  Scratch sc;
  if (int rc = split_state(pl.workspace_bytes, s, &sc)) return rc;
  return launch_split<QT, T, BM>(a, b, bias, c, m, n, k, pl, sc, s);
}
// More than 128 rows go to pairs, unless there are so few weight tiles that tiles of half as many rows, which unpack a weight twice, fill the SMs
// better: a super-block takes 1.2 - 1.4 times as long in a pair as in a CTA of 128 rows, and the rings of two and three terms of Q2_K and Q3_K are too short for K
// slices of pairs.  us, pairs / 128 rows: Q2_K bfloat16 [300 x 2816], M = 200 29.4 / 10.5, [1024 x 2816] 28.1 / 12.4, Q6_K 17.0 / 13.3; the other way round Q3_K
// [5120 x 5376] 40.6 / 45.2, [8192 x 11008], M = 256 90 / 119.  Where the pairs can be sliced, or with two terms, their estimate is high, and the line lower.
template <int QT, typename T> static bool halves(int m, int n, int k) {
  if constexpr (split_terms<QT, T>() == 1) return false;
  float pairs = 0.f, ctas = 0.f;
  const Plan pl = plan_bm<QT, T, 256>(m, n, k, &pairs);
  plan_bm<QT, T, 128>(m, n, k, &ctas);
  constexpr float kLine = split_terms<QT, T>() == 3 && !SplitGeo<QT, T, 256>::Of::SLICED ? 0.97f : 0.8f;
  return ctas < kLine * pairs * (1.f + float(pl.bn) / 640.f);
}
template <int QT, typename T>
static int run(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  if (m <= 64) return run_bm<QT, T, 64>(a, b, bias, c, m, n, k, s);
  return m <= 128 || halves<QT, T>(m, n, k) ? run_bm<QT, T, 128>(a, b, bias, c, m, n, k, s) : run_bm<QT, T, 256>(a, b, bias, c, m, n, k, s);
}

}  // namespace umma

// RC_RANGE: not a problem of this kernel; the arguments have passed check_gemm_args.
int gemm_split(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(b) & 15) return RC_RANGE;       // tensor-map base
#define B200_SPLIT(QT)                                                                      \
  case QT:                                                                                  \
    return dtype == DINO_BF16  ? umma::run<QT, __nv_bfloat16>(a, b, bias, c, m, n, k, s)   \
           : dtype == DINO_F16 ? umma::run<QT, __half>(a, b, bias, c, m, n, k, s)          \
                               : RC_RANGE;
  switch (qtype) {                        // the types whose rows can miss a 16-byte multiple
    B200_SPLIT(QTYPE_Q8_0)
    B200_SPLIT(QTYPE_Q6_K)
    B200_SPLIT(QTYPE_Q4_0)
    B200_SPLIT(QTYPE_Q2_K)
    B200_SPLIT(QTYPE_Q3_K)
    B200_SPLIT(QTYPE_MXFP4)
    B200_SPLIT(QTYPE_NVFP4)
    default: return RC_RANGE;
  }
#undef B200_SPLIT
}

}  // namespace b200gguf
