// Entry and instantiations of the tcgen05 GEMM with split operands (umma_split.cuh).
#include "umma_split.cuh"

namespace b200gguf {
namespace umma {

Plan split_plan(int m, int n, int k, int bm, int ctas_per_sm, bool sliced, int terms);                                          // umma_gemm.cu
int split_state(size_t workspace_bytes, cudaStream_t stream, Scratch* sc);

template <int QT, typename T, int BM>
static int run_bm(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  const Plan pl = split_plan(m, n, k, BM, SplitGeo<QT, T, BM>::Of::kCtasPerSm, SplitGeo<QT, T, BM>::Of::SLICED, SplitGeo<QT, T, BM>::kTerms);
  Scratch sc;
  if (int rc = split_state(pl.workspace_bytes, s, &sc)) return rc;
  return launch_split<QT, T, BM>(a, b, bias, c, m, n, k, pl, sc, s);
}
template <int QT, typename T>
static int run(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  return m <= 64 ? run_bm<QT, T, 64>(a, b, bias, c, m, n, k, s) : m <= 128 ? run_bm<QT, T, 128>(a, b, bias, c, m, n, k, s) : run_bm<QT, T, 256>(a, b, bias, c, m, n, k, s);
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
