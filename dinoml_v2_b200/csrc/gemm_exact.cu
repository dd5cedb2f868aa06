// Instantiations and entry of the exact tensor-core GEMM (gemm_exact.cuh): float32 activations of every weight type, 16-bit
// activations of the types whose weight rows can miss a 16-byte multiple.
#include "gemm_exact.cuh"

namespace b200gguf {

// RC_RANGE: not a problem of this kernel; the arguments have passed check_gemm_args.
int gemm_exact(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, cudaStream_t s) {
#define B200_EXACT(QT, SIXTEEN)                                                                    \
  case QT:                                                                                         \
    if (dtype == DINO_F32) return exact::launch<QT, float>(a, b, bias, c, m, n, k, s);            \
    if constexpr (SIXTEEN) {                                                                       \
      if (dtype == DINO_BF16) return exact::launch<QT, __nv_bfloat16>(a, b, bias, c, m, n, k, s); \
      if (dtype == DINO_F16) return exact::launch<QT, __half>(a, b, bias, c, m, n, k, s);         \
    }                                                                                              \
    return RC_RANGE;
  switch (qtype) {
    B200_EXACT(QTYPE_Q8_0, true)
    B200_EXACT(QTYPE_Q6_K, true)
    B200_EXACT(QTYPE_Q4_K, false)
    B200_EXACT(QTYPE_Q5_K, false)
    B200_EXACT(QTYPE_Q4_0, true)
    B200_EXACT(QTYPE_Q2_K, true)
    B200_EXACT(QTYPE_Q3_K, true)
    B200_EXACT(QTYPE_MXFP4, true)
    B200_EXACT(QTYPE_NVFP4, true)
    default: return RC_RANGE;
  }
#undef B200_EXACT
}

}  // namespace b200gguf
