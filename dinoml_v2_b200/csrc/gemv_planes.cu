// The integer decode GEMV (gemv_stream.cuh with the arithmetic of gemv_int_planes.cuh) for the problems outside the stream family's
// documented range, one or two activation rows: float32 activations, weight rows that are not multiples of 16 bytes (Q6_K with
// K = 11008, 32-weight blocks with K = 2880, ...) and Q8_0.  The mma and simt families hand their calls of that kind here.
#include "gemv_stream.cuh"

namespace b200gguf {

namespace {

template <int QT, typename T, bool RAG>
int launch_rows(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, const PeerOut& peers, cudaStream_t s) {
  return m == 1 ? stream::launch_int<QT, T, 1, RAG>(a, b, bias, c, n, k, peers, s) : stream::launch_int<QT, T, 2, RAG>(a, b, bias, c, n, k, peers, s);
}
template <int QT, bool RAG>
int launch_dtype(int dtype, const void* a, const void* b, const void* bias, void* c, int m, int n, int k, const PeerOut& peers, cudaStream_t s) {
  if (dtype == DINO_F32) return launch_rows<QT, float, RAG>(a, b, bias, c, m, n, k, peers, s);
  if constexpr (RAG || QT == QTYPE_Q8_0) {       // aligned rows of the other types with 16-bit activations belong to the stream family
    if (dtype == DINO_BF16) return launch_rows<QT, __nv_bfloat16, RAG>(a, b, bias, c, m, n, k, peers, s);
    if (dtype == DINO_F16) return launch_rows<QT, __half, RAG>(a, b, bias, c, m, n, k, peers, s);
  }
  return RC_RANGE;
}

}  // namespace

// RC_RANGE: not a problem of this kernel (the caller goes on to its own); the arguments have passed check_gemm_args.
int gemv_planes(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, const PeerOut& peers,
                cudaStream_t s) {
  if (m < 1 || m > 2) return RC_RANGE;
  const int bs = qtype_block_size(qtype);
  const int64_t row_bytes = int64_t(k / bs) * qtype_block_bytes(qtype);
  const uintptr_t base = reinterpret_cast<uintptr_t>(b);
  const bool aligned = ((uintptr_t(row_bytes) | base) & 15) == 0 && k % 256 == 0;
  if ((base | uintptr_t(row_bytes)) & (qtype == QTYPE_Q2_K ? 3 : 1)) return RC_RANGE;      // 2-byte (Q2_K: word) loads
#define B200_PLANES(QT, RAGGED)                                                                                            \
  case QT:                                                                                                                  \
    if (aligned) return launch_dtype<QT, false>(dtype, a, b, bias, c, m, n, k, peers, s);                                   \
    if constexpr (RAGGED) return launch_dtype<QT, true>(dtype, a, b, bias, c, m, n, k, peers, s);                           \
    return RC_RANGE;
  switch (qtype) {
    B200_PLANES(QTYPE_Q8_0, true)
    B200_PLANES(QTYPE_Q6_K, true)
    B200_PLANES(QTYPE_Q4_K, false)          // 144- and 176-byte super-blocks: rows are 16-byte multiples
    B200_PLANES(QTYPE_Q5_K, false)
    B200_PLANES(QTYPE_Q4_0, true)
    B200_PLANES(QTYPE_Q2_K, true)
    B200_PLANES(QTYPE_Q3_K, true)
    default: return RC_RANGE;
  }
#undef B200_PLANES
}

}  // namespace b200gguf
