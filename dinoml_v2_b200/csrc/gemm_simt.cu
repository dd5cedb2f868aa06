// The "simt" family of the fused GGUF gemm_rcr: C[M,N] = A[M,K] * dequant(W[N,K])^T (+ bias) for every type, activation dtype, M and
// any K that is a multiple of the block - float32 activations and weight rows that are not multiples of 16 bytes in the first place.
// The entry at the end picks the kernel by size: the byte-operand GEMV (gemv_planes.cu), the exact tensor-core GEMM (gemm_exact.cuh), tcgen05
// with split weights (umma_split.cuh), and for what they leave - one or two rows of the FP4 types, 16-bit activations on aligned rows when
// this family is asked for by name - the CUDA-core kernel below: one warp per weight row; lanes stride over 8-wide K units, decode
// them exactly as the dequantizer does, and accumulate in fp32 with FMA; a shuffle tree finishes the row.  It reads W once per group
// of MT activation rows (behavioural ancestor: the reference's one-wave-per-column prototype,
// kernels/rocm/src/ck_gguf_q8_gemm.hip:1168-1207).
#include "gemv_mma_common.cuh"

namespace b200gguf {

int gemm_split(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, cudaStream_t s);
int gemm_exact(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, cudaStream_t s);
int gemv_planes(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, const PeerOut& peers, cudaStream_t s);

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

constexpr int kSimtWarps = 8;

template <int QT, typename T, int MT>
__global__ void __launch_bounds__(kSimtWarps * 32)
gemm_rcr_simt_kernel(const T* __restrict__ a, const uint8_t* __restrict__ b, const T* __restrict__ bias,
                     T* __restrict__ c, int m, int n, int k) {
  constexpr int kUnitsPerBlock = QTraits<QT>::kBlock / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * kSimtWarps + warp;
  const int m0 = blockIdx.y * MT;
  if (col >= n) return;
  const int64_t row_bytes = int64_t(k / QTraits<QT>::kBlock) * QTraits<QT>::kBytes;
  const uint8_t* wrow = b + int64_t(col) * row_bytes;
  float acc[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) acc[i] = 0.f;
  const int units = k >> 3;
  for (int u = lane; u < units; u += 32) {
    const int blk = u / kUnitsPerBlock;
    const int kk0 = (u - blk * kUnitsPerBlock) * 8;
    float w[8];
    decode8<QT>(wrow + int64_t(blk) * QTraits<QT>::kBytes, kk0, w);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if (m0 + i < m) {
        float x[8];
        load8<T>(a + int64_t(m0 + i) * k + int64_t(u) * 8, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i] = fmaf(x[j], w[j], acc[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
  }
  if (lane == 0) {
    const float bv = bias != nullptr ? to_float<T>(bias[col]) : 0.f;
#pragma unroll
    for (int i = 0; i < MT; ++i)
      if (m0 + i < m) c[int64_t(m0 + i) * n + col] = from_float<T>(acc[i] + bv);
  }
}

template <int QT, typename T>
static int launch_simt_t(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, cudaStream_t s) {
  const dim3 block(kSimtWarps * 32);
  if (m == 1) {
    const dim3 grid((n + kSimtWarps - 1) / kSimtWarps, 1);
    gemm_rcr_simt_kernel<QT, T, 1><<<grid, block, 0, s>>>(static_cast<const T*>(a), static_cast<const uint8_t*>(b),
                                                          static_cast<const T*>(bias), static_cast<T*>(c), m, n, k);
  } else {
    const dim3 grid((n + kSimtWarps - 1) / kSimtWarps, (m + 3) / 4);
    if (grid.y > 65535) return RC_RANGE;
    gemm_rcr_simt_kernel<QT, T, 4><<<grid, block, 0, s>>>(static_cast<const T*>(a), static_cast<const uint8_t*>(b),
                                                          static_cast<const T*>(bias), static_cast<T*>(c), m, n, k);
  }
  return cudaGetLastError() == cudaSuccess ? RC_OK : RC_LAUNCH;
}

template <int QT>
static int launch_simt_q(const void* a, const void* b, const void* bias, void* c, int dtype, int m, int n, int k,
                         cudaStream_t s) {
  switch (dtype) {
    case DINO_F32: return launch_simt_t<QT, float>(a, b, bias, c, m, n, k, s);
    case DINO_F16: return launch_simt_t<QT, __half>(a, b, bias, c, m, n, k, s);
    case DINO_BF16: return launch_simt_t<QT, __nv_bfloat16>(a, b, bias, c, m, n, k, s);
    default: return RC_DTYPE;
  }
}

// Shared argument validation of every fused-gemm variant.
int check_gemm_args(const void* a, const void* b, const void* c, int qtype, int dtype, int m, int n, int k) {
  if (a == nullptr || b == nullptr || c == nullptr) return RC_NULL;
  if (m <= 0 || n <= 0 || k <= 0) return RC_DIMS;
  const int bs = qtype_block_size(qtype);
  if (bs == 0) return RC_QTYPE;
  if (k % bs) return RC_KBLOCK;
  if (dtype != DINO_F32 && dtype != DINO_F16 && dtype != DINO_BF16) return RC_DTYPE;
  const uintptr_t aa = reinterpret_cast<uintptr_t>(a), ba = reinterpret_cast<uintptr_t>(b);
  const int64_t row_bytes = int64_t(k / bs) * qtype_block_bytes(qtype);
  const uintptr_t wmask = uintptr_t(qtype_alignment(qtype) - 1);
  if ((aa & 15) || (ba & wmask) || (uintptr_t(row_bytes) & wmask)) return RC_ALIGN;
  return RC_OK;
}

int gemm_rcr_simt(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k,
                  cudaStream_t s) {
  if (int rc = check_gemm_args(a, b, c, qtype, dtype, m, n, k)) return rc;
  // Up to six rows: the byte-operand GEMV, two rows at a time, where the type has it.  It reads the weight up to three times and is
  // still ahead of one pass of the exact GEMM, whose mma.sync work is for 32 rows whatever M is, in the L2 or out of it.  float32 Q8_0,
  // M = 3 / 5, us: [4096 x 4096], 18 MB: 12.1 / 18.2 against 24.4; [28672 x 8192], 250 MB: 88 / 134 against 320; [128256 x 4096], 558 MB:
  // 173 / 259 against 550; Q4_K [65536 x 8192] 113 / 172 against 646.  bfloat16 has a third of that MMA work: Q8_0 [32000 x 2880], 98 MB,
  // 47 / 69 against 92, [128256 x 4128], 563 MB, 298 / 475 against 444; Q4_0 [5760 x 2880] 13.5 / 20.5 against 16.9, Q3_K [4096 x 2560]
  // 10.2 / 15.8 against 13.9: at M = 5 and 6 the shortest and the longest of these would be 7 - 20 % better off there.
  if (m <= 6) {
    const size_t esz = dtype == DINO_F32 ? 4 : 2;
    int rc = RC_OK;
    for (int r = 0; r < m && rc == RC_OK; r += 2)
      rc = gemv_planes(static_cast<const uint8_t*>(a) + size_t(r) * k * esz, b, bias, static_cast<uint8_t*>(c) + size_t(r) * n * esz, qtype, dtype,
                       m - r < 2 ? 1 : 2, n, k, no_peers(), s);
    if (rc != RC_RANGE) return rc;
  }
  // Else the same exact products by mma.sync (one or two rows of the FP4 types stay below: 16 us against 24 us).
  // 16-bit activations on tcgen05 where the weight has enough super-block tiles for all SMs, or tiles and rows together pay for the
  // start of that kernel (us, there / here: Q8_0 [4096 x 2880] float16, M = 8: 10.4 / 14.2; MXFP4 [5760 x 2880] bfloat16, M = 24: 11.0 / 18.9;
  // [2048 x 2880], 192 tiles, M = 64: MXFP4 8.4 / 15.3, Q8_0 10.9 / 16.1; Q6_K [1024 x 2816], 88 tiles, M = 200: 16.8 / 27.9).  Since that kernel
  // cuts K across clusters it is ahead below this line too (M = 32: MXFP4 7.2 / 12.0, Q8_0 10.1 / 12.5; Q6_K M = 100 11.5 / 16.0), but its sums
  // are 6e-6 off where these are 2e-7: what was summed here stays here.
  const int64_t tiles = int64_t((n + 127) / 128) * ((k + 255) / 256);
  if (m >= 7 && (m > 128 || tiles >= 256 || tiles * m >= 12288))
    if (int rc = gemm_split(a, b, bias, c, qtype, dtype, m, n, k, s); rc != RC_RANGE) return rc;
  if (m >= 3)
    if (int rc = gemm_exact(a, b, bias, c, qtype, dtype, m, n, k, s); rc != RC_RANGE) return rc;
  switch (qtype) {
    case QTYPE_Q8_0: return launch_simt_q<QTYPE_Q8_0>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q4_K: return launch_simt_q<QTYPE_Q4_K>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q6_K: return launch_simt_q<QTYPE_Q6_K>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q4_0: return launch_simt_q<QTYPE_Q4_0>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q5_K: return launch_simt_q<QTYPE_Q5_K>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q2_K: return launch_simt_q<QTYPE_Q2_K>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_Q3_K: return launch_simt_q<QTYPE_Q3_K>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_MXFP4: return launch_simt_q<QTYPE_MXFP4>(a, b, bias, c, dtype, m, n, k, s);
    case QTYPE_NVFP4: return launch_simt_q<QTYPE_NVFP4>(a, b, bias, c, dtype, m, n, k, s);
    default: return RC_QTYPE;
  }
}

}  // namespace b200gguf
