// Host side of the persistent decode GEMV (kernel: gemv_stream.cuh): scratch, status word, configurations, the instantiations with
// 16-byte weight rows and 16-bit activations.
#include "gemv_stream.cuh"

namespace b200gguf {
namespace stream {

static __device__ int g_stream_status;

int* stream_status_ptr() {
  static int* ptr[kGemvMaxDevices] = {};
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kGemvMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (ptr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_stream_status) != cudaSuccess) return nullptr;
    ptr[dev] = static_cast<int*>(p);
  }
  return ptr[dev];
}

static ScratchSets<StreamScratch> g_sets;        // zeroed once; every word a launch writes is emptied again by the CTA that consumes it

int sm_count() {
  static int counts[kGemvMaxDevices] = {};      // written once per device with the same value
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kGemvMaxDevices) return sms;
  if (counts[dev] > 0) return counts[dev];
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  return counts[dev] = sms;
}

static int zeroed(uint64_t** p, size_t bytes, cudaStream_t stream) {
  // allocated outside of stream capture only: callers warm a shape up once before capturing a graph
  if (cudaMalloc(p, bytes) != cudaSuccess) { *p = nullptr; return RC_LAUNCH; }
  cudaMemsetAsync(*p, 0, bytes, stream);
  return RC_OK;
}

int stream_scratch(cudaStream_t stream, bool slices, Scratch* out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return RC_LAUNCH;
  std::lock_guard<std::mutex> lock(g_sets.mutex);
  Scratch& sc = g_sets.at(dev, stream);
  if (sc.partial == nullptr)
    if (int rc = zeroed(&sc.partial, kStreamPartialBytes, stream)) return rc;
  if (slices && sc.slice_words == nullptr)
    if (int rc = zeroed(&sc.slice_words, kStreamSliceBytes, stream)) return rc;
  *out = sc;
  return RC_OK;
}

// Tuning configurations (the `config` byte of a variant code, see dinoml_b200_gguf.h).  0 = the default for the shape.
//   1: 8 consumer warps, 5 ring slots (Q6_K: 4), one CTA per SM - two launches fit side by side on an SM
//   2: 16 consumer warps, 6 ring slots (Q6_K: 4), one CTA per SM
//   3: 16 consumer warps, 8 ring slots (Q6_K: 6), one CTA per SM
//   4: 8 consumer warps, 4 ring slots (Q6_K: 3), two CTAs per SM
// A Q6_K stage is 26.3 KB against 18.5 KB for Q4_K, hence the shallower rings.
// Bit 7 of the configuration byte (0x80 | 1..4) selects the bandwidth probe of that configuration (bfloat16, M = 1).
constexpr int kStreamConfigs = 4;
constexpr int kProbeBit = 0x80;
template <int QT, typename T, int MXC>
static int launch_m(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, int config, const PeerOut& peers,
                    cudaStream_t s) {
  constexpr bool Q6 = QT == QTYPE_Q6_K || QT == QTYPE_Q5_K;      // the larger stages (26.3 / 23.0 KB): shallower rings
  if constexpr (int_path<QT, MXC>()) {
    // one or two rows: 8 consumer warps whatever the configuration, which picks the CTAs per SM.  Where the digit planes of a long K (4 K
    // bytes per row) leave no room for the ring the default cuts K into slices; past that the 16-bit operand path takes the call.
    constexpr int D = int_depth<QT>();
    // Two rows of Q6_K: its 16-weight sub-blocks need an MMA each there, which pays only where a CTA has several tiles for its planes
    // ([11008 x 4096]: 12.3 us against 13.4 with 16-bit operands; [4096 x 4096]: 6.8 against 6.2, [4096 x 14336]: 19.7 against 16.5).
    if (QT == QTYPE_Q6_K && MXC == 2 && config == 0 && (n + kRows - 1) / kRows <= 2 * sm_count())
      return launch_m<QT, T, 4>(a, b, bias, c, m, n, k, config, peers, s);
    const bool whole = fits<QT, MXC, 1, D>(((k + 255) / 256 + kKC - 1) / kKC, 1);
    switch (whole ? config : 0) {
      case 0: {
        const int rc = launch_int<QT, T, MXC, false>(a, b, bias, c, n, k, peers, s);
        return rc != RC_RANGE ? rc : launch_m<QT, T, 4>(a, b, bias, c, m, n, k, config & ~kProbeBit, peers, s);
      }
      case 1: case 2: case 3: return launch_cfg<QT, T, MXC, 1, D>(a, b, bias, c, m, n, k, 1, peers, s);
      case 4: return launch_cfg<QT, T, MXC, 1, D>(a, b, bias, c, m, n, k, 2, peers, s);
      case kProbeBit | 1: case kProbeBit | 2: case kProbeBit | 3: case kProbeBit | 4:
        if constexpr (MXC == 1 && std::is_same<T, __nv_bfloat16>::value)
          return launch_cfg<QT, T, 1, 1, D, true>(a, b, bias, c, m, n, k, config == (kProbeBit | 4) ? 2 : 1, peers, s);
        return RC_RANGE;
      default: return RC_RANGE;
    }
  } else {
  if (config & kProbeBit) {
    if constexpr (MXC == 1 && std::is_same<T, __nv_bfloat16>::value) {
      switch (config & ~kProbeBit) {
        case 1: return launch_cfg<QT, T, 1, 1, Q6 ? 4 : 5, true>(a, b, bias, c, m, n, k, 1, peers, s);
        case 2: return launch_cfg<QT, T, 1, 2, Q6 ? 4 : 6, true>(a, b, bias, c, m, n, k, 1, peers, s);
        case 3: return launch_cfg<QT, T, 1, 2, Q6 ? 6 : 8, true>(a, b, bias, c, m, n, k, 1, peers, s);
        case 4: return launch_cfg<QT, T, 1, 1, Q6 ? 3 : 4, true>(a, b, bias, c, m, n, k, 2, peers, s);
        default: return RC_RANGE;
      }
    }
    return RC_RANGE;
  }
  if (config == 0) {
    // default: two CTAs of 8 consumer warps per SM; a weight with fewer tiles than SMs runs one CTA of 16 consumer warps each
    config = (n + kRows - 1) / kRows <= sm_count() ? 2 : 4;
  }
  switch (config) {
    case 1: return launch_cfg<QT, T, MXC, 1, Q6 ? 4 : 5>(a, b, bias, c, m, n, k, 1, peers, s);
    case 2: return launch_cfg<QT, T, MXC, 2, Q6 ? 4 : 6>(a, b, bias, c, m, n, k, 1, peers, s);
    case 3: return launch_cfg<QT, T, MXC, 2, Q6 ? 6 : 8>(a, b, bias, c, m, n, k, 1, peers, s);
    case 4: return launch_cfg<QT, T, MXC, 1, Q6 ? 3 : 4>(a, b, bias, c, m, n, k, 2, peers, s);
    default: return RC_RANGE;
  }
  }
}

template <int QT, typename T>
static int launch_q(const void* a, const void* b, const void* bias, void* c, int m, int n, int k, int config, const PeerOut& peers,
                    cudaStream_t s) {
  if (m == 1) return launch_m<QT, T, 1>(a, b, bias, c, m, n, k, config, peers, s);
  if (m == 2) return launch_m<QT, T, 2>(a, b, bias, c, m, n, k, config, peers, s);
  if (m <= 4) return launch_m<QT, T, 4>(a, b, bias, c, m, n, k, config, peers, s);
  return launch_m<QT, T, 8>(a, b, bias, c, m, n, k, config, peers, s);
}

}  // namespace stream

bool stream_reserve_scratch(cudaStream_t s, cudaStream_t like) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  bool made = false, slices = false;
  {
    std::lock_guard<std::mutex> lock(stream::g_sets.mutex);
    if (const StreamScratch* set = stream::g_sets.find(dev, like)) { made = true; slices = set->slice_words != nullptr; }
  }
  stream::Scratch unused;
  return !made || stream::stream_scratch(s, slices, &unused) == RC_OK;
}

void stream_release_scratch(cudaStream_t s) {
  std::lock_guard<std::mutex> lock(stream::g_sets.mutex);
  stream::g_sets.release(s);
}

bool gemv_stream_supports(int qtype, int dtype, int m, int n, int k) {
  (void)n;
  if (!(dtype == DINO_BF16 || dtype == DINO_F16) || m < 1 || m > 8) return false;
  if (qtype == QTYPE_Q4_K || qtype == QTYPE_Q5_K) return k % 256 == 0;      // 144 / 176-byte blocks: rows are always 16-byte multiples
  if (qtype == QTYPE_Q6_K) return k % 2048 == 0;      // 210-byte blocks: row pieces start on 16-byte boundaries only then
  // the further types: whole 256-weight groups and weight rows that are multiples of 16 bytes (bulk-copy sources)
  int sb_bytes = 0;
  switch (qtype) {
    case QTYPE_Q4_0: sb_bytes = 8 * 18; break;
    case QTYPE_Q2_K: sb_bytes = 84; break;
    case QTYPE_Q3_K: sb_bytes = 110; break;
    case QTYPE_MXFP4: sb_bytes = 8 * 17; break;
    case QTYPE_NVFP4: sb_bytes = 4 * 36; break;
    default: return false;
  }
  return k % 256 == 0 && (int64_t(k / 256) * sb_bytes) % 16 == 0;
}
int gemv_stream_configs() { return stream::kStreamConfigs; }

// peers: extra destinations of the result / gated epilogue (null = none); config: tuning configuration, 0 = default.
int gemm_rcr_stream_peers(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, int config,
                          const PeerOut* peer_out, cudaStream_t s) {
  const PeerOut peers = peer_out != nullptr ? *peer_out : no_peers();
  if (int rc = check_gemm_args(a, b, c, qtype, dtype, m, n, k)) return rc;
  if (dtype == DINO_F32) return RC_DTYPE;
  if (m > 8) return RC_RANGE;
  if (qtype == QTYPE_Q8_0) return RC_QTYPE;
  if (!gemv_stream_supports(qtype, dtype, m, n, k)) return RC_ALIGN;
  if ((reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(a)) & 15) return RC_ALIGN;   // bulk-copy sources, vector loads
#define B200_STREAM_QTYPE(QT)                                                                                        \
  if (qtype == QT)                                                                                                    \
    return dtype == DINO_BF16 ? stream::launch_q<QT, __nv_bfloat16>(a, b, bias, c, m, n, k, config, peers, s)        \
                              : stream::launch_q<QT, __half>(a, b, bias, c, m, n, k, config, peers, s);
  B200_STREAM_QTYPE(QTYPE_Q6_K)
  B200_STREAM_QTYPE(QTYPE_Q4_0)
  B200_STREAM_QTYPE(QTYPE_Q5_K)
  B200_STREAM_QTYPE(QTYPE_Q2_K)
  B200_STREAM_QTYPE(QTYPE_Q3_K)
  B200_STREAM_QTYPE(QTYPE_MXFP4)
  B200_STREAM_QTYPE(QTYPE_NVFP4)
#undef B200_STREAM_QTYPE
  return dtype == DINO_BF16 ? stream::launch_q<QTYPE_Q4_K, __nv_bfloat16>(a, b, bias, c, m, n, k, config, peers, s)
                            : stream::launch_q<QTYPE_Q4_K, __half>(a, b, bias, c, m, n, k, config, peers, s);
}

int gemm_rcr_stream(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k, int config,
                    cudaStream_t s) {
  return gemm_rcr_stream_peers(a, b, bias, c, qtype, dtype, m, n, k, config, nullptr, s);
}

// Reads (and clears) the stream kernels' status word of the current device.
int stream_device_status() {
  int* status = stream::stream_status_ptr();
  int value = 0;
  if (status == nullptr) return -1;
  if (cudaMemcpy(&value, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (value != 0) {
    // a launch that gave up may have left partial sums behind: empty them with the word
    cudaMemset(status, 0, sizeof(int));
    int dev = -1;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(stream::g_sets.mutex);
    stream::g_sets.for_each(dev, [](StreamScratch& set) { set.empty(nullptr); });
    cudaStreamSynchronize(nullptr);             // before a launch on any stream
  }
  return value;
}

}  // namespace b200gguf
