// Host side of the tcgen05 prefill GEMM: per-(device, stream) scratch, the stream-K plan, the allocation-free scratch and the
// entry that checks a problem and hands it to the weight type's translation unit.  The kernel is in umma_gemm.cuh.
#include <mutex>

#include "umma_gemm.cuh"

namespace b200gguf {

namespace umma {

static ScratchSets<UmmaScratch> g_sets;

// A larger workspace, outside of stream capture only: callers warm a shape up once before capturing a graph.  At least twice the old
// size, which stays for graphs captured with it: what a set holds is bounded by twice its largest workspace.
static bool grow(UmmaScratch& st, size_t need) {
  const size_t size = need > 2 * st.workspace_bytes ? need : 2 * st.workspace_bytes;
  float* p = nullptr;
  if (cudaMalloc(&p, size) != cudaSuccess) return false;
  if (st.workspace != nullptr) st.outgrown.push_back(st.workspace);
  st.workspace = p;
  st.workspace_bytes = size;
  return true;
}

static UmmaScratch* device_state(size_t need_workspace, cudaStream_t stream) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(g_sets.mutex);
  UmmaScratch& st = g_sets.at(dev, stream);
  if (st.status == nullptr) {
    if (cudaMalloc(&st.status, sizeof(int) * (1 + kMaxCtas)) != cudaSuccess) return nullptr;
    st.empty(stream);
  }
  if (need_workspace > st.workspace_bytes) {
    if (!grow(st, need_workspace)) return nullptr;
  }
  return &st;
}

static Plan plan_for(int m, int n, int k, int bm) {
  Plan pl;
  pl.bm = bm;
  pl.m_tiles = (m + pl.bm - 1) / pl.bm;
  // The M rows in equal tiles of a multiple of 16: M = 333 is two tiles of 176 rows, not 256 + 77 padded to 512 (the MMA time and
  // the activation bytes go with the rows of a tile).
  pl.bn = ((m + pl.m_tiles - 1) / pl.m_tiles + 15) / 16 * 16;
  const long long tiles = static_cast<long long>(pl.m_tiles) * ((n + kRowsW - 1) / kRowsW);
  const int nsb = (k + 255) / 256;
  pl.units = tiles * nsb;
  int sm_count = 148;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  if (sm_count > kMaxCtas) sm_count = kMaxCtas;
  // at least four super-blocks per CTA: a small problem is not cut into more pieces than its finishers can add up quickly
  const long long most = pl.units / 4 > 1 ? pl.units / 4 : 1;
  pl.ctas = int(most < sm_count ? most : sm_count);
  pl.workspace_bytes = tiles % pl.ctas == 0 ? 0 : size_t(pl.ctas) * pl.bm * kRowsW * sizeof(float);
  return pl;
}

static Plan make_plan(int m, int n, int k) { return plan_for(m, n, k, m <= 64 ? 64 : m <= 128 ? 128 : 256); }

// For the split-operand kernels (umma_split.cu): the same plan at their tile height, the same scratch.
Plan split_plan(int m, int n, int k, int bm) { return plan_for(m, n, k, bm); }
int split_state(size_t workspace_bytes, cudaStream_t stream, Scratch* sc) {
  UmmaScratch* st = device_state(workspace_bytes, stream);
  if (st == nullptr) return RC_LAUNCH;
  sc->workspace = st->workspace;
  sc->status = st->status;
  sc->flags = st->status + 1;
  return RC_OK;
}

// ---- allocation-free scratch -------------------------------------------------------------------
// Partial-tile workspace, flags and status word that live in the library's own device image instead of cudaMalloc'ed
// memory.  Every GPU that loads the library carries these 16 MiB until the process exits.
constexpr size_t kStaticScratchBytes = size_t(16) << 20;
static __device__ __align__(256) float g_static_scratch[kStaticScratchBytes / sizeof(float)];
static __device__ int g_static_status[1 + kMaxCtas];     // zero-initialised like any static device array

constexpr int kMaxDevices = 64;
struct StaticScratch { float* workspace = nullptr; int* status = nullptr; bool ready = false; };
static StaticScratch g_static[kMaxDevices];

// In host code `g_static_scratch` is only a handle for the symbol, not a device address; the address the kernels
// need is looked up once per device, with that device current.
static int static_scratch(Scratch* out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return RC_LAUNCH;
  std::lock_guard<std::mutex> lock(g_sets.mutex);
  StaticScratch& st = g_static[dev];
  if (!st.ready) {
    void* ws = nullptr;
    void* status = nullptr;
    if (cudaGetSymbolAddress(&ws, g_static_scratch) != cudaSuccess) return RC_LAUNCH;
    if (cudaGetSymbolAddress(&status, g_static_status) != cudaSuccess) return RC_LAUNCH;
    st.workspace = static_cast<float*>(ws);
    st.status = static_cast<int*>(status);
    st.ready = true;
  }
  out->workspace = st.workspace;
  out->status = st.status;
  out->flags = st.status + 1;
  return RC_OK;
}

static int launch_bm(int qtype, int dtype, const void* a, const void* b, const void* bias, void* c, int m, int n, int k, bool use_static,
                     const PeerOut& peers, cudaStream_t s) {
  const Plan pl = make_plan(m, n, k);
  Scratch sc{nullptr, nullptr, nullptr};
  if (use_static) {
    if (pl.workspace_bytes > kStaticScratchBytes) return RC_RANGE;
    if (int rc = static_scratch(&sc)) return rc;
  } else {
    UmmaScratch* st = device_state(pl.workspace_bytes, s);
    if (st == nullptr) return RC_LAUNCH;
    sc.workspace = st->workspace;
    sc.status = st->status;
    sc.flags = st->status + 1;
  }
  switch (qtype) {
    case QTYPE_Q4_K: return launch_q4_k(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q5_K: return launch_q5_k(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q6_K: return launch_q6_k(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q8_0: return launch_q8_0(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q4_0: return launch_q4_0(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_MXFP4: return launch_mxfp4(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_NVFP4: return launch_nvfp4(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q2_K: return launch_q2_k(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    case QTYPE_Q3_K: return launch_q3_k(dtype, a, b, bias, c, m, n, k, pl, sc, peers, s);
    default: return RC_QTYPE;
  }
}

}  // namespace umma

void umma_release_scratch(cudaStream_t s) {
  std::lock_guard<std::mutex> lock(umma::g_sets.mutex);
  umma::g_sets.release(s);
}

// Packed bytes per 256 weights of a row, 0 for a qtype this kernel does not unpack.
static int super_block_bytes(int qtype) {
  switch (qtype) {
    case QTYPE_Q4_K: case QTYPE_Q4_0: case QTYPE_NVFP4: return 144;
    case QTYPE_Q5_K: return 176;
    case QTYPE_Q6_K: return 210;
    case QTYPE_Q8_0: return 272;
    case QTYPE_MXFP4: return 136;
    case QTYPE_Q2_K: return 84;
    case QTYPE_Q3_K: return 110;
    default: return 0;
  }
}

bool gemm_umma_supports(int qtype, int dtype, int m, int n, int k) {
  (void)n;
  if (super_block_bytes(qtype) == 0 || !(dtype == DINO_BF16 || dtype == DINO_F16) || m < 9 || k % 256 != 0) return false;
  const int64_t row_bytes = int64_t(k / 256) * super_block_bytes(qtype);
  return row_bytes % 16 == 0;   // the packed-weight tensor map needs 16-byte row pitches
}

size_t gemm_umma_workspace(int qtype, int dtype, int m, int n, int k) {
  if (!gemm_umma_supports(qtype, dtype, m, n, k)) return 0;
  return umma::make_plan(m, n, k).workspace_bytes;
}

static int gemm_rcr_umma_impl(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k,
                              bool use_static, const PeerOut& peers, cudaStream_t s) {
  if (int rc = check_gemm_args(a, b, c, qtype, dtype, m, n, k)) return rc;
  if (dtype == DINO_F32) return RC_DTYPE;
  if (super_block_bytes(qtype) == 0) return RC_QTYPE;
  // The kernel walks whole 256-weight super-blocks and derives the weight row pitch from k / 256: a Q8_0 weight whose K
  // is only a multiple of 32 would be misaddressed from the second row on.
  if (k % 256 != 0) return RC_ALIGN;
  if ((reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(a)) & 15) return RC_ALIGN;   // tensor-map bases
  if ((int64_t(k) * 2) & 15) return RC_ALIGN;                       // activation row pitch
  if ((int64_t(k / 256) * super_block_bytes(qtype)) & 15) return RC_ALIGN;   // packed-weight row pitch
  return umma::launch_bm(qtype, dtype, a, b, bias, c, m, n, k, use_static, peers, s);
}

int gemm_rcr_umma(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k,
                  cudaStream_t s) {
  return gemm_rcr_umma_impl(a, b, bias, c, qtype, dtype, m, n, k, false, no_peers(), s);
}

// Same kernel, finished tiles also stored to the extra destinations (see PeerOut).
int gemm_rcr_umma_peers(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k,
                        const PeerOut* peers, cudaStream_t s) {
  return gemm_rcr_umma_impl(a, b, bias, c, qtype, dtype, m, n, k, false, peers != nullptr ? *peers : no_peers(), s);
}

// Same kernel, scratch in the library's static device array: no cudaMalloc / cudaFree anywhere on this path.
int gemm_rcr_umma_static(const void* a, const void* b, const void* bias, void* c, int qtype, int dtype, int m, int n, int k,
                         cudaStream_t s) {
  if (m < 17) return RC_RANGE;   // small M belongs to the GEMV kernels, which need no scratch
  return gemm_rcr_umma_impl(a, b, bias, c, qtype, dtype, m, n, k, true, no_peers(), s);
}
size_t gemm_umma_static_scratch_bytes() { return umma::kStaticScratchBytes; }

// Reads (and clears) the device status word the bounded waits write; 0 = no wait ever gave up.  A launch that gave up
// may have left partial-tile flags raised, so they are cleared with the word.
int umma_device_status() {
  int dev = 0, value = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  std::lock_guard<std::mutex> lock(umma::g_sets.mutex);
  value = umma::g_sets.take_kept_word(dev);
  bool read = true;
  umma::g_sets.for_each(dev, [&](UmmaScratch& set) {           // every stream's word on this device; the first non-zero one is reported
    int word = 0;
    if (cudaMemcpy(&word, set.status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) { read = false; return; }
    if (word == 0) return;
    set.empty(nullptr);
    if (value == 0) value = word;
  });
  if (!read) return -1;
  if (dev >= 0 && dev < umma::kMaxDevices && umma::g_static[dev].ready) {   // the static-scratch path's word: always read and cleared
    int word = 0;
    if (cudaMemcpy(&word, umma::g_static[dev].status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (word != 0) {
      cudaMemset(umma::g_static[dev].status, 0, sizeof(int) * (1 + umma::kMaxCtas));
      if (value == 0) value = word;
    }
  }
  if (value != 0) cudaStreamSynchronize(nullptr);               // the flags are down before a launch on any stream
  return value;
}

}  // namespace b200gguf
