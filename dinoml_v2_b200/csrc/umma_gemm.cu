// Host side of the tcgen05 prefill GEMM: per-(device, stream) scratch, the stream-K plan, the allocation-free scratch and the
// entry that checks a problem and hands it to the weight type's translation unit.  The kernel is in umma_gemm.cuh.
#include <atomic>
#include <cmath>
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

// Clusters of `size` CTAs that the current device runs at once, with one or two CTAs per SM: fewer than the SMs alone would give, since
// a cluster stays within a GPC (B200, one CTA per SM: 33 clusters of four, 15 of eight).
__global__ void __launch_bounds__(16 * 32 + 96, 1) footprint_of_one() {}
__global__ void __launch_bounds__(8 * 32 + 96, 2) footprint_of_two() {}
constexpr int kMostSlices = 16;                                   // CTAs of a cluster: sixteen where the weight has so few tiles that enough clusters fit
static int ask_clusters(int size, int ctas_per_sm) {
  const bool two = ctas_per_sm == 2;
  void (*kern)() = two ? footprint_of_two : footprint_of_one;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(size) * 1024);
  cfg.blockDim = dim3(two ? 8 * 32 + 96 : 16 * 32 + 96);
  cfg.dynamicSmemBytes = two ? kSmemHalf : kSmemBudget;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(size);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cfg.dynamicSmemBytes)) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    clusters = 0;
  }
  return clusters;
}

// What a plan asks about the current device, looked up once per plan; the counts themselves once per device and size (a plan looks at up to 32 of
// them, in calls whose kernel takes 5 us).
struct Device {
  int dev = 0, sm_count = 148;
  Device() {
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    else cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  int max_clusters(int size, int ctas_per_sm) const {
    constexpr int kKept = 64;
    static std::atomic<int> kept[kKept][2][kMostSlices + 1];         // 1 + the count, 0: not asked yet
    if (size < 1 || size > kMostSlices || dev < 0) return 0;
    if (dev >= kKept) return ask_clusters(size, ctas_per_sm);
    std::atomic<int>& known = kept[dev][ctas_per_sm - 1][size];
    int value = known.load(std::memory_order_relaxed);
    if (value == 0) known.store(value = 1 + ask_clusters(size, ctas_per_sm), std::memory_order_relaxed);
    return value - 1;
  }
};

// ctas_per_sm: of the kernel that runs tiles of this height; pairs (bm = 256) are half as many workers.  most_slices: of K, in a cluster.  terms:
// of a weight, a super-block takes that much longer.  *cost: super-blocks that the plan takes the time of.
static Plan plan_for(const Device& device, int m, int n, int k, int bm, int ctas_per_sm, int most_slices, float terms, float* cost_of_plan = nullptr) {
  Plan pl;
  pl.ctas_per_sm = ctas_per_sm;
  const int wide = bm == 256 ? 2 : 1;
  pl.bm = bm;
  pl.m_tiles = (m + pl.bm - 1) / pl.bm;
  // The M rows in equal tiles of a multiple of 16 (pairs: 32): M = 333 is tiles of 192 and 160 rows, not 256 + 77 padded to 512 (the MMA
  // time and the activation bytes go with the rows of a tile).
  pl.bn = ((m + pl.m_tiles - 1) / pl.m_tiles + 16 * wide - 1) / (16 * wide) * (16 * wide);
  const long long tiles = static_cast<long long>(pl.m_tiles) * ((n + wide * kRowsW - 1) / (wide * kRowsW));
  const int nsb = (k + 255) / 256;
  pl.units = tiles * nsb;
  const int sm_count = device.sm_count;
  int slots = sm_count * ctas_per_sm / wide;
  if (slots * wide > kMaxCtas) slots = kMaxCtas / wide;
  if (slots < 1) slots = 1;
  // Three ways to cut the work, compared by their time in super-blocks:
  //   * whole tiles, one per worker, or K slices of them in clusters whose sums meet in shared memory, where all of them run at once: a CTA's own
  //     super-blocks, more of them where another CTA shares its SM, and the join;
  //   * stream-K: an equal share of all units, and the hand-over of cut tiles through the L2, which grows with the rows of a tile.
  // us, [4096 x 4096] Q4_K, M = 16: slices 2 / 4 / 8 9.2 / 7.1 / 8.2, stream-K 10.6; [4096 x 14336] 26.2 / 19.4 / 15.1, stream-K 17.6;
  // [11008 x 4096] 2 / 3 13.0 / 12.6, stream-K 14.5; M = 64, [32768 x 4096]: whole 26.8, stream-K 29.7; [20480 x 4096] 25.8 / 23.1; M = 200,
  // [11008 x 4096]: whole 24.8, stream-K 27.8; [1024 x 4096] 2 / 3 / 4 16.0 / 13.9 / 12.4, whole 21.7, stream-K 18.9.
  // Two CTAs per SM: clusters that would not all fit with one per SM share some, which costs more the longer K is.  37 clusters of four where 33 fit,
  // M = 12, [4696 x 8960]: 14.9, of seven 12.5; Q6_K [4736 x 14336], M = 16: 26.9 / 20.9; [4608 x 4096]: 7.9 / 9.2.
  // (stream-K: at least four super-blocks per worker, a small problem is not cut into more pieces than its finishers can add up quickly.)
  const long long most = pl.units / 4 > 1 ? pl.units / 4 : 1;
  pl.workers = int(most < slots ? most : slots);
  const float join = (wide == 2 ? 1.f : 0.f) / terms, each = (wide == 2 ? 0.7f : 0.3f) / terms, pieces = float(pl.workers) / float(tiles);
  const float hand_over = ((wide == 2 ? 9.f : ctas_per_sm == 1 ? 7.f : 3.f + float(pl.bn) / 16.f) + 0.4f * pieces) / terms;
  float best = float(pl.units * wide) / float(sm_count) + hand_over;
  pl.slices = 0;                                                     // stream-K
  for (int s = 1; s <= most_slices && s <= nsb && tiles <= device.max_clusters(s * wide, ctas_per_sm); ++s) {
    const float load = float(tiles * s * wide) / float(sm_count), own = float(nsb) / float(s);
    const bool alone = load <= 1.f && tiles <= device.max_clusters(s * wide, 1);
    const float more = fmaxf(load, 1.f), share = alone ? 1.f : s == 1 ? 1.75f : fminf(1.75f, sqrtf(more * sqrtf(more)) + own / 64.f);
    const float cost = 0.5f * (float((nsb + s - 1) / s) + own) * share + (s > 1 ? join + each * float(s) : 0.f);
    if (cost < best) { pl.slices = s; best = cost; }
  }
  if (cost_of_plan != nullptr) *cost_of_plan = best;
  if (pl.slices > 0) {
    pl.workers = int(tiles);
    pl.shared = (nsb + pl.slices - 1) / pl.slices <= 12;
    pl.workspace_bytes = 0;
    return pl;
  }
  pl.slices = 1;
  pl.shared = pl.units <= 12ll * pl.workers;
  pl.workspace_bytes = tiles % pl.workers == 0 ? 0 : size_t(pl.workers) * wide * pl.bn * kRowsW * sizeof(float);
  return pl;
}

static int tile_height(int m) { return m <= 64 ? 64 : m <= 128 ? 128 : 256; }
static Plan make_plan(int qtype, int m, int n, int k) {
  const Device device;
  const int bm = tile_height(m), tiles = (n + kRowsW - 1) / kRowsW, sms = device.sm_count;
  const bool eight = eight_fit(qtype, bm) && (bm == 64 || (2 * tiles > sms && tiles <= sms && k <= 16 * 256));
  // (a Q8_0 super-block takes a quarter longer than the others where the activations are not the bound: [11008 x 4096], M = 65: whole 22.8 us, stream-K 22.4)
  Plan pl = plan_for(device, m, n, k, bm, eight ? 2 : 1, kMostSlices / (bm == 256 ? 2 : 1), qtype == QTYPE_Q8_0 && bm == 128 ? 1.25f : 1.f);
  if (qtype == QTYPE_Q8_0) {
    // A Q8_0 row has a scale per 32 weights and nothing that two threads would both unpack, but twice the bytes: up to 64 rows its teams take turns, so
    // that the ring holds two super-blocks for each (us, shared / turns: [6144 x 4096], M = 16 13.5 / 12.5, [28672 x 4096] 38.0 / 35.3); above, the ring is two
    // in all, and where workers cut tiles both teams take every one ([28672 x 4096], M = 100 42.8 / 44.1, M = 129 47.6 / 48.9, [3000 x 7168], M = 700 35.2 / 35.9).
    const bool stream_k = pl.slices == 1 && pl.workers != pl.units / ((k + 255) / 256);
    const long long each = stream_k ? pl.units / pl.workers : ((k + 255) / 256 + pl.slices - 1) / pl.slices;
    pl.shared = each <= (bm == 64 ? 1 : bm == 128 || stream_k ? 32 : 12);
  }
  return pl;
}
// What the built-in scratch takes is decided by this figure: a partial tile of whole height on every SM, where a tile count that the SMs do
// not divide needs one.
static size_t nominal_workspace(int m, int n, int k) {
  const int bm = tile_height(m), nsb = (k + 255) / 256;
  const long long tiles = static_cast<long long>((m + bm - 1) / bm) * ((n + kRowsW - 1) / kRowsW), most = tiles * nsb / 4;
  const int sm_count = Device().sm_count;
  const long long ctas = most < 1 ? 1 : most < sm_count ? most : sm_count;
  return tiles % ctas == 0 ? 0 : size_t(ctas) * bm * kRowsW * sizeof(float);
}

// For the split-operand kernels (umma_split.cu): the same plan at their tile height, the same scratch.
Plan split_plan(int m, int n, int k, int bm, int ctas_per_sm, bool sliced, int terms, float* cost) {
  return plan_for(Device(), m, n, k, bm, ctas_per_sm, !sliced ? 1 : kMostSlices / (bm == 256 ? 2 : 1), float(terms), cost);
}
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
  Plan pl = make_plan(qtype, m, n, k);
  Scratch sc{nullptr, nullptr, nullptr};
  if (use_static) {
    if (nominal_workspace(m, n, k) > kStaticScratchBytes) return RC_RANGE;
    if (pl.workspace_bytes > kStaticScratchBytes) {       // fewer workers, so that their partial tiles fit
      const size_t each = pl.workspace_bytes / pl.workers;
      pl.workers = int(kStaticScratchBytes / each);
      pl.workspace_bytes = pl.workers * each;
    }
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

bool umma_reserve_scratch(cudaStream_t s, cudaStream_t like) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  bool made = false;
  size_t bytes = 0;
  {
    std::lock_guard<std::mutex> lock(umma::g_sets.mutex);
    if (const UmmaScratch* set = umma::g_sets.find(dev, like)) { made = true; bytes = set->workspace_bytes; }
  }
  return !made || umma::device_state(bytes, s) != nullptr;
}

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
  const size_t need = umma::make_plan(qtype, m, n, k).workspace_bytes, nominal = umma::nominal_workspace(m, n, k);
  return need > nominal ? need : nominal;
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
