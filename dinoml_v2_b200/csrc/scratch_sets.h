// Workspaces that the launches of one stream share, one set per (device, stream): launches on one stream are ordered (one that
// starts early writes only after the kernel before it has completed) and may share a set, launches on different streams may
// overlap on the GPU and must not.  Host code over the CUDA runtime only.
//
// A set outlives its stream: released ones wait for the next new stream of their device.  Launches hand words to one another inside a
// set (partial sums that carry their own flag, raised flags), and every word is taken down again by its reader - unless a bounded wait
// gave up in between.  So a set is emptied when its stream is released, and an error code that it carries is kept for the next
// status read.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace b200gguf {

// Persistent GEMV (gemv_stream.cuh): partial sums of cut tiles, 16 x 8 words per CTA, and the slice words of launches that cut K.  Empty
// words are zero.  Its status word belongs to the device, not to a set.
constexpr int kStreamMaxCtas = 320;                                                             // cut-tile words are laid out by CTA
constexpr size_t kStreamPartialBytes = size_t(kStreamMaxCtas) * 16 * 8 * sizeof(uint64_t);
constexpr size_t kStreamSliceBytes = size_t(1) << 20;      // slice words of a launch: tiles x slices x 16 rows x activation rows x 8 bytes
struct StreamScratch {
  uint64_t *partial = nullptr, *slice_words = nullptr;
  bool made() const { return partial != nullptr; }
  bool empty(cudaStream_t s) {
    return (partial == nullptr || cudaMemsetAsync(partial, 0, kStreamPartialBytes, s) == cudaSuccess) &&
           (slice_words == nullptr || cudaMemsetAsync(slice_words, 0, kStreamSliceBytes, s) == cudaSuccess);
  }
  int word(cudaStream_t) { return 0; }
  void give_back() {
    if (partial != nullptr) cudaFree(partial);
    if (slice_words != nullptr) cudaFree(slice_words);
  }
};

// tcgen05 GEMMs: partial tiles, and the status word followed by a flag per CTA.
constexpr int kUmmaMaxCtas = 1024;    // flag words per set: a stream-K launch has at most so many CTAs (up to two per SM), and only those use flags
struct UmmaScratch {
  int* status = nullptr;            // [0] = status word, [1 .. kUmmaMaxCtas] = partial-tile flags
  float* workspace = nullptr;
  size_t workspace_bytes = 0;
  std::vector<void*> outgrown;      // smaller workspaces that captured graphs may still use; given back with the set
  bool made() const { return status != nullptr; }
  bool empty(cudaStream_t s) { return status == nullptr || cudaMemsetAsync(status, 0, sizeof(int) * (1 + kUmmaMaxCtas), s) == cudaSuccess; }
  int word(cudaStream_t s) {        // waits for s
    int value = 0;
    if (status != nullptr && (cudaMemcpyAsync(&value, status, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess))
      return 0;
    return value;
  }
  void give_back() {
    if (status != nullptr) cudaFree(status);
    if (workspace != nullptr) cudaFree(workspace);
    for (void* p : outgrown) cudaFree(p);
  }
};

template <typename Set>
class ScratchSets {
 public:
  static constexpr size_t kMaxSpare = 4;      // per device
  std::mutex mutex;                           // held by the caller of everything below

  // The set of a stream: its own, a spare one, or one that is not made() yet.
  Set& at(int dev, cudaStream_t stream) {
    Set& set = sets_[std::make_pair(dev, stream)];
    std::vector<Set>& spare = spare_[dev];
    if (!set.made() && !spare.empty()) {
      set = std::move(spare.back());
      spare.pop_back();
    }
    return set;
  }
  // The set that a stream has, null if it has none.
  const Set* find(int dev, cudaStream_t stream) const {
    const auto it = sets_.find(std::make_pair(dev, stream));
    return it != sets_.end() && it->second.made() ? &it->second : nullptr;
  }
  // `stream` is about to be destroyed and has no work left: its set is emptied and kept for a later stream (a bounded number) or freed.
  void release(cudaStream_t stream) {
    for (auto it = sets_.begin(); it != sets_.end();) {
      if (it->first.second != stream) { ++it; continue; }
      const int dev = it->first.first;
      Set& set = it->second;
      if (set.made()) {
        if (const int word = set.word(stream); word != 0 && kept_word_[dev] == 0) kept_word_[dev] = word;
        std::vector<Set>& spare = spare_[dev];
        if (spare.size() < kMaxSpare && set.empty(stream) && cudaStreamSynchronize(stream) == cudaSuccess) spare.push_back(std::move(set));
        else set.give_back();
      }
      it = sets_.erase(it);
    }
  }
  // The sets in use on a device (spare ones are empty).
  template <typename F> void for_each(int dev, F f) {
    for (auto& entry : sets_)
      if (entry.first.first == dev && entry.second.made()) f(entry.second);
  }
  // Error code of a set whose stream is gone (read once).
  int take_kept_word(int dev) {
    const int word = kept_word_[dev];
    kept_word_[dev] = 0;
    return word;
  }

 private:
  std::map<std::pair<int, cudaStream_t>, Set> sets_;
  std::map<int, std::vector<Set>> spare_;
  std::map<int, int> kept_word_;
};

}  // namespace b200gguf
