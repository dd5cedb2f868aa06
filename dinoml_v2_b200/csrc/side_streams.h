// Streams beside the one a session's runs are issued on, for launches that run side by side.  Host code over the CUDA runtime only.
//
// Kernels keep workspaces per (device, stream), so whoever launches on these streams, or captures on them, uses the workspaces of these
// streams.  There is a set of them per issuing stream: launches and captured graphs of one issuing stream are ordered and may share it, those of two
// streams may overlap and must not (unless the caller orders them: runs that are waited for).  The work of a captured graph runs on the stream that the graph is launched on, where the side
// streams' own order says nothing about it; so an event is recorded behind every such launch, and a set is given back only after it.
#pragma once
#include <cuda_runtime_api.h>

#include <map>

namespace b200gguf {

class SideStreams {
 public:
  static constexpr int kSides = 3;
  struct Set {
    cudaStream_t side[kSides] = {};
    cudaEvent_t forked = nullptr, joined[kSides] = {};
    cudaEvent_t last = nullptr;               // behind the last graph that uses the workspaces of these streams
    bool pending = false;                     // `last` has been recorded
  };

  // The set of an issuing stream, made when first asked for; null if that fails.
  Set* at(cudaStream_t issuing) {
    Set& set = sets_[issuing];
    bool made = event(&set.forked) && event(&set.last);
    for (int i = 0; i < kSides && made; ++i)
      made = (set.side[i] != nullptr || cudaStreamCreateWithFlags(&set.side[i], cudaStreamNonBlocking) == cudaSuccess) && event(&set.joined[i]);
    if (!made) cudaGetLastError();
    return made ? &set : nullptr;
  }
  // A graph that was captured with the set of `issuing` has been launched on `issuing`.
  cudaError_t launched(cudaStream_t issuing) {
    const auto it = sets_.find(issuing);
    if (it == sets_.end()) return cudaSuccess;
    const cudaError_t err = cudaEventRecord(it->second.last, issuing);
    if (err == cudaSuccess) it->second.pending = true;
    return err;
  }
  // Gives back every set but that of `keep`, once nothing uses it any more: workspaces(stream) for each side stream, then the streams.  Null: all.
  template <typename F> void release(const cudaStream_t* keep, F workspaces) {
    for (auto it = sets_.begin(); it != sets_.end();) {
      if (keep != nullptr && it->first == *keep) { ++it; continue; }
      Set& set = it->second;
      if (set.pending) cudaEventSynchronize(set.last);
      for (int i = 0; i < kSides; ++i) {
        if (set.side[i] != nullptr) {
          cudaStreamSynchronize(set.side[i]);
          workspaces(set.side[i]);
          cudaStreamDestroy(set.side[i]);
        }
        if (set.joined[i] != nullptr) cudaEventDestroy(set.joined[i]);
      }
      if (set.forked != nullptr) cudaEventDestroy(set.forked);
      if (set.last != nullptr) cudaEventDestroy(set.last);
      it = sets_.erase(it);
    }
  }

 private:
  static bool event(cudaEvent_t* e) { return *e != nullptr || cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess; }
  std::map<cudaStream_t, Set> sets_;
};

}  // namespace b200gguf
