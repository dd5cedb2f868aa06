"""CPU test of the workspaces kept per stream (csrc/scratch_sets.h), compiled against a fake CUDA runtime whose stream work is carried out
when the stream is waited for: what a stream that is gone leaves behind - words of a launch that gave up, an error code - must not
reach the next stream, and the error code must still be read."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dinoml_v2_b200" / "csrc"
HARNESS = r"""
#include "scratch_sets.h"
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <set>
using namespace b200gguf;

static std::map<cudaStream_t, std::vector<std::function<void()>>> queued;
static std::set<void*> live;
static bool fail_memset = false;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); std::memset(*p, 0xEE, n); live.insert(*p); return cudaSuccess; }
cudaError_t cudaFree(void* p) { assert(live.erase(p) == 1); std::free(p); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  if (fail_memset) return cudaErrorUnknown;
  queued[s].push_back([=] { std::memset(p, v, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  queued[st].push_back([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  for (auto& f : queued[s]) f();
  queued[s].clear();
  return cudaSuccess;
}
}
static cudaStream_t stream(int i) { return reinterpret_cast<cudaStream_t>(size_t(i)); }

int main() {
  {
    ScratchSets<UmmaScratch> sets;
    auto made = [&](int dev, cudaStream_t s) -> UmmaScratch& {
      UmmaScratch& set = sets.at(dev, s);
      if (!set.made()) { assert(cudaMalloc(reinterpret_cast<void**>(&set.status), sizeof(int) * (1 + kUmmaMaxCtas)) == cudaSuccess); set.empty(s); cudaStreamSynchronize(s); }
      return set;
    };
    UmmaScratch& a = made(0, stream(1));
    int* words = a.status;
    a.status[0] = 7;                                     // a wait gave up ...
    a.status[1 + 3] = 1;                                 // ... and a flag stayed raised
    sets.release(stream(1));
    assert(made(1, stream(2)).status != words);         // another device's stream does not get it
    UmmaScratch& b = made(0, stream(3));
    assert(b.status == words);                           // the set is used again
    for (int i = 0; i <= kUmmaMaxCtas; ++i) assert(b.status[i] == 0);
    assert(sets.take_kept_word(1) == 0 && sets.take_kept_word(0) == 7 && sets.take_kept_word(0) == 0);
    int in_use = 0;
    sets.for_each(0, [&](UmmaScratch&) { ++in_use; });
    assert(in_use == 1);
    // a set that cannot be emptied is given back instead of kept
    fail_memset = true;
    const size_t before = live.size();
    sets.release(stream(3));
    fail_memset = false;
    assert(live.size() == before - 1);
    // a bounded number is kept; workspaces go with their set
    for (int i = 10; i < 20; ++i) {
      UmmaScratch& set = made(0, stream(i));
      cudaMalloc(reinterpret_cast<void**>(&set.workspace), 64);
      set.outgrown.push_back(nullptr);
      cudaMalloc(&set.outgrown.back(), 32);
    }
    for (int i = 10; i < 20; ++i) sets.release(stream(i));
    assert(live.size() == 1 + 3 * ScratchSets<UmmaScratch>::kMaxSpare);
  }
  {
    ScratchSets<StreamScratch> sets;
    StreamScratch& a = sets.at(0, stream(1));
    assert(!a.made());
    cudaMalloc(reinterpret_cast<void**>(&a.partial), kStreamPartialBytes);
    cudaMalloc(reinterpret_cast<void**>(&a.slice_words), kStreamSliceBytes);
    a.empty(stream(1));
    cudaStreamSynchronize(stream(1));
    uint64_t* words = a.partial;
    a.partial[5] = (1ull << 32) | 0x3f800000u;           // a sum that nobody took
    a.slice_words[kStreamSliceBytes / 8 - 1] = 1ull << 32;
    sets.release(stream(1));
    StreamScratch& b = sets.at(0, stream(2));
    assert(b.partial == words && b.slice_words != nullptr);
    for (size_t i = 0; i < kStreamPartialBytes / 8; ++i) assert(b.partial[i] == 0);
    for (size_t i = 0; i < kStreamSliceBytes / 8; ++i) assert(b.slice_words[i] == 0);
  }
  std::puts("ok");
}
"""


def test_sets_of_streams_that_are_gone(tmp_path):
    from dinoml_v2_b200 import build
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    try:
        include = Path(build.nvcc()).resolve().parents[1] / "include"
    except RuntimeError:
        pytest.skip("no CUDA headers")
    (tmp_path / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", f"-I{CSRC}", f"-I{include}", str(tmp_path / "harness.cpp"), "-o", str(tmp_path / "harness")], check=True)
    assert subprocess.run([str(tmp_path / "harness")], check=True, capture_output=True, text=True).stdout == "ok\n"
