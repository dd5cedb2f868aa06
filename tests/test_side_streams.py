"""CPU test of the streams beside a session's own (csrc/side_streams.h), compiled against a fake CUDA runtime whose stream work is carried out
when something waits for it: workspaces are given back only once the graphs that use them have run on the stream they were launched on,
and the sets of two issuing streams have no stream in common."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dinoml_v2_b200" / "csrc"
HARNESS = r"""
#include "side_streams.h"
#include <cassert>
#include <cstdio>
#include <functional>
#include <set>
#include <vector>
using namespace b200gguf;

struct Event { cudaStream_t stream = nullptr; size_t upto = 0; };
static std::map<cudaStream_t, std::vector<std::function<void()>>> queued;
static std::map<cudaStream_t, size_t> done;
static std::set<cudaStream_t> streams;
static std::set<cudaEvent_t> events;
static int creations_left = 1 << 30;
static void run(cudaStream_t s, size_t upto) { while (done[s] < upto) queued[s][done[s]++](); }
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  if (creations_left-- <= 0) return cudaErrorMemoryAllocation;
  static size_t next = 1000;
  *s = reinterpret_cast<cudaStream_t>(next++);
  streams.insert(*s);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { assert(streams.erase(s) == 1); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s, queued[s].size()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (creations_left-- <= 0) return cudaErrorMemoryAllocation;
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  events.insert(*e);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { assert(events.erase(e) == 1); delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { *reinterpret_cast<Event*>(e) = Event{s, queued[s].size()}; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { run(reinterpret_cast<Event*>(e)->stream, reinterpret_cast<Event*>(e)->upto); return cudaSuccess; }
}
static cudaStream_t stream(int i) { return reinterpret_cast<cudaStream_t>(size_t(i)); }

int main() {
  SideStreams sides;
  SideStreams::Set *a = sides.at(stream(1)), *b = sides.at(stream(2));
  assert(a != nullptr && b != nullptr && sides.at(stream(1)) == a);
  std::set<cudaStream_t> all(a->side, a->side + SideStreams::kSides);
  all.insert(b->side, b->side + SideStreams::kSides);
  assert(all.size() == 2 * SideStreams::kSides && streams == all);
  // two graphs behind other work on stream 1, one on stream 2: each uses the workspaces of its sides when it runs
  std::set<cudaStream_t> given_back;
  int ran = 0;
  auto launch = [&](SideStreams::Set* set, cudaStream_t on) {
    SideStreams::Set of = *set;
    queued[on].push_back([&, of] { for (cudaStream_t s : of.side) assert(given_back.count(s) == 0); ++ran; });
    assert(sides.launched(on) == cudaSuccess);
  };
  launch(a, stream(1));
  launch(b, stream(2));
  launch(a, stream(1));
  queued[stream(1)].push_back([] { assert(!"later work of the caller's stream is not waited for"); });
  auto back = [&](cudaStream_t s) { given_back.insert(s); };
  const cudaStream_t keep = stream(2);
  sides.release(&keep, back);
  assert(ran == 2 && given_back.size() == SideStreams::kSides && streams.size() == SideStreams::kSides && sides.at(stream(2)) == b);
  sides.release(nullptr, back);
  assert(ran == 3 && given_back == all && streams.empty() && events.empty());
  // a stream that is asked for after its set has gone gets a new one; what cannot be made leaves nothing behind
  assert(sides.at(stream(1)) != nullptr);
  sides.release(nullptr, back);
  for (int left = 0; left < 8; ++left) {
    creations_left = left;
    assert(sides.at(stream(3)) == nullptr);
    sides.release(nullptr, back);
    assert(streams.empty() && events.empty());
  }
  std::puts("ok");
}
"""


def test_sets_are_given_back_behind_their_graphs(tmp_path):
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
