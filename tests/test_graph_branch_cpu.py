"""GraphBranch (csrc/fargo_internal.h) against stand-ins for the runtime's capture
calls: the edges that a begin / leave / join sequence sets, and for every call
that can fail, that the failure is kept and no later call changes the capture as
if nothing had happened."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cudaprotoplanetarydisksfloat_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r'''
#include <cstdio>
#include <set>
#include <vector>
#include "fargo_internal.h"

// the capture: its status, the nodes the next one depends on, and the call that fails (0: none)
static cudaStreamCaptureStatus g_status;
static std::vector<cudaGraphNode_t> g_deps;
static int g_calls, g_fail;
static bool failing() { return ++g_calls == g_fail; }
static void launch(long id) { g_deps.assign(1, (cudaGraphNode_t)id); }
extern "C" {
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus* st, unsigned long long*, cudaGraph_t*,
                                     const cudaGraphNode_t** deps, size_t* n) {
  if (failing()) return cudaErrorUnknown;
  *st = g_status;
  *deps = g_deps.data();
  *n = g_deps.size();
  return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t* deps, size_t n, unsigned flags) {
  if (failing()) return cudaErrorUnknown;
  if (flags == cudaStreamSetCaptureDependencies) g_deps.clear();
  for (size_t k = 0; k < n; k++) g_deps.push_back(deps[k]);
  return cudaSuccess;
}
}
static void reset(cudaStreamCaptureStatus st, int fail) {
  g_status = st;
  g_calls = 0;
  g_fail = fail;
  launch(1);
}
static bool deps(std::multiset<long> want) {
  std::multiset<long> got;
  for (auto d : g_deps) got.insert((long)d);
  return got == want;
}
int main() {
  int bad = 0;
  {  // a branch of nodes 2, 3 beside node 4, joined
    reset(cudaStreamCaptureStatusActive, 0);
    GraphBranch b;
    bad += !b.begin(nullptr);
    launch(2), launch(3);
    b.leave();
    bad += !deps({1});
    launch(4);
    b.join();
    bad += !deps({4, 3}) || b.err != cudaSuccess;
  }
  {  // outside a capture: nothing, and no error
    reset(cudaStreamCaptureStatusNone, 0);
    GraphBranch b;
    bad += b.begin(nullptr) || b.err != cudaSuccess || g_calls != 1;
  }
  {  // an invalidated capture
    reset(cudaStreamCaptureStatusInvalidated, 0);
    GraphBranch b;
    bad += b.begin(nullptr) || b.err == cudaSuccess;
  }
  for (int fail = 1; fail <= 4; fail++) {  // begin's query, leave's query and update, join's update
    reset(cudaStreamCaptureStatusActive, fail);
    GraphBranch b;
    const bool fork = b.begin(nullptr);
    bad += fork != (fail > 1);
    launch(2);
    if (fork) b.leave();
    launch(4);
    if (fork) b.join();
    bad += b.err == cudaSuccess;
    bad += g_calls != fail;  // no call after the failing one
  }
  {  // more nodes than it holds
    reset(cudaStreamCaptureStatusActive, 0);
    g_deps.assign(GraphBranch::kMost + 1, (cudaGraphNode_t)5);
    GraphBranch b;
    bad += b.begin(nullptr) || b.err == cudaSuccess;
  }
  std::printf("%d\n", bad);
  return bad;
}
'''


def test_every_failure_is_kept(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(PKG, "csrc"),
                           "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(CUDA, "include"), str(src), "-o",
                           str(exe)])
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
