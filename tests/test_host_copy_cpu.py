"""The copy ring of csrc/host_copy.cpp without a GPU: the file compiled against a
few host stand-ins for the runtime's calls.

Once the ring is there, a copy allocates nothing: an exception in the middle of
one would leave its pieces with the threads, and a slot taken for good.

A page-locked destination is filled by one copy of the driver's, not by way of
the ring (a second pass through host memory).

A forked child that drops what it inherited (a multiprocessing worker whose
copied object is collected) must return: it has neither the ring's threads nor
the right to its locks.  The program forks while another thread copies, so that
locks are held at some of the forks, and gives each child a time limit."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cudaprotoplanetarydisksfloat_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

STUBS = r'''
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>
#include <sys/wait.h>
#include <unistd.h>
#include "host_copy.h"

static std::atomic<long> g_pinned{0};
static void* g_locked = nullptr;  // a destination that counts as page-locked, and the copies straight into it
static std::atomic<long> g_straight{0};
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n); g_pinned++; return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); g_pinned--; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = p == g_locked ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  g_straight += d == g_locked;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
}
static std::vector<char> source(size_t n) {
  std::vector<char> v(n);
  for (size_t k = 0; k < n; k++) v[k] = (char)(k * 2654435761u >> 13);
  return v;
}
'''

FORK = STUBS + r'''
int main() {
  const size_t n = (size_t)30 << 20;
  const std::vector<char> src = source(n);
  const int user = host_copy_retain();
  std::atomic<bool> stop{false};
  std::atomic<int> bad{0};
  std::vector<char> first(n);
  HostPiece p{first.data(), src.data(), n};
  bad += host_copy(&p, 1, 0, nullptr) != cudaSuccess || first != src;
  if (g_pinned != 1) return 2;  // the ring was taken
  std::thread t([&] {
    std::vector<char> dst(n);
    while (!stop) {
      HostPiece q{dst.data(), src.data(), n};
      bad += host_copy(&q, 1, 0, nullptr) != cudaSuccess || dst != src;
      const int u = host_copy_retain();
      host_copy_release(u);
    }
  });
  for (int k = 0; k < 40 && !bad; k++) {
    const pid_t c = fork();
    if (c == 0) {
      alarm(5);  // ends a child that waits for locks or threads it does not have
      host_copy_release(user);
      const int u = host_copy_retain();  // and its own use is its own
      std::vector<char> dst(n);
      HostPiece q{dst.data(), src.data(), n};
      const bool ok = host_copy(&q, 1, 0, nullptr) == cudaSuccess && dst == src;
      host_copy_release(u);
      _exit(ok ? 0 : 1);
    }
    int st = 0;
    waitpid(c, &st, 0);
    if (!WIFEXITED(st) || WEXITSTATUS(st)) bad++;
    usleep(1000);
  }
  stop = true;
  t.join();
  host_copy_release(user);
  if (g_pinned != 0) return 3;  // the parent's ring goes with its last user
  return bad ? 1 : 0;
}
'''


LOCKED = STUBS + r'''
int main() {
  const int user = host_copy_retain();
  int bad = 0;
  for (const size_t n : {(size_t)3 << 20, (size_t)30 << 20}) {
    const std::vector<char> src = source(n);
    // fresh pages (malloc of this size maps them) and touched ones
    for (int touched = 0; touched < 2; touched++) {
      char* dst = (char*)std::malloc(n);
      if (touched) std::memset(dst, 1, n);
      g_locked = dst;
      g_straight = 0;
      HostPiece p{dst, src.data(), n};
      bad += host_copy(&p, 1, 0, nullptr) != cudaSuccess || std::memcmp(dst, src.data(), n) != 0;
      bad += g_straight != 1 || g_pinned != 0;  // one copy into it, no ring made
      std::free(dst);
    }
  }
  host_copy_release(user);
  return bad;
}
'''


NO_ALLOC = STUBS + r'''
static std::atomic<long> g_news{0};
void* operator new(size_t n) {
  g_news++;
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
int main() {
  const size_t n = (size_t)70 << 20;  // 70 pieces: every slot several times
  const std::vector<char> src = source(n);
  std::vector<char> dst(n);
  const int user = host_copy_retain();
  HostPiece p{dst.data(), src.data(), n};
  int bad = host_copy(&p, 1, 0, nullptr) != cudaSuccess;
  const long before = g_news;
  for (int k = 0; k < 5; k++) bad += host_copy(&p, 1, 0, nullptr) != cudaSuccess || dst != src;
  bad += g_news != before;
  host_copy_release(user);
  return bad;
}
'''


def _run(tmp_path, text):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(text)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"),
                           str(src), os.path.join(CSRC, "host_copy.cpp"), "-o", str(exe), "-pthread"])
    return subprocess.run([str(exe)], timeout=300).returncode


def test_forked_child_leaves_the_ring(tmp_path):
    assert _run(tmp_path, FORK) == 0


def test_page_locked_destination_takes_no_detour(tmp_path):
    assert _run(tmp_path, LOCKED) == 0


def test_copies_allocate_nothing(tmp_path):
    assert _run(tmp_path, NO_ALLOC) == 0
