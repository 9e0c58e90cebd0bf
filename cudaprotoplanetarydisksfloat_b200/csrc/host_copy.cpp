// host_copy.cpp -- see host_copy.h
#include "host_copy.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

namespace {

constexpr size_t kSlot = size_t(1) << 20;   // largest piece of a copy
constexpr size_t kLeast = size_t(512) << 10;  // smallest, of copies too short for two full slots a thread
constexpr int kSlots = 16;                  // 16 MiB of page-locked memory per device
constexpr int kThreads = 8;
// The ring is taken from these sizes up: into pages that have no memory yet
// (their faults are most of the time: 12.6 MB 5.9 ms by the driver's own path,
// 1.0 ms by the ring), and into pages that have (waking threads costs 0.3 ms:
// 3.1 MB 0.30 against 0.65 ms, 12.6 MB 0.85 against 1.0 ms, 50 MB 3.3 against
// 2.4 ms).
constexpr size_t kFresh = size_t(2) << 20;
constexpr size_t kBacked = size_t(24) << 20;

// The page-locked ring of one device and the threads that empty it.
class Ring {
 public:
  // false: not available (no memory, no threads); the plain path is taken
  bool open() {
    if (cudaMallocHost(&buf_, kSlot * kSlots) != cudaSuccess) {
      buf_ = nullptr;
      (void)cudaGetLastError();
      return false;
    }
    for (auto& e : ev_)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
      }
    const int n = std::max(1, std::min<int>(kThreads, (int)std::thread::hardware_concurrency() / 2));
    try {
      for (int k = 0; k < n; k++) threads_.emplace_back([this] { work(); });
    } catch (...) {
      return !threads_.empty();
    }
    return true;
  }
  ~Ring() {
    {
      std::lock_guard<std::mutex> l(m_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) t.join();
    for (auto& e : ev_)
      if (e) cudaEventDestroy(e);
    if (buf_) cudaFreeHost(buf_);
  }

  cudaError_t copy(const HostPiece* piece, int n, size_t total, cudaStream_t stream) {
    const size_t step = std::min(kSlot, std::max(kLeast, total / (2 * kThreads) & ~size_t(4095)));
    int p = 0;          // the next piece to issue and the bytes of it already issued
    size_t at = 0;
    long issued = 0, landed = 0;
    cudaError_t err = cudaSuccess;
    Job flight[kSlots];
    for (;;) {
      // as many copies in flight as there are free slots
      while (err == cudaSuccess && p < n && issued - landed < kSlots && free_slot(issued % kSlots, issued == landed)) {
        const int s = (int)(issued % kSlots);
        const size_t b = std::min(step, piece[p].bytes - at);
        flight[s] = {static_cast<char*>(piece[p].dst) + at, buf_ + s * kSlot, b, s};
        err = cudaMemcpyAsync(flight[s].from, static_cast<const char*>(piece[p].src) + at, b, cudaMemcpyDeviceToHost,
                              stream);
        if (err == cudaSuccess) err = cudaEventRecord(ev_[s], stream);
        if (err != cudaSuccess) break;
        issued++;
        at += b;
        if (at == piece[p].bytes) p++, at = 0;
      }
      if (landed == issued) break;
      const int s = (int)(landed % kSlots);
      const cudaError_t e = cudaEventSynchronize(ev_[s]);
      if (e != cudaSuccess) {
        err = e;
        break;
      }
      {
        std::lock_guard<std::mutex> l(m_);
        busy_[s] = true;
        jobs_[given_++ % kSlots] = flight[s];
      }
      wake_.notify_one();
      landed++;
    }
    if (err != cudaSuccess) cudaStreamSynchronize(stream);  // nothing lands in the ring any more
    std::unique_lock<std::mutex> l(m_);
    done_.wait(l, [this] { return std::none_of(busy_, busy_ + kSlots, [](bool b) { return b; }); });
    return err;
  }

  std::mutex user;  // held by the copy that uses the ring

 private:
  struct Job {
    char* to;
    char* from;
    size_t bytes;
    int slot;
  };
  bool free_slot(long s, bool wait) {
    std::unique_lock<std::mutex> l(m_);
    if (wait) done_.wait(l, [&] { return !busy_[s]; });
    return !busy_[s];
  }
  void work() {
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      wake_.wait(l, [this] { return stop_ || taken_ != given_; });
      if (taken_ == given_) return;
      const Job j = jobs_[taken_++ % kSlots];
      l.unlock();
      std::memcpy(j.to, j.from, j.bytes);
      l.lock();
      busy_[j.slot] = false;
      done_.notify_all();
    }
  }
  char* buf_ = nullptr;
  cudaEvent_t ev_[kSlots] = {};
  std::vector<std::thread> threads_;
  std::mutex m_;
  std::condition_variable wake_, done_;
  Job jobs_[kSlots];  // at most one per slot: nothing is allocated while copies are in flight
  unsigned long given_ = 0, taken_ = 0;
  bool busy_[kSlots] = {};
  bool stop_ = false;
};

// The rings of one process, by device.  Plain pointers: what is still open when
// the process ends is left to the system (its threads and the CUDA context go
// first).
struct Process {
  const pid_t pid = getpid();
  std::mutex m;
  int users = 0;
  std::map<int, Ring*> rings;
};
std::atomic<Process*> g_process{nullptr};

// This process's own.  A forked child has a copy of the parent's object, whose
// locks may be held and whose rings' threads are not there: it is never locked
// nor destroyed, the child makes one of its own.
Process& process() {
  const pid_t pid = getpid();
  Process* p = g_process.load();
  while (!p || p->pid != pid) {
    Process* own = new Process();
    if (g_process.compare_exchange_strong(p, own)) return *own;
    delete own;
  }
  return *p;
}

// Whether the middle page of the buffer has no memory yet.
bool fresh(const void* p, size_t bytes) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  const size_t at = (reinterpret_cast<size_t>(p) + bytes / 2) & ~(page - 1);
  unsigned char v = 1;
  return mincore(reinterpret_cast<void*>(at), page, &v) == 0 && !(v & 1);
}

// Ordinary pageable memory.  Anything the runtime knows (page-locked, managed or
// device memory) it fills itself, by one DMA.
bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
  (void)cudaGetLastError();
  return false;
}

Ring* ring_of(int device) {
  Process& own = process();
  std::lock_guard<std::mutex> l(own.m);
  auto it = own.rings.find(device);
  if (it != own.rings.end()) return it->second;
  Ring*& r = own.rings[device];  // null if it cannot be made
  r = new Ring();
  if (!r->open()) {
    delete r;
    r = nullptr;
  }
  return r;
}

}  // namespace

int host_copy_retain() {
  Process& own = process();
  std::lock_guard<std::mutex> l(own.m);
  own.users++;
  return (int)own.pid;
}

void host_copy_release(int user) {
  if (user != (int)getpid()) return;  // the parent's
  Process& own = process();
  std::lock_guard<std::mutex> l(own.m);
  if (--own.users > 0) return;
  for (auto& r : own.rings) delete r.second;
  own.rings.clear();
}

cudaError_t host_copy(const HostPiece* piece, int n, int device, cudaStream_t stream) {
  size_t total = 0;
  for (int k = 0; k < n; k++) total += piece[k].bytes;
  bool through = total >= kBacked;
  for (int k = 0; k < n && !through && total >= kFresh; k++) through = fresh(piece[k].dst, piece[k].bytes);
  for (int k = 0; k < n && through; k++) through = pageable(piece[k].dst);
  if (through) {
    try {
      Ring* r = ring_of(device);
      if (r) {
        std::unique_lock<std::mutex> l(r->user, std::try_to_lock);
        if (l.owns_lock()) return r->copy(piece, n, total, stream);
      }
    } catch (...) {  // no memory for the bookkeeping: the plain path
    }
  }
  for (int k = 0; k < n; k++) {
    const cudaError_t e = cudaMemcpyAsync(piece[k].dst, piece[k].src, piece[k].bytes, cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaStreamSynchronize(stream);
}
