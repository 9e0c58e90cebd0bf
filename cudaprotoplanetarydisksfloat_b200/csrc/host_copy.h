// host_copy.h -- device-to-host copies of large fields into pageable memory.
//
// A cudaMemcpy into pageable memory runs through the driver's staging buffer on
// the calling thread, which also takes the page faults of a destination that
// was just allocated: 16 disks' fields (98 MB) took 9 ms into touched pages and
// 42 ms into fresh ones.  Here the copies go through a page-locked ring, and a
// few threads move its pieces to the destination while the next ones land (the
// faults are theirs, side by side).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

struct HostPiece {
  void* dst;
  const void* src;
  size_t bytes;
};

// One user (a batch) more or less: host_copy_retain's result goes to
// host_copy_release.  The rings and threads are made by the first large copy on
// a device and given back with the last user.  A forked child that drops a batch
// it inherited leaves the parent's rings alone.
int host_copy_retain();
void host_copy_release(int user);

// Copies device memory to host memory behind what the stream holds, and waits
// for it.  A destination that is not pageable is the driver's to fill.  Safe from several threads: while one uses the ring, another's copy
// takes the plain path.
cudaError_t host_copy(const HostPiece* piece, int n, int device, cudaStream_t stream);
