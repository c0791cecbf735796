// Copies between device memory and the caller's host arrays.
//
// A copy from or to pageable memory runs through the driver's own staging on
// one thread: 19 GB/s up to ~50 MB, 12 GB/s at 134 MB, and 4.7 GB/s into pages not
// touched yet, where that thread takes the page faults.  Copies of kStagedCopyBytes or more go through a block of
// page-locked slots instead: each of eight threads moves chunks between its two
// slots and the caller's array while the copy engine fills or drains the other
// one.  Measured, driver / staged with a block at hand (ms; medians):
//
//   MB                 16           24           32           47           134
//   up                 0.87 / 1.39  1.29 / 1.69  1.70 / 2.10  2.56 / 2.58  11.2 / 5.5
//   into touched pages 0.82 / 1.30  1.21 / 1.26  1.61 / 1.66  2.33 / 1.89  8.0 / 5.3
//   into new pages     -            -            6.7 / 2.0    10.1 / 2.7   29 / 8
//
// (malloc hands out new pages from 32 MB on.)  48 MB is where both directions gain
// whatever the pages; an array in new pages would gain from 32 MB on.
#ifndef GG_COPY_CUH
#define GG_COPY_CUH

#include <cuda_runtime.h>

#include <cstddef>

namespace gg {

struct HostCopy {
  void* host;
  const void* device;
  size_t bytes;
  // the device array holds int64 fixed-point energies (LSB 2^-32 MeV), the host
  // array receives doubles (same size)
  bool fixed_point;
};

constexpr size_t kStagedCopyBytes = 48u << 20;

// Queues the copies on `stream` of `device` and waits for them.  The host
// arrays may be pageable, page-locked or managed, each as a whole
// (cudaErrorInvalidValue if not).  scratch: device memory that fixed-point arrays
// are converted in, piece by piece if it is smaller; needed where there are any.
cudaError_t copies_to_host(int device, cudaStream_t stream, const HostCopy* copies, int count, void* scratch = nullptr,
                           size_t scratch_bytes = 0);
// One copy to the device; returns when it has landed.
cudaError_t copy_to_device(int device, cudaStream_t stream, void* target, const void* host, size_t bytes);

// The page-locked blocks (at most two of 8 MB per device, made once they pay) are
// kept while some object that copies holds them, and freed with the last.
void hold_staging(int device);
void release_staging(int device);

}  // namespace gg

#endif
