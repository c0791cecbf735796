// Copies between device memory and the caller's host arrays.
//
// A copy from or to pageable memory runs through the driver's own staging on
// one thread.  That is fast up to ~32 MB (16-18 GB/s on the measured host) and
// slow beyond (11 GB/s up, 4.5 GB/s into pages not touched yet), where a copy is
// bound by one core's page faults and moves.  Copies of kStagedCopyBytes or more
// go through a block of page-locked slots instead: each of eight threads moves
// chunks between its two slots and the caller's array while the copy engine fills
// or drains the other one.  Measured, driver against staged: 134 MB up 12.0 / 5.2
// ms, into new pages 29.9 / 8.3 ms; 64 MB 4.3 / 2.7 and 13.5 / 4.2 ms; 20 MB 1.04 /
// 1.45 and 1.26 / 1.19 ms; 3 MB 0.25 / 0.26 and 0.21 / 0.38 ms.
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
