// Staged host copies (gg_copy.cuh).
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "gg_copy.cuh"
#include "gg_internal.cuh"

namespace gg {
namespace {

constexpr int kWorkers = 8;                  // threads of one copy, the caller among them
constexpr int kSlots = 2 * kWorkers;         // two per thread: one moves while the other is copied
constexpr size_t kSlotBytes = 512 * 1024;    // 10 us of PCIe 5 time a slot
constexpr int kBlocksPerDevice = 2;          // copies that can be staged at the same time on one device

struct Block {
  unsigned char* slots = nullptr;
  cudaEvent_t events[kSlots] = {};
  bool leased = false;
};
struct DevicePool {
  int holders = 0;
  double missed = 0.0;  // ms that the copies so far would have saved with one block more
  std::vector<Block*> blocks;
};
std::mutex g_mutex;
std::map<int, DevicePool> g_pools;

void destroy_block(Block* b) {
  for (cudaEvent_t e : b->events)
    if (e) cudaEventDestroy(e);
  if (b->slots) cudaFreeHost(b->slots);
  delete b;
}

// ms that the staged path saves on a copy: per MB 0.05 up (0.04 at 134 MB, 0.057
// at 256 MB), 0.02 into pages that are there and 0.16 into new ones, where the
// driver's one thread takes the page faults.
double saved_up(size_t bytes) { return 0.05e-6 * static_cast<double>(bytes); }
double saved_down(const void* host, size_t bytes) {
  // the page in the middle stands for the array's
  const uintptr_t page = static_cast<uintptr_t>(sysconf(_SC_PAGESIZE));
  const uintptr_t middle = (reinterpret_cast<uintptr_t>(host) + bytes / 2) & ~(page - 1);
  unsigned char there = 1;
  if (mincore(reinterpret_cast<void*>(middle), page, &there) != 0) there = 1;
  return ((there & 1) ? 0.02e-6 : 0.16e-6) * static_cast<double>(bytes);
}
// ms that making and freeing a block takes (8 MB of page-locked memory: 4 to 9 and 1).
constexpr double kBlockCost = 9.0;

// A free block of the device's pool, or a new one once the copies that had to do
// without have missed as much as it costs: a program that moves one volume of 50
// MB and ends keeps the driver's 4 ms (11 to 20 with a block made for it), one
// that moves many pays for the block once.  NULL otherwise, and when memory is
// short (the copy then takes the driver's path).
Block* lease(int device, double saved) {
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_pools.find(device);
  if (it == g_pools.end() || it->second.holders == 0) return nullptr;
  DevicePool& pool = it->second;
  for (Block* b : pool.blocks)
    if (!b->leased) {
      b->leased = true;
      return b;
    }
  if (pool.blocks.size() >= kBlocksPerDevice) return nullptr;
  pool.missed += saved;
  if (pool.missed < kBlockCost) return nullptr;
  pool.missed = 0.0;
  Block* b = new Block();
  bool ok = cudaHostAlloc(reinterpret_cast<void**>(&b->slots), kSlots * kSlotBytes, cudaHostAllocPortable) == cudaSuccess;
  for (cudaEvent_t& e : b->events) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    destroy_block(b);
    return nullptr;
  }
  b->leased = true;
  pool.blocks.push_back(b);
  return b;
}
void give_back(Block* b) {
  std::lock_guard<std::mutex> lock(g_mutex);
  b->leased = false;
}

// int64 fixed point (LSB 2^-32 MeV) to double, written through to host memory:
// the rounding of the integer to a double and an exact power of two, as the
// host conversion's.
__global__ void fixed_to_double_kernel(const long long* __restrict__ q, double* __restrict__ out, size_t n) {
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = static_cast<double>(q[i]) * (1.0 / kEdepScale);
}
cudaError_t fixed_to_double(const void* q, void* out, size_t bytes, cudaStream_t stream) {
  const size_t n = bytes / 8;
  if (n == 0) return cudaSuccess;
  const size_t blocks = (n + 255) / 256;
  fixed_to_double_kernel<<<static_cast<int>(blocks < 592 ? blocks : 592), 256, 0, stream>>>(
      static_cast<const long long*>(q), static_cast<double*>(out), n);
  return cudaGetLastError();
}

struct Chunk {
  unsigned char* host;
  unsigned char* device;
  size_t bytes;
  bool fixed_point;
};

// Moves the chunks of one call through the block: the caller and up to
// kWorkers - 1 threads take the next chunk from a counter, so that fewer
// threads (none could be started) only take longer.
cudaError_t staged(int device, cudaStream_t stream, Block* block, const std::vector<Chunk>& chunks, bool to_host) {
  std::atomic<size_t> next{0};
  std::atomic<int> error{cudaSuccess};
  auto work = [&](int worker) {
    auto failed = [&](cudaError_t e) {
      int none = cudaSuccess;
      if (e != cudaSuccess) error.compare_exchange_strong(none, e);
      return error.load() != cudaSuccess;
    };
    if (failed(cudaSetDevice(device))) return;
    const Chunk* held[2] = {nullptr, nullptr};  // to the host: copied into this slot, not yet moved out
    bool used[2] = {false, false};
    for (int turn = 0;; turn ^= 1) {
      unsigned char* slot = block->slots + (2 * worker + turn) * kSlotBytes;
      const cudaEvent_t event = block->events[2 * worker + turn];
      const size_t k = next.fetch_add(1);
      const Chunk* c = k < chunks.size() && error.load() == cudaSuccess ? &chunks[k] : nullptr;
      if (to_host) {
        if (c) {  // this slot's last chunk was moved out a turn ago
          const cudaError_t e = c->fixed_point ? fixed_to_double(c->device, slot, c->bytes, stream)
                                               : cudaMemcpyAsync(slot, c->device, c->bytes, cudaMemcpyDeviceToHost, stream);
          if (failed(e) || failed(cudaEventRecord(event, stream))) break;
          held[turn] = c;
        }
        const int other = turn ^ 1;
        if (held[other]) {
          if (failed(cudaEventSynchronize(block->events[2 * worker + other]))) break;
          std::memcpy(held[other]->host, block->slots + (2 * worker + other) * kSlotBytes, held[other]->bytes);
          held[other] = nullptr;
        }
        if (!c && !held[turn]) break;
      } else {
        if (!c) break;
        if (used[turn] && failed(cudaEventSynchronize(event))) break;
        std::memcpy(slot, c->host, c->bytes);
        if (failed(cudaMemcpyAsync(c->device, slot, c->bytes, cudaMemcpyHostToDevice, stream)) ||
            failed(cudaEventRecord(event, stream)))
          break;
        used[turn] = true;
      }
    }
  };
  const size_t workers = std::min<size_t>({static_cast<size_t>(kWorkers), chunks.size(),
                                           std::max<size_t>(1, std::thread::hardware_concurrency() / 2)});
  std::vector<std::thread> threads;
  try {
    threads.reserve(workers);
    for (size_t w = 1; w < workers; ++w) threads.emplace_back(work, static_cast<int>(w));
  } catch (...) {  // no more threads: those running and the caller do the rest
  }
  work(0);
  for (std::thread& t : threads) t.join();
  // nothing of this call is in flight in the block once it is given back
  const cudaError_t e = cudaStreamSynchronize(stream);
  return error.load() != cudaSuccess ? static_cast<cudaError_t>(error.load()) : e;
}

// Whether the driver copies straight from or to this host array.  An array of
// which only one end is page-locked is refused, as the driver refuses it.
cudaError_t is_page_locked(const void* host, size_t bytes, bool* locked) {
  const auto known = [](const void* p) {
    cudaPointerAttributes a{};
    const bool k = cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();  // an address unknown to CUDA is not an error here
    return k;
  };
  *locked = known(host);
  return *locked == known(static_cast<const unsigned char*>(host) + bytes - 1) ? cudaSuccess : cudaErrorInvalidValue;
}

// One array by the copy engine, energies in pieces that the scratch holds.
// Nothing but the driver's copies writes to the caller's array: they check its
// whole range where it is page-locked.
cudaError_t queue_copy(const HostCopy& c, void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  if (!c.fixed_point) return cudaMemcpyAsync(c.host, c.device, c.bytes, cudaMemcpyDeviceToHost, stream);
  scratch_bytes &= ~static_cast<size_t>(7);
  if (!scratch || scratch_bytes == 0) return cudaErrorInvalidValue;
  for (size_t at = 0; at < c.bytes; at += scratch_bytes) {
    const size_t bytes = std::min(scratch_bytes, c.bytes - at);
    cudaError_t e = fixed_to_double(static_cast<const unsigned char*>(c.device) + at, scratch, bytes, stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(static_cast<unsigned char*>(c.host) + at, scratch, bytes, cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t copies_to_host(int device, cudaStream_t stream, const HostCopy* copies, int count, void* scratch,
                           size_t scratch_bytes) {
  std::vector<Chunk> chunks;
  std::vector<HostCopy> plain;
  Block* block = nullptr;
  size_t total = 0;
  try {
    std::vector<HostCopy> through;
    for (int i = 0; i < count; ++i) {
      if (copies[i].bytes == 0) continue;
      bool locked = false;
      const cudaError_t known = is_page_locked(copies[i].host, copies[i].bytes, &locked);
      if (known != cudaSuccess) return known;
      (locked ? plain : through).push_back(copies[i]);
      if (!locked) total += copies[i].bytes;
    }
    if (total >= kStagedCopyBytes) {
      double saved = 0.0;
      for (const HostCopy& c : through) saved += saved_down(c.host, c.bytes);
      block = lease(device, saved);
    }
    for (const HostCopy& c : through) {
      if (!block) plain.push_back(c);
      for (size_t at = 0; block && at < c.bytes; at += kSlotBytes)
        chunks.push_back(Chunk{static_cast<unsigned char*>(c.host) + at,
                               static_cast<unsigned char*>(const_cast<void*>(c.device)) + at,
                               std::min(kSlotBytes, c.bytes - at), c.fixed_point});
    }
  } catch (...) {
    if (block) give_back(block);
    return cudaErrorMemoryAllocation;
  }
  cudaError_t e = cudaSuccess;
  for (const HostCopy& c : plain)
    if (e == cudaSuccess) e = queue_copy(c, scratch, scratch_bytes, stream);
  if (block) {
    if (e == cudaSuccess) e = staged(device, stream, block, chunks, true);
    give_back(block);
  }
  const cudaError_t s = cudaStreamSynchronize(stream);
  return e != cudaSuccess ? e : s;
}

cudaError_t copy_to_device(int device, cudaStream_t stream, void* target, const void* host, size_t bytes) {
  if (bytes == 0) return cudaSuccess;
  Block* block = nullptr;
  if (bytes >= kStagedCopyBytes) {
    bool locked = false;
    const cudaError_t known = is_page_locked(host, bytes, &locked);
    if (known != cudaSuccess) return known;
    if (!locked) block = lease(device, saved_up(bytes));
  }
  if (block) {
    std::vector<Chunk> chunks;
    try {
      for (size_t at = 0; at < bytes; at += kSlotBytes)
        chunks.push_back(Chunk{static_cast<unsigned char*>(const_cast<void*>(host)) + at,
                               static_cast<unsigned char*>(target) + at, std::min(kSlotBytes, bytes - at), false});
    } catch (...) {
      give_back(block);
      return cudaErrorMemoryAllocation;
    }
    const cudaError_t e = staged(device, stream, block, chunks, false);
    give_back(block);
    return e;
  }
  const cudaError_t e = cudaMemcpyAsync(target, host, bytes, cudaMemcpyHostToDevice, stream);
  const cudaError_t s = cudaStreamSynchronize(stream);
  return e != cudaSuccess ? e : s;
}

void hold_staging(int device) {
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_pools[device].holders;
}

void release_staging(int device) {
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_pools.find(device);
  if (it == g_pools.end() || --it->second.holders > 0) return;
  for (Block* b : it->second.blocks) destroy_block(b);  // no holder, so no copy has one leased
  g_pools.erase(it);
}

}  // namespace gg
