// host_copy.cu -- copies of large arrays between pageable host memory and the
// device (the staged host arrays of the C entry points, the batch's upload
// and download).
//
// A pageable cudaMemcpy moves 4 to 11 GB/s here: one thread copies through the
// driver's staging buffer, and on the way out it also takes the page faults of
// a fresh destination.  The link carries 50.  Here several threads take 2 MB
// pieces in turn, each through a pinned slot of its own on a stream of its
// own, so that the pieces on the link, the host copies and the page faults
// overlap: 99 MB into a fresh array 21 ms -> 5; first-order distance of a
// 200x256x256 host array (105 MB each way) 74 -> 52 ms a call.
// The slots (16 MB) are kept between calls; lsmgpu_release_scratch gives them
// back.  One copy uses them at a time; another that comes meanwhile, a small
// one, a capturing stream, and memory that is pinned already take the plain
// copy.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include <cstring>

#include "capi_common.h"

namespace lsmgpu {
namespace {

constexpr size_t kPiece = (size_t)2 << 20;
constexpr size_t kLeast = (size_t)8 << 20;   // below: the plain copy
constexpr int kSlots = 8;

struct Slots {
  std::mutex mu;
  int device = -1;               // of the streams; -1: nothing allocated
  char* pinned = nullptr;
  cudaStream_t stream[kSlots] = {};
  cudaEvent_t ready = nullptr;
} g_slots;

void drop_slots() {
  for (cudaStream_t& s : g_slots.stream) {
    if (s) cudaStreamDestroy(s);
    s = nullptr;
  }
  if (g_slots.ready) cudaEventDestroy(g_slots.ready);
  g_slots.ready = nullptr;
  if (g_slots.pinned) cudaFreeHost(g_slots.pinned);
  g_slots.pinned = nullptr;
  g_slots.device = -1;
  cudaGetLastError();
}

// the slots for `device`, or false (the caller holds the mutex)
bool have_slots(int device) {
  if (g_slots.device == device) return true;
  drop_slots();
  bool ok = cudaHostAlloc((void**)&g_slots.pinned, kSlots * kPiece, cudaHostAllocPortable) ==
                cudaSuccess &&
            cudaEventCreateWithFlags(&g_slots.ready, cudaEventDisableTiming) == cudaSuccess;
  for (int q = 0; ok && q < kSlots; q++)
    ok = cudaStreamCreateWithFlags(&g_slots.stream[q], cudaStreamNonBlocking) == cudaSuccess;
  if (!ok) {
    drop_slots();
    return false;
  }
  g_slots.device = device;
  return true;
}

bool pageable(const void* host) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

// behind the work on st: in pieces, complete on return, or plainly on st
cudaError_t copy(char* host, char* dev, size_t bytes, bool to_host, cudaStream_t st) {
  int device = 0;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  std::unique_lock<std::mutex> lock(g_slots.mu, std::defer_lock);
  if (bytes < kLeast || cudaGetDevice(&device) != cudaSuccess ||
      cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      !pageable(host) || !lock.try_lock() || !have_slots(device)) {
    cudaGetLastError();
    return to_host ? cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st)
                   : cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
  }
  cudaError_t e = cudaEventRecord(g_slots.ready, st);
  if (e != cudaSuccess) return e;
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  std::atomic<size_t> next{0};
  std::atomic<int> error{(int)cudaSuccess};
  auto work = [&](int q) {
    cudaStream_t s = g_slots.stream[q];
    char* slot = g_slots.pinned + q * kPiece;
    cudaError_t r = cudaSetDevice(device);
    if (r == cudaSuccess) r = cudaStreamWaitEvent(s, g_slots.ready, 0);
    while (r == cudaSuccess && error.load() == (int)cudaSuccess) {
      const size_t i = next.fetch_add(1);
      if (i >= pieces) return;
      const size_t off = i * kPiece, n = std::min(kPiece, bytes - off);
      if (!to_host) memcpy(slot, host + off, n);
      r = to_host ? cudaMemcpyAsync(slot, dev + off, n, cudaMemcpyDeviceToHost, s)
                  : cudaMemcpyAsync(dev + off, slot, n, cudaMemcpyHostToDevice, s);
      if (r == cudaSuccess) r = cudaStreamSynchronize(s);
      if (r == cudaSuccess && to_host) memcpy(host + off, slot, n);
    }
    if (r != cudaSuccess) error.store((int)r);
  };
  // the calling thread is one of the workers; fewer threads where no more
  // can be started
  const int hw = (int)std::thread::hardware_concurrency();
  const int workers = std::max(1, std::min({kSlots, hw, (int)std::min<size_t>(pieces, kSlots)}));
  std::vector<std::thread> threads;
  try {
    threads.reserve(workers);
    for (int q = 1; q < workers; q++) threads.emplace_back(work, q);
  } catch (...) {
  }
  work(0);
  for (std::thread& t : threads) t.join();
  return (cudaError_t)error.load();
}

}  // namespace

cudaError_t copy_to_host(void* host, const void* dev, size_t bytes, cudaStream_t st) {
  return copy((char*)host, (char*)dev, bytes, true, st);
}
cudaError_t copy_to_device(void* dev, const void* host, size_t bytes, cudaStream_t st) {
  return copy((char*)host, (char*)dev, bytes, false, st);
}

void release_copy_slots() {
  std::lock_guard<std::mutex> lock(g_slots.mu);
  drop_slots();
}

}  // namespace lsmgpu
