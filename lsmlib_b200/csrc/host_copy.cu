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
// The slots (16 MB for each device that copies) are kept between calls;
// lsmgpu_release_scratch gives them back.  One copy uses a device's slots at a
// time; another that comes meanwhile, a small one, a capturing stream, memory
// that is pinned already, and memory of a device that is not the calling
// thread's current one take the plain copy.
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
constexpr int kMaxDevices = 64;

struct Slots {
  std::mutex mu;
  char* pinned = nullptr;        // nullptr: nothing allocated
  cudaStream_t stream[kSlots] = {};
  cudaEvent_t ready = nullptr;
} g_slots[kMaxDevices];

void drop_slots(Slots& slots) {
  for (cudaStream_t& s : slots.stream) {
    if (s) cudaStreamDestroy(s);
    s = nullptr;
  }
  if (slots.ready) cudaEventDestroy(slots.ready);
  slots.ready = nullptr;
  if (slots.pinned) cudaFreeHost(slots.pinned);
  slots.pinned = nullptr;
  cudaGetLastError();
}

// The thread's allocations and waits here concern no capture of another
// thread, and must not be refused for its sake or invalidate it.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// the slots are there, or false; on their device (the caller holds the mutex)
bool have_slots(Slots& slots) {
  if (slots.pinned) return true;
  bool ok = cudaHostAlloc((void**)&slots.pinned, kSlots * kPiece, cudaHostAllocPortable) ==
                cudaSuccess &&
            cudaEventCreateWithFlags(&slots.ready, cudaEventDisableTiming) == cudaSuccess;
  for (int q = 0; ok && q < kSlots; q++)
    ok = cudaStreamCreateWithFlags(&slots.stream[q], cudaStreamNonBlocking) == cudaSuccess;
  if (!ok) drop_slots(slots);
  return ok;
}

// the current device, if it is the one that holds dev; else -1
int copying_device(const void* dev) {
  int device = -1;
  cudaPointerAttributes at;
  if (cudaGetDevice(&device) != cudaSuccess || device >= kMaxDevices ||
      cudaPointerGetAttributes(&at, dev) != cudaSuccess || at.type != cudaMemoryTypeDevice ||
      at.device != device)
    return -1;
  return device;
}

bool pageable(const void* host) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

// The pieces of one copy by several threads, behind the work on st; false if
// that work cannot be waited for (nothing copied then).
bool copy_pieces(Slots& slots, int device, char* host, char* dev, size_t bytes, bool to_host,
                 cudaStream_t st, cudaError_t* result) {
  if (cudaEventRecord(slots.ready, st) != cudaSuccess) return false;
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  std::atomic<size_t> next{0};
  std::atomic<int> error{(int)cudaSuccess};
  auto work = [&](int q) {
    RelaxedCapture relaxed;
    cudaStream_t s = slots.stream[q];
    char* slot = slots.pinned + q * kPiece;
    // (worker 0 is the calling thread, whose device it is)
    cudaError_t r = q == 0 ? cudaSuccess : cudaSetDevice(device);
    if (r == cudaSuccess) r = cudaStreamWaitEvent(s, slots.ready, 0);
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
  *result = (cudaError_t)error.load();
  return true;
}

// behind the work on st: in pieces, complete on return, or plainly on st
cudaError_t copy(char* host, char* dev, size_t bytes, bool to_host, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const int device = bytes < kLeast ? -1 : copying_device(dev);
  if (device >= 0 && cudaStreamIsCapturing(st, &cap) == cudaSuccess &&
      cap == cudaStreamCaptureStatusNone && pageable(host)) {
    RelaxedCapture relaxed;
    Slots& slots = g_slots[device];
    std::unique_lock<std::mutex> lock(slots.mu, std::try_to_lock);
    cudaError_t e = cudaSuccess;
    if (lock.owns_lock() && have_slots(slots) &&
        copy_pieces(slots, device, host, dev, bytes, to_host, st, &e))
      return e;
  }
  cudaGetLastError();
  return to_host ? cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st)
                 : cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
}

}  // namespace

cudaError_t copy_to_host(void* host, const void* dev, size_t bytes, cudaStream_t st) {
  return copy((char*)host, (char*)dev, bytes, true, st);
}
cudaError_t copy_to_device(void* dev, const void* host, size_t bytes, cudaStream_t st) {
  return copy((char*)host, (char*)dev, bytes, false, st);
}

void release_copy_slots() {
  for (Slots& slots : g_slots) {
    std::lock_guard<std::mutex> lock(slots.mu);
    if (slots.pinned) drop_slots(slots);
  }
}

}  // namespace lsmgpu
