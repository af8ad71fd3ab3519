"""Large host copies with two devices: the source that the library builds, on a
stand-in of the runtime that keeps host memory for device memory, knows which
device a stream, event or pointer belongs to, and refuses what the runtime
refuses (an event recorded on another device's stream)."""
import subprocess

import pytest

from lsmlib_b200 import build

HEADER = r"""
#include <cstddef>
#include <map>
struct CUstream_st { int device; };
struct CUevent_st { int device; };
extern thread_local int t_device;       // the thread's current device
extern thread_local bool t_main;        // the thread that calls the copies
extern int t_pinned, t_pinned_most, t_hosts, t_streams, t_set_main;
extern std::map<const char*, int> t_dev;   // "device" buffers: base -> device
extern size_t t_bytes;                  // of each
"""

RUNTIME = r"""
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include "fake.h"

thread_local int t_device = 0;
thread_local bool t_main = false;
int t_pinned = 0, t_pinned_most = 0, t_hosts = 0, t_streams = 0, t_set_main = 0;
std::map<const char*, int> t_dev;
size_t t_bytes;
static std::mutex t_mu;

extern "C" {
// (what nvcc's host code registers its device code with)
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}

cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (t_main) t_set_main++;
  t_device = d;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  std::lock_guard<std::mutex> l(t_mu);
  *p = std::malloc(n);
  t_hosts++;
  if (++t_pinned > t_pinned_most) t_pinned_most = t_pinned;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { t_pinned--; std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = new CUstream_st{t_device};
  t_streams++;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { t_streams--; delete s; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = new CUevent_st{t_device};
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return e->device == s->device ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  *a = cudaPointerAttributes{};
  a->type = cudaMemoryTypeUnregistered;
  for (auto& b : t_dev)
    if ((const char*)p >= b.first && (const char*)p < b.first + t_bytes) {
      a->type = cudaMemoryTypeDevice;
      a->device = b.second;
    }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
}
"""

PROGRAM = r"""
#include <cstdio>
#include "fake.h"
#include "host_copy.cu"

static int roundtrip(char* dev, cudaStream_t st, int seed) {
  std::vector<char> in(t_bytes), out(t_bytes, 0);
  for (size_t i = 0; i < t_bytes; i++) in[i] = (char)(i * 7 + (i >> 13) + seed);
  return lsmgpu::copy_to_device(dev, in.data(), t_bytes, st) == cudaSuccess &&
         lsmgpu::copy_to_host(out.data(), dev, t_bytes, st) == cudaSuccess && in == out;
}

int main() {
  t_main = true;
  t_bytes = ((size_t)8 << 20) + 4321;
  std::vector<char> a(t_bytes), b(t_bytes);
  t_dev[a.data()] = 0;
  t_dev[b.data()] = 1;
  CUstream_st s0{0}, s1{1};
  int ok = 1;
  // each device's slots once, however the devices alternate
  for (int q = 0; q < 4; q++) {
    t_device = 0;
    ok &= roundtrip(a.data(), &s0, q);
    t_device = 1;
    ok &= roundtrip(b.data(), &s1, q);
  }
  std::printf("alternating %d allocations %d\n", ok, t_hosts);
  // memory and stream of a device that is not the current one
  t_device = 1;
  const int other = roundtrip(a.data(), &s0, 9);
  // ... and a stream of another device than the memory's
  t_device = 0;
  const int mixed = roundtrip(a.data(), &s1, 10);
  std::printf("other device %d mixed %d device now %d set by the caller %d\n", other, mixed,
              t_device, t_set_main);
  lsmgpu::release_copy_slots();
  std::printf("left %d %d, most %d\n", t_pinned, t_streams, t_pinned_most);
  return 0;
}
"""


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    d = tmp_path_factory.mktemp("hostcopy")
    for name, text in (("fake.h", HEADER), ("fake.cpp", RUNTIME), ("main.cu", PROGRAM)):
        (d / name).write_text(text)
    exe = str(d / "t")
    subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "-O1", "-cudart", "none", "-I",
                                                build.CSRC, "-I", build.INCLUDE,
                                                str(d / "main.cu"), str(d / "fake.cpp"),
                                                "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout.splitlines()


def test_alternating_devices_keep_their_slots(report):
    assert report[0] == "alternating 1 allocations 2"


def test_another_device_than_the_current_one(report):
    assert report[1] == "other device 1 mixed 1 device now 0 set by the caller 0"


def test_release(report):
    assert report[2] == "left 0 0, most 2"
