"""The host arrays of Action-, NodeModel- and estimator-level calls (csrc/entry_io.h)
against a fake of the CUDA calls: every call leaves with the stream idle, one that
fails half-way too, whose blocks the next call overwrites."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

// ---- the fake: copies are queued, and done (or found undone) later
typedef int cudaError_t;
typedef int cudaStream_t;
enum { cudaSuccess = 0, cudaErrorFake = 2, cudaHostAllocMapped = 0 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
static int queued, synced, freed_async, fail_copy = -1, fail_malloc;
static cudaError_t cudaGetLastError() { return 0; }
static const char* cudaGetErrorString(cudaError_t) { return "fake"; }
static cudaError_t cudaStreamSynchronize(cudaStream_t) { queued = 0; ++synced; return 0; }
template <class T> static cudaError_t cudaMalloc(T** p, size_t n) {
  if (fail_malloc) return cudaErrorFake;
  *p = (T*)malloc(n);
  return 0;
}
static cudaError_t cudaFree(void* p) { free(p); return 0; }
static cudaError_t cudaHostAlloc(void** p, size_t n, int) { *p = malloc(n); return 0; }
static cudaError_t cudaFreeHost(void* p) { free(p); return 0; }
template <class T> static cudaError_t cudaMallocAsync(T** p, size_t n, cudaStream_t) {
  *p = (T*)malloc(n);
  return 0;
}
static cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  if (queued) freed_async += 100;  // freed under queued work
  free(p);
  ++freed_async;
  return 0;
}
static cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fail_copy-- == 0) return cudaErrorFake;
  memcpy(d, s, n);
  ++queued;
  return 0;
}
static cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  memset(p, v, n);
  ++queued;
  return 0;
}
enum { PIMC_OK = 0, PIMC_ERR_CUDA = -3 };
static int fail(int code, const std::string&) { return code; }
#define CU(call)                                        \
  do {                                                  \
    if ((call) != cudaSuccess) return fail(PIMC_ERR_CUDA, #call); \
  } while (0)
template <class T> struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  int alloc(size_t c) {
    free();
    n = c;
    if (cudaMalloc(&p, c * sizeof(T)) != cudaSuccess) { p = nullptr; n = 0; return -1; }
    return 0;
  }
  void free() { if (p) cudaFree(p); p = nullptr; n = 0; }
};
#include "entry_io.h"

// a call: bytes in and out, and where it gives up (0: nowhere, 1: after open, as when a
// launch fails)
static int call(IoBlocks& b, size_t bytes, int stop, std::vector<char>& in, std::vector<char>& out) {
  in.assign(bytes, 7);
  out.assign(bytes, 1);
  EntryIo io(b, 0);
  const int i = io.in(in.data(), bytes), o = io.out(out.data(), bytes, true);
  const int t = io.in_device(in.data(), 64);
  if (int rc = io.open()) return rc;
  ++queued;  // the kernel
  if (stop) return PIMC_ERR_CUDA;
  memcpy(io.dev<char>(o), io.dev<char>(i), bytes);
  (void)t;
  return io.close();
}

int main() {
  int bad = 0;
  const auto expect = [&](bool ok, const char* what) { if (!ok) { std::printf("%s\n", what); ++bad; } };
  std::vector<char> in, out;
  for (size_t bytes : {size_t(1000), size_t(1) << 20, size_t(80) << 20}) {
    IoBlocks b;
    synced = 0;
    expect(call(b, bytes, 0, in, out) == PIMC_OK && out == in, "results");
    expect(queued == 0, "work queued after a call");
    expect(synced == 1 + (bytes == 1000 || bytes == (1 << 20)), "a second wait");  // (the block grew)
    expect(call(b, bytes, 1, in, out) == PIMC_ERR_CUDA, "the error");
    expect(queued == 0, "work queued after a launch that failed");
    for (int k = 0; k < 3; ++k) {  // the k-th copy fails
      fail_copy = k;
      const int rc = call(b, bytes, 0, in, out);
      expect(fail_copy >= 0 || rc == PIMC_ERR_CUDA, "the copy's error");
      fail_copy = -1;
      expect(queued == 0, "work queued after a copy that failed");
    }
    expect(b.mutex.try_lock(), "the mutex is held");
    b.mutex.unlock();
    expect(call(b, bytes, 0, in, out) == PIMC_OK && out == in, "results after errors");
    b.free();
    fail_malloc = 1;
    if (bytes == 1 << 20) expect(call(b, bytes, 0, in, out) == PIMC_ERR_CUDA, "no memory");
    fail_malloc = 0;
    b.free();
  }
  expect(freed_async > 0 && freed_async < 100, "memory freed under queued work");
  return bad;
}
"""


def test_calls_leave_the_stream_idle(tmp_path):
    src, exe = tmp_path / "io.cc", tmp_path / "io"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I",
                    os.path.join(REPO, "pi-qmc_gb300", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
