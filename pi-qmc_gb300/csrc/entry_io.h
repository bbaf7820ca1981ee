// Host arrays of the calls that take or return them (a part of engine.cu, apart so that
// it can be compiled against a fake of the CUDA calls: fail, CU, DevBuf and the CUDA
// runtime's declarations come before it).
#pragma once
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

// An engine's blocks for them.
struct IoBlocks {
  std::mutex mutex;
  DevBuf<char> dev;
  char* host = nullptr;
  void free() {
    dev.free();
    if (host) cudaFreeHost(host);
    host = nullptr;
  }
};

// The arrays of one call between the caller's memory and the device.  A call names
// its inputs, outputs and scratch, open() places them, dev() gives their device
// addresses, and close() waits for the stream and delivers the outputs.  Small calls
// (kIoMapped of inputs and outputs) run on a pinned host block of the engine that the
// kernels read and write themselves: no copies are queued.  Larger ones copy from
// and to the caller's memory through a device block, kept up to kIoKeep.  (Allocated
// from the stream's pool in each call, which gives its memory back at every
// synchronisation: a node evaluation of one pair took 275 us, now 61.)  The engine's
// blocks serve one call at a time: a call holds the engine's mutex, and leaves with
// the stream idle, after an error too.
constexpr size_t kIoMapped = 128 << 10, kIoKeep = 64 << 20;

class EntryIo {
 public:
  EntryIo(IoBlocks& blocks, cudaStream_t stream)
      : blocks_(blocks), stream_(stream), lock_(blocks.mutex) {}
  ~EntryIo() {
    // (a call that gives up between open and the end of close may have work queued that
    // uses the blocks and the caller's arrays)
    if (queued_) cudaStreamSynchronize(stream_);
    if (own_) cudaFreeAsync(own_, stream_);
  }
  int in(const void* p, size_t bytes) { return add(const_cast<void*>(p), bytes, kIn); }
  // (a table that every CTA reads: to device memory in either case)
  int in_device(const void* p, size_t bytes) { return add(const_cast<void*>(p), bytes, kInDevice); }
  int out(void* p, size_t bytes, bool zeroed = false) {
    return add(p, bytes, zeroed ? kOutZero : kOut);
  }
  int scratch(size_t bytes) { return add(nullptr, bytes, kScratch); }
  int open() {
    queued_ = true;
    size_t io = 0, tmp = 0;
    for (const Part& p : parts_) (p.kind >= kInDevice ? tmp : io) += p.bytes;
    mapped_ = io <= kIoMapped;
    if (mapped_ && !blocks_.host &&
        cudaHostAlloc((void**)&blocks_.host, kIoMapped, cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      blocks_.host = nullptr;
      mapped_ = false;
    }
    const size_t need = tmp + (mapped_ ? 0 : io);
    char* dev = nullptr;
    if (need > kIoKeep) {
      CU(cudaMallocAsync(&own_, need, stream_));
      dev = own_;
    } else if (need) {
      if (blocks_.dev.n < need) {
        CU(cudaStreamSynchronize(stream_));
        if (blocks_.dev.alloc(std::min(kIoKeep, std::max<size_t>(2 * blocks_.dev.n, need))))
          return fail(PIMC_ERR_CUDA, "cudaMalloc call buffers");
      }
      dev = blocks_.dev.p;
    }
    size_t hoff = 0, doff = 0;
    for (Part& p : parts_) {
      const bool on_host = mapped_ && p.kind < kInDevice;
      size_t& off = on_host ? hoff : doff;
      p.dev = (on_host ? blocks_.host : dev) + off;
      off += p.bytes;
      if (mapped_ && p.kind == kIn) memcpy(p.dev, p.host, p.size);
      if (mapped_ && p.kind == kOutZero) memset(p.dev, 0, p.size);
      if (((!mapped_ && p.kind == kIn) || p.kind == kInDevice) && p.size)
        CU(cudaMemcpyAsync(p.dev, p.host, p.size, cudaMemcpyHostToDevice, stream_));
      if (!mapped_ && p.kind == kOutZero) CU(cudaMemsetAsync(p.dev, 0, p.size, stream_));
    }
    return PIMC_OK;
  }
  template <class T>
  T* dev(int k) const {
    return (T*)parts_[k].dev;
  }
  int close() {
    if (!mapped_)
      for (const Part& p : parts_)
        if (p.kind == kOut || p.kind == kOutZero)
          CU(cudaMemcpyAsync(p.host, p.dev, p.size, cudaMemcpyDeviceToHost, stream_));
    CU(cudaStreamSynchronize(stream_));
    queued_ = false;
    if (mapped_)
      for (const Part& p : parts_)
        if (p.kind == kOut || p.kind == kOutZero) memcpy(p.host, p.dev, p.size);
    return PIMC_OK;
  }

 private:
  enum Kind { kIn, kOut, kOutZero, kInDevice, kScratch };
  struct Part {
    void* host;
    size_t size, bytes;  // bytes: rounded up, so that the next part stays aligned
    Kind kind;
    char* dev;
  };
  int add(void* p, size_t size, Kind kind) {
    parts_.push_back({p, size, (size + 255) & ~(size_t)255, kind, nullptr});
    return (int)parts_.size() - 1;
  }
  IoBlocks& blocks_;
  cudaStream_t stream_;
  std::lock_guard<std::mutex> lock_;
  std::vector<Part> parts_;
  char* own_ = nullptr;
  bool mapped_ = false, queued_ = false;
};
