// result_slot.hpp -- scratch and result words of blocking probe calls.
//
// A blocking call needs the tile queue and status words of its kernel on the
// device and the match count on the host.  Allocating, zeroing, copying back
// and freeing them cost four API calls and two device operations per probe,
// more than the probe of a small batch.  A slot keeps both for one call at a
// time: the device words are zero between calls (the fused kernel clears them
// behind itself), and the host words are pinned and mapped, so the kernel
// writes its outcome there directly.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <vector>

namespace dtlg {

struct ResultSlot {
  void* dev = nullptr;                        // device scratch, zeroed
  unsigned long long* host = nullptr;         // pinned: [0] outcome word, [2..3] a copied workspace header
  unsigned long long* host_dev = nullptr;     // the same words, as the device sees them
  uint32_t ticket = 0;                        // of the slot's latest call
  bool fresh = true;                          // device scratch not zeroed yet
};

// The slots of one device: a call takes one and gives it back, so threads and
// streams never share one.  At most kMax exist; a call that finds none left
// (or cannot make one) goes without.
class ResultSlots {
 public:
  static constexpr int kMax = 16;

  ResultSlot* acquire(size_t dev_bytes) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (!free_.empty()) {
        ResultSlot* s = free_.back();
        free_.pop_back();
        return s;
      }
      if (made_ == kMax) return nullptr;
      made_++;
    }
    // allocations are no part of a capture that another thread may have open
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    ResultSlot* s = new ResultSlot();
    cudaError_t e = cudaMalloc(&s->dev, dev_bytes);
    if (e == cudaSuccess)
      e = cudaHostAlloc(reinterpret_cast<void**>(&s->host), 64, cudaHostAllocMapped | cudaHostAllocPortable);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&s->host_dev), s->host, 0);
    if (e == cudaSuccess) s->host[0] = 0;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
      cudaGetLastError();
      drop(s);
      return nullptr;
    }
    return s;
  }

  void release(ResultSlot* s) {
    std::lock_guard<std::mutex> lk(mu_);
    free_.push_back(s);
  }

  // A slot whose call failed: its kernel may never have run, or still run, so
  // it is not used again (freeing waits for the device).
  void drop(ResultSlot* s) {
    if (s->dev) cudaFree(s->dev);
    if (s->host) cudaFreeHost(s->host);
    delete s;
    std::lock_guard<std::mutex> lk(mu_);
    made_--;
  }

 private:
  std::mutex mu_;
  std::vector<ResultSlot*> free_;
  int made_ = 0;
};

}  // namespace dtlg
