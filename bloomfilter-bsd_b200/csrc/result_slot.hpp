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

namespace dtlg {

struct ResultSlot {
  void* dev = nullptr;                        // device scratch, zeroed
  unsigned long long* host = nullptr;         // pinned: [0] outcome word, [2..3] a copied workspace header
  unsigned long long* host_dev = nullptr;     // the same words, as the device sees them
  uint32_t ticket = 0;                        // of the slot's latest call
  bool fresh = true;                          // device scratch not zeroed yet
  bool made = false;                          // in use or free, not dropped
};

// The slots of one device: a call takes one and gives it back, so threads and
// streams never share one.  At most kMax exist; a call that finds none left
// (or cannot make one) goes without.  The bookkeeping has a fixed size, so that
// nothing here throws: the callers are C entry points.
class ResultSlots {
 public:
  static constexpr int kMax = 16;

  ResultSlot* acquire(size_t dev_bytes) noexcept {
    ResultSlot* s = nullptr;
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (n_free_ != 0) return free_[--n_free_];
      for (ResultSlot& c : slots_) {
        if (!c.made) {
          c = ResultSlot{};
          c.made = true;
          s = &c;
          break;
        }
      }
    }
    if (!s) return nullptr;
    RelaxedCapture relaxed;
    cudaError_t e = cudaMalloc(&s->dev, dev_bytes);
    if (e == cudaSuccess)
      e = cudaHostAlloc(reinterpret_cast<void**>(&s->host), 64, cudaHostAllocMapped | cudaHostAllocPortable);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&s->host_dev), s->host, 0);
    if (e != cudaSuccess) {
      cudaGetLastError();
      drop(s);
      return nullptr;
    }
    s->host[0] = 0;
    return s;
  }

  void release(ResultSlot* s) noexcept {
    std::lock_guard<std::mutex> lk(mu_);
    free_[n_free_++] = s;
  }

  // A slot whose call failed: its kernel may never have run, or still run, so
  // it is not used again (freeing waits for the device).
  void drop(ResultSlot* s) noexcept {
    RelaxedCapture relaxed;
    if (s->dev) cudaFree(s->dev);
    if (s->host) cudaFreeHost(s->host);
    std::lock_guard<std::mutex> lk(mu_);
    s->made = false;
  }

 private:
  // Allocating and freeing are no part of a capture that another thread may
  // have open, and would end it in the default mode.
  struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };

  std::mutex mu_;
  ResultSlot slots_[kMax];
  ResultSlot* free_[kMax] = {};
  int n_free_ = 0;
};

}  // namespace dtlg
