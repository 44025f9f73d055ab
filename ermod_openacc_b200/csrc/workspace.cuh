// workspace.cuh -- working memory of a call, kept for the next one.
//
// An allocation of a free energy's size (60 to 250 MB) with its release takes 0.7 ms, now and then
// several.  At most kKeep buffers are kept for a device, the largest that came back, none above
// kKeepBytes.  They are taken out under the lock, so that calls from several threads have one each.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <utility>
#include <vector>

namespace erm {

unsigned long long allocation_id(const void* p);   // staging.cu

struct Workspace {
  int device = -1;
  unsigned char* p = nullptr;
  unsigned long long id = 0;      // p's allocation_id
  size_t bytes = 0;
  cudaStream_t st = nullptr;
};

class WorkspaceCache {
 public:
  static constexpr size_t kKeepBytes = (size_t)256 << 20;
  static constexpr int kKeep = 2;

  // A workspace of at least `need` bytes on the current device, `device`: the smallest kept one that
  // fits, else a new one, for which the device's kept ones are given back where memory is short.
  bool take(int device, size_t need, Workspace& w) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      forget_lost();
      size_t best = kept_.size();
      for (size_t i = 0; i < kept_.size(); ++i)
        if (kept_[i].device == device && kept_[i].bytes >= need && (best == kept_.size() || kept_[i].bytes < kept_[best].bytes))
          best = i;
      if (best < kept_.size()) {
        w = kept_[best];
        kept_.erase(kept_.begin() + best);
        return true;
      }
    }
    if (make(device, need, w)) return true;
    free_kept(device);
    return make(device, need, w);
  }

  // `clean`: the call ended without a CUDA error, its stream is idle
  void give(Workspace& w, bool clean) {
    if (clean && w.bytes <= kKeepBytes && w.id != 0) {
      std::lock_guard<std::mutex> lk(mu_);
      int n = 0;
      Workspace* least = nullptr;
      for (Workspace& o : kept_)
        if (o.device == w.device) {
          ++n;
          if (!least || o.bytes < least->bytes) least = &o;
        }
      if (n < kKeep) {
        try {
          kept_.push_back(w);
          w = Workspace();
        } catch (...) {             // no room to note it: freed below
        }
      } else if (least->bytes < w.bytes) {
        std::swap(*least, w);       // the smaller one goes
        if (lost(w)) w = Workspace();
      }
    }
    free(w);
  }

  void release() {
    int device = 0;
    const bool had = cudaGetDevice(&device) == cudaSuccess;
    free_kept(-1);
    if (had) cudaSetDevice(device);
  }

 private:
  static bool lost(const Workspace& w) { return allocation_id(w.p) != w.id; }

  static void free(Workspace& w) {
    if (w.p) cudaFree(w.p);
    if (w.st) cudaStreamDestroy(w.st);
    w = Workspace();
  }

  static bool make(int device, size_t need, Workspace& w) {
    w.device = device;
    w.bytes = need;
    if (cudaStreamCreateWithFlags(&w.st, cudaStreamNonBlocking) == cudaSuccess &&
        cudaMalloc((void**)&w.p, need) == cudaSuccess) {
      w.id = allocation_id(w.p);
      return true;
    }
    cudaGetLastError();
    free(w);
    return false;
  }

  // those that a device reset has freed, streams and all
  void forget_lost() {
    for (size_t i = 0; i < kept_.size();)
      if (lost(kept_[i])) kept_.erase(kept_.begin() + i);
      else ++i;
  }

  // every kept one of `device` (-1: of all)
  void free_kept(int device) {
    std::lock_guard<std::mutex> lk(mu_);
    forget_lost();
    for (size_t i = 0; i < kept_.size();)
      if (device < 0 || kept_[i].device == device) {
        cudaSetDevice(kept_[i].device);
        free(kept_[i]);
        kept_.erase(kept_.begin() + i);
      } else {
        ++i;
      }
  }

  std::mutex mu_;
  std::vector<Workspace> kept_;
};

}  // namespace erm
