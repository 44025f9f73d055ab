// staging.cu -- large copies between the device and ordinary (pageable) host memory.
//
// The runtime's own copy of pageable memory runs through one host thread: 15.6 MB (the ermax^2
// correlation matrix of the default mesh) took 0.88 ms either way, against 0.30 ms for the same
// bytes to or from pinned memory, and engstore then divided them on the host in another 1.1 ms.
// Here the bytes pass through a ring of pinned slots; up to kWorkers threads move them between the
// ring and the caller's memory (where first touches of fresh pages are then shared out too) while
// the next slots are in flight, and engstore's division runs on the device, in the kernel that
// writes the slot.  A division's engstore at 1396 bins, with the small accumulators in one copy: 4.0 ->
// 0.9 ms.  Where the ring cannot be had, the runtime's own copy does.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "engine.cuh"

namespace erm {
namespace {

constexpr size_t kSlotBytes = (size_t)1 << 20;
constexpr int kSlots = 12, kWorkers = 4;       // kSlots: a multiple of every worker count up to kWorkers

// one ring a process (12 MB), made on first use; a copy holds the lock until its last byte has moved
std::mutex g_mu;
unsigned char* g_ring = nullptr;
unsigned long long g_ring_id = 0;              // its allocation_id: a host's cudaDeviceReset frees the ring

// out = in / q, FP64 quotients as the host forms them
__global__ void k_divide(size_t n, const double* __restrict__ in, double q, double* __restrict__ out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = in[i] / q;
}

struct Copy {
  unsigned char* host;
  unsigned char* dev;
  size_t bytes;
  bool to_host;
  double q;              // to the host: divide FP64 values by this (0: copy the bytes)
  cudaStream_t s;
};

// the copy without the ring
cudaError_t direct(const Copy& cp) {
  cudaError_t e = cp.to_host ? cudaMemcpyAsync(cp.host, cp.dev, cp.bytes, cudaMemcpyDeviceToHost, cp.s)
                             : cudaMemcpyAsync(cp.dev, cp.host, cp.bytes, cudaMemcpyHostToDevice, cp.s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cp.s);
  if (e == cudaSuccess && cp.q != 0.0)
    for (size_t i = 0; i < cp.bytes / sizeof(double); ++i) ((double*)cp.host)[i] /= cp.q;
  return e;
}

bool have_ring() {
  if (g_ring && allocation_id(g_ring) != g_ring_id) g_ring = nullptr;
  if (g_ring) return true;
  if (cudaHostAlloc((void**)&g_ring, kSlotBytes * kSlots, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_ring = nullptr;
    return false;
  }
  g_ring_id = allocation_id(g_ring);
  if (g_ring_id != 0) return true;
  cudaFreeHost(g_ring);
  g_ring = nullptr;
  return false;
}

cudaError_t run(const Copy& cp) {
  std::unique_lock<std::mutex> lk(g_mu);
  const int n = (int)((cp.bytes + kSlotBytes - 1) / kSlotBytes);
  std::vector<std::atomic<int>> moved;          // to the host: copied out of its slot
  std::vector<std::thread> pool;
  try {
    moved = std::vector<std::atomic<int>>(n);
    pool.reserve(kWorkers);
  } catch (...) {
    lk.unlock();
    return direct(cp);
  }
  cudaEvent_t ev[kSlots] = {};
  bool ready = have_ring();
  for (auto& e : ev) ready = ready && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ready) {
    cudaGetLastError();
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    lk.unlock();
    return direct(cp);
  }
  int device = 0;
  cudaGetDevice(&device);
  const int nw = std::max(1, std::min({kWorkers, n, (int)std::thread::hardware_concurrency()}));
  std::atomic<int> err{(int)cudaSuccess};
  std::atomic<int> queued{0};                   // to the host: slots whose device work is in the stream
  for (auto& m : moved) m.store(0);
  auto note = [&](cudaError_t e) { if (e != cudaSuccess) err.store((int)e); return e == cudaSuccess; };
  auto part = [&](int c) { return std::min(kSlotBytes, cp.bytes - (size_t)c * kSlotBytes); };
  auto slot = [&](int c) { return g_ring + (size_t)(c % kSlots) * kSlotBytes; };
  auto queue_out = [&](int c) {                 // device to slot
    const size_t b = part(c);
    if (cp.q != 0.0) {
      k_divide<<<64, 256, 0, cp.s>>>(b / sizeof(double), (const double*)(cp.dev + (size_t)c * kSlotBytes), cp.q,
                                     (double*)slot(c));
      note(cudaGetLastError());
    } else {
      note(cudaMemcpyAsync(slot(c), cp.dev + (size_t)c * kSlotBytes, b, cudaMemcpyDeviceToHost, cp.s));
    }
    note(cudaEventRecord(ev[c % kSlots], cp.s));
  };
  auto worker = [&](int w) {
    cudaSetDevice(device);
    for (int c = w; c < n; c += nw) {
      if (cp.to_host) {
        while (queued.load(std::memory_order_acquire) <= c) std::this_thread::yield();
        note(cudaEventSynchronize(ev[c % kSlots]));
        std::memcpy(cp.host + (size_t)c * kSlotBytes, slot(c), part(c));
        moved[c].store(1, std::memory_order_release);
      } else {
        // a slot's earlier copy was queued by the same worker (kSlots is a multiple of nw)
        if (c >= kSlots) note(cudaEventSynchronize(ev[c % kSlots]));
        std::memcpy(slot(c), cp.host + (size_t)c * kSlotBytes, part(c));
        note(cudaMemcpyAsync(cp.dev + (size_t)c * kSlotBytes, slot(c), part(c), cudaMemcpyHostToDevice, cp.s));
        note(cudaEventRecord(ev[c % kSlots], cp.s));
      }
    }
  };
  for (int w = cp.to_host ? 0 : 1; w < nw; ++w) {
    try {
      pool.emplace_back(worker, w);
    } catch (...) {                             // no thread to be had: its share falls to this one, below
      break;
    }
  }
  const int started = (int)pool.size() + (cp.to_host ? 0 : 1);
  if (cp.to_host) {
    // slots in order; one that is still being emptied by a worker is waited for, one whose worker
    // did not start is emptied here
    for (int c = 0; c < n; ++c) {
      if (c >= kSlots) {
        const int o = c - kSlots;
        while (o % nw < started && !moved[o].load(std::memory_order_acquire)) std::this_thread::yield();
      }
      queue_out(c);
      queued.store(c + 1, std::memory_order_release);
      if (c % nw >= started) {
        note(cudaEventSynchronize(ev[c % kSlots]));
        std::memcpy(cp.host + (size_t)c * kSlotBytes, slot(c), part(c));
        moved[c].store(1, std::memory_order_release);
      }
    }
  } else {
    worker(0);
    for (int w = started; w < nw; ++w) worker(w);
  }
  for (auto& t : pool) t.join();
  note(cudaStreamSynchronize(cp.s));            // the ring is the next copy's
  for (auto& e : ev) cudaEventDestroy(e);
  return (cudaError_t)err.load();
}

}  // namespace

unsigned long long allocation_id(const void* p) {
  using Query = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
  static std::atomic<Query> query{nullptr};
  Query f = query.load();
  if (!f) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &sym, cudaEnableDefault, &found) != cudaSuccess || !sym) {
      cudaGetLastError();
      return 0;
    }
    f = (Query)sym;
    query.store(f);
  }
  unsigned long long id = 0;
  return f(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, (CUdeviceptr)p) == CUDA_SUCCESS ? id : 0;
}

cudaError_t staged_to_host(void* dst, const void* src, size_t bytes, double q, cudaStream_t s) {
  return run(Copy{(unsigned char*)dst, (unsigned char*)src, bytes, true, q, s});
}
cudaError_t staged_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  return run(Copy{(unsigned char*)src, (unsigned char*)dst, bytes, false, 0.0, s});
}

}  // namespace erm

extern "C" void ermod_staging_release(void) {
  std::lock_guard<std::mutex> lk(erm::g_mu);
  if (erm::g_ring && erm::allocation_id(erm::g_ring) == erm::g_ring_id) cudaFreeHost(erm::g_ring);
  erm::g_ring = nullptr;
}
