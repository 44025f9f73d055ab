"""The pinned ring of large copies (csrc/staging.cu) on the host, with a stand-in for the CUDA calls it makes:
every length around a slot and the ring, no pinned memory, no events, a device reset between two copies."""
import os
import shutil
import subprocess


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ermod_openacc_b200", "csrc")

# "device" memory is host memory and every copy happens at once; pinned allocations are counted and can fail
FAKES = r"""
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
cudaError_t fk_host_alloc(void**, size_t, unsigned);
cudaError_t fk_free_host(void*);
cudaError_t fk_event_create(cudaEvent_t*, unsigned);
cudaError_t fk_event(cudaEvent_t);
cudaError_t fk_record(cudaEvent_t, cudaStream_t);
cudaError_t fk_copy(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t);
cudaError_t fk_sync(cudaStream_t);
cudaError_t fk_get_device(int*);
cudaError_t fk_set_device(int);
cudaError_t fk_last();
cudaError_t fk_entry(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*);
#define cudaHostAlloc fk_host_alloc
#define cudaFreeHost fk_free_host
#define cudaEventCreateWithFlags fk_event_create
#define cudaEventDestroy fk_event
#define cudaEventSynchronize fk_event
#define cudaEventRecord fk_record
#define cudaMemcpyAsync fk_copy
#define cudaStreamSynchronize fk_sync
#define cudaGetDevice fk_get_device
#define cudaSetDevice fk_set_device
#define cudaGetLastError fk_last
#define cudaGetDriverEntryPoint fk_entry
"""

MAIN = r"""
#include "fakes.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>
#include "engine.cuh"
extern "C" void ermod_staging_release(void);

static std::mutex mu;
static std::map<void*, unsigned long long> live;      // pinned allocations and their numbers
static unsigned long long next_id = 1;
static bool fail_pinned = false, fail_events = false;
static int frees_of_lost = 0, last = 0;
static void* at = nullptr;                            // a reset lets the next allocation take the same address

cudaError_t fk_host_alloc(void** p, size_t n, unsigned) {
  if (fail_pinned) { last = 2; return cudaErrorMemoryAllocation; }
  std::lock_guard<std::mutex> lk(mu);
  if (!at) at = malloc(n);
  *p = at;
  live[at] = next_id++;
  return cudaSuccess;
}
cudaError_t fk_free_host(void* p) {
  if (!live.count(p)) ++frees_of_lost;
  live.erase(p);
  return cudaSuccess;
}
cudaError_t fk_event_create(cudaEvent_t* e, unsigned) {
  if (fail_events) { *e = nullptr; last = 2; return cudaErrorMemoryAllocation; }
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t fk_event(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t fk_record(cudaEvent_t e, cudaStream_t) { return fk_event(e); }
cudaError_t fk_copy(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t fk_sync(cudaStream_t) { return cudaSuccess; }
cudaError_t fk_get_device(int* d) { *d = 0; return cudaSuccess; }
cudaError_t fk_set_device(int) { return cudaSuccess; }
cudaError_t fk_last() { const int e = last; last = 0; return (cudaError_t)e; }
static CUresult fk_attr(void* out, CUpointer_attribute a, CUdeviceptr p) {
  std::lock_guard<std::mutex> lk(mu);
  const auto it = live.find((void*)p);
  if (a != CU_POINTER_ATTRIBUTE_BUFFER_ID || it == live.end()) return CUDA_ERROR_INVALID_VALUE;
  *(unsigned long long*)out = it->second;
  return CUDA_SUCCESS;
}
cudaError_t fk_entry(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult*) {
  *f = (void*)fk_attr;
  return cudaSuccess;
}

static int bad = 0;
static void check(const char* what, bool ok) {
  if (!ok) { printf("FAILED: %s\n", what); bad = 1; }
}
static bool copies(size_t bytes, double q) {
  std::vector<double> a((bytes + 7) / 8), b(a.size(), -1.0), c(a.size(), -2.0);
  for (size_t i = 0; i < a.size(); ++i) a[i] = 0.1 + (double)i;
  bool ok = erm::staged_to_device(b.data(), a.data(), bytes, 0) == cudaSuccess && !memcmp(a.data(), b.data(), bytes);
  ok = ok && erm::staged_to_host(c.data(), a.data(), bytes, q, 0) == cudaSuccess;
  if (q == 0.0) return ok && !memcmp(a.data(), c.data(), bytes);
  for (size_t i = 0; i < bytes / 8; ++i) ok = ok && c[i] == a[i] / q;
  return ok;
}

int main() {
  const size_t slot = (size_t)1 << 20;
  for (size_t bytes : {(size_t)8, slot - 8, slot, slot + 8, 4 * slot, 11 * slot + 5, 12 * slot, 12 * slot + 8, 13 * slot,
                       31 * slot + 24})
    check("ring", copies(bytes, 0.0));
  check("one ring", live.size() == 1);
  live.clear();                                        // cudaDeviceReset
  check("after a reset", copies(5 * slot, 0.0) && live.size() == 1);
  live.clear();
  live[at] = next_id++;                                // a reset, and the address is another's now
  ermod_staging_release();
  check("another's memory is not freed", live.size() == 1);
  live.clear();
  check("a ring again", copies(3 * slot, 0.0) && live.size() == 1);
  ermod_staging_release();
  check("released", live.empty() && frees_of_lost == 0);
  ermod_staging_release();
  fail_pinned = true;
  check("no pinned memory", copies(5 * slot + 8, 0.0) && copies(2 * slot, 3.0) && last == 0);
  fail_pinned = false;
  fail_events = true;
  check("no events", copies(5 * slot + 8, 0.0) && copies(2 * slot, 3.0) && last == 0);
  fail_events = false;
  check("all well again", copies(5 * slot, 0.0));
  if (!bad) printf("ok\n");
  return bad;
}
"""


def test_ring_and_its_fallback(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "fakes.h").write_text(FAKES)
    (tmp_path / "main.cu").write_text(MAIN)
    exe = str(tmp_path / "staging")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-include", str(tmp_path / "fakes.h"),
                    "-I", CSRC, "-o", exe, str(tmp_path / "main.cu"), os.path.join(CSRC, "staging.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
