"""slvfe's kept working memory (csrc/workspace.cuh) on the host, with a stand-in for the CUDA calls it makes."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ermod_openacc_b200", "csrc")

MAIN = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <map>
static std::map<void*, size_t> live;                  // allocations and their sizes
static int device = 3, streams = 0, mallocs = 0;
static size_t room = (size_t)1 << 40;                 // bytes that may be live
static cudaError_t fk_malloc(void** p, size_t n) {
  size_t used = 0;
  for (auto& a : live) used += a.second;
  if (used + n > room) return cudaErrorMemoryAllocation;
  *p = new char;
  live[*p] = n;
  ++mallocs;
  return cudaSuccess;
}
static cudaError_t fk_free(void* p) { return live.erase(p) ? cudaSuccess : cudaErrorInvalidValue; }
static cudaError_t fk_stream(cudaStream_t* s, unsigned) { *s = (cudaStream_t)1; ++streams; return cudaSuccess; }
static cudaError_t fk_end(cudaStream_t) { --streams; return cudaSuccess; }
static cudaError_t fk_get(int* d) { *d = device; return cudaSuccess; }
static cudaError_t fk_set(int d) { device = d; return cudaSuccess; }
static cudaError_t fk_last() { return cudaSuccess; }
#define cudaMalloc fk_malloc
#define cudaFree fk_free
#define cudaStreamCreateWithFlags fk_stream
#define cudaStreamDestroy fk_end
#define cudaGetDevice fk_get
#define cudaSetDevice fk_set
#define cudaGetLastError fk_last
#include "workspace.cuh"
unsigned long long erm::allocation_id(const void* p) { return live.count((void*)p) ? (unsigned long long)p : 0; }

static int bad = 0;
static void check(const char* what, bool ok) {
  if (!ok) { printf("FAILED: %s\n", what); bad = 1; }
}
static erm::WorkspaceCache c;
static size_t call(int dev, size_t need, bool clean = true) {   // one call; the size that it was given
  erm::Workspace w;
  device = dev;
  if (!c.take(dev, need, w)) return 0;
  const size_t got = w.bytes;
  c.give(w, clean);
  check("handed over", w.p == nullptr && w.st == nullptr);
  return got;
}

int main() {
  const size_t MB = (size_t)1 << 20;
  erm::Workspace a, b;
  check("two at a time", c.take(0, 10 * MB, a) && c.take(0, 20 * MB, b));
  c.give(a, true);
  c.give(b, true);
  check("the smallest that fits", call(0, 5 * MB) == 10 * MB && call(0, 15 * MB) == 20 * MB && mallocs == 2);
  check("a larger size", call(0, 100 * MB) == 100 * MB && mallocs == 3);
  check("is kept in place of the smallest", call(0, 90 * MB) == 100 * MB && mallocs == 3 && live.size() == 2);
  check("and the larger of the others", call(0, 20 * MB) == 20 * MB && mallocs == 3);
  check("a smaller one is not", c.take(0, 100 * MB, a) && c.take(0, 20 * MB, b));
  erm::Workspace d;
  check("third", c.take(0, 1 * MB, d));
  c.give(a, true);
  c.give(b, true);
  c.give(d, true);
  check("two kept", live.size() == 2 && call(0, 1 * MB) == 20 * MB);
  check("above the bound", call(0, 300 * MB) == 300 * MB && live.size() == 2);
  check("after an error", call(0, 60 * MB, false) == 100 * MB && live.size() == 1);
  check("each device its own", call(1, 30 * MB) == 30 * MB && call(0, 30 * MB) == 30 * MB && live.size() == 3);
  room = 70 * MB;                                      // 20 + 30 MB of device 0 and 30 MB of device 1 are kept
  check("no memory: the device's kept ones go", call(0, 40 * MB) == 40 * MB && live.size() == 2);
  check("none at all", call(0, 80 * MB) == 0 && streams == 1 && live.size() == 1);
  room = (size_t)1 << 40;
  call(0, 50 * MB);
  live.clear();                                        // cudaDeviceReset
  mallocs = 0;
  check("after a reset", call(0, 50 * MB) == 50 * MB && mallocs == 1 && live.size() == 1);
  device = 3;
  c.release();
  check("released, the caller's device as it was", live.empty() && device == 3);
  if (!bad) printf("ok\n");
  return bad;
}
"""


def test_kept_workspaces(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = tmp_path / "main.cu"
    src.write_text(MAIN)
    exe = str(tmp_path / "ws")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-I", CSRC, "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
