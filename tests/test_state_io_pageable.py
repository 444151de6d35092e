"""State transfers where page-locked memory or threads cannot be had: the
library's own source, compiled for the host with an allocator or threads that
always fail and device memory played by host memory, must still move every
value."""
import subprocess

import pytest

from fall3d_b200 import build as B

HARNESS = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include <vector>
static int pins = 0;
static cudaError_t no_pin(void**, size_t) { ++pins; return cudaErrorMemoryAllocation; }
static cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
static cudaError_t fine() { return cudaSuccess; }
static cudaError_t attributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
#define cudaMallocHost no_pin
#define cudaMemcpyAsync copy
#define cudaPointerGetAttributes attributes
#define cudaStreamSynchronize(st) fine()
#define cudaSetDevice(d) fine()
#define cudaGetLastError() fine()
#include "state_io.cu"
using namespace f3d;

// the interior and the two-deep face ghosts, everything else as it was
static int wrong(const RowsOut& r, const std::vector<double>& host, const std::vector<double>& v) {
  int bad = 0;
  const bool halo = r.X != r.nx;
  const long long h = halo ? 2 : 0, hz = r.Z != r.nz ? 2 : 0;
  for (long long b = 0; b < r.nb; ++b)
    for (long long k = 0; k < r.Z; ++k)
      for (long long j = 0; j < r.Y; ++j)
        for (long long i = 0; i < r.X; ++i) {
          const long long q[3] = {i - h, j - h, k - hz}, n[3] = {r.nx, r.ny, r.nz};
          long long at[3], out = 0;
          for (int d = 0; d < 3; ++d) {
            out += q[d] < 0 || q[d] >= n[d];
            at[d] = q[d] < 0 ? 0 : q[d] >= n[d] ? n[d] - 1 : q[d];
          }
          const bool set = out == 0 || (out == 1 && r.faces);
          const double want = set ? v[((b * r.nz + at[2]) * r.ny + at[1]) * r.nx + at[0]] : -7.0;
          bad += host[((b * r.Z + k) * r.Y + j) * r.X + i] != want;
        }
  return bad;
}

int main() {
  int bad = 0;
  const long long shapes[][4] = {{5, 3, 2, 1}, {131, 70, 33, 5}, {200001, 2, 1, 1}};
  for (auto& s : shapes)
    for (int form = 0; form < 3; ++form) {
      const long long nx = s[0], ny = s[1], nz = s[2], nb = s[3], n = nx * ny * nz * nb;
      std::vector<double> c64(n), v(n);
      std::vector<float> hi(n), lo(n);
      for (long long q = 0; q < n; ++q) {
        c64[q] = 1.0 / (q + 3);
        hi[q] = (float)c64[q];
        lo[q] = (float)(c64[q] - hi[q]);
        v[q] = form == 0 ? c64[q] : form == 1 ? (double)hi[q] : (double)hi[q] + (double)lo[q];
      }
      MemberDev m{};
      m.nx = (int)nx; m.ny = (int)ny; m.nz = (int)nz; m.nb = (int)nb;
      if (form == 0) m.c64 = c64.data();
      else m.c32 = hi.data();
      if (form == 2) m.c32lo = lo.data();
      std::vector<double> host((nx + 4) * (ny + 4) * (nz + 4) * nb, -7.0);
      StateIO io;
      const RowsOut r = rows3d(m, host.data(), true);
      bad += io.download(r, 0, nullptr) != cudaSuccess;
      bad += wrong(r, host, v);
      if (form == 0) {
        std::vector<double> a((nx + 4) * (ny + 4) * nb, -7.0), up(n, 0.0);
        const RowsOut r2 = rows2d(c64.data(), nx, ny, nb, a.data());
        bad += io.download(r2, 0, nullptr) != cudaSuccess;
        std::vector<double> v2(v.begin(), v.begin() + nx * ny * nb);
        bad += wrong(r2, a, v2);
        bad += io.upload(up.data(), c64.data(), n * 8, 0, nullptr) != cudaSuccess;
        bad += up != c64;
      }
    }
  printf("pins %d bad %d\n", pins, bad);
  return bad != 0 || pins == 0;
}
"""


THREADS = r"""
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>
#include <vector>
static cudaError_t pin(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
static cudaError_t unpin(void* p) { free(p); return cudaSuccess; }
static cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
static cudaError_t event(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
static cudaError_t fine() { return cudaSuccess; }
static cudaError_t attributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
namespace std {
struct no_thread {  // starts once, then finds no memory
  static inline int made = 0;
  std::thread t;
  no_thread() = default;
  template <class F>
  explicit no_thread(F f) {
    if (made++) throw std::bad_alloc();
    t = std::thread(f);
  }
  void join() { t.join(); }
};
}
#define cudaMallocHost pin
#define cudaFreeHost unpin
#define cudaMemcpyAsync copy
#define cudaPointerGetAttributes attributes
#define cudaEventCreateWithFlags event
#define cudaEventDestroy(e) fine()
#define cudaEventRecord(e, st) fine()
#define cudaEventSynchronize(e) fine()
#define cudaStreamSynchronize(st) fine()
#define cudaSetDevice(d) fine()
#define thread no_thread
#include "state_io.cu"

int main() {
  std::vector<char> a(20000003), b(a.size(), 0);
  for (size_t q = 0; q < a.size(); ++q) a[q] = (char)(q * 2654435761u >> 13);
  f3d::StateIO io;
  const bool ok = io.upload(b.data(), a.data(), a.size(), 0, nullptr) == cudaSuccess && a == b;
  return ok && std::no_thread::made == 3 ? 0 : 1;
}
"""


# slots that cannot be page-locked; threads that cannot be started
@pytest.mark.parametrize("harness", [HARNESS, THREADS], ids=["slots", "threads"])
def test_transfers_without(tmp_path, harness):
    src, exe = tmp_path / "harness.cu", tmp_path / "harness"
    src.write_text(harness)
    try:
        nv = B.nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    subprocess.run([nv, str(src), "-o", str(exe), "-O1", "-std=c++17", "-I" + B.CSRC] + B.ARCH, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
