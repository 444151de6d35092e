// state_io.cu -- the transfers of state_io.h.
//
// What bounds them is the host: the caller's array is written (or read) once
// by the CPU, and one thread moves 10-20 GB/s where PCIe carries ~50.  So the
// widening to FP64 and the sum of the compensated pair run on the device, no
// host array is made on the way (a fresh 460 MB vector costs more in page
// faults than its whole transfer), and large transfers are copied by four
// threads with two slots each: one slot fills while the other is emptied.
// On the B200 a state of 400 x 300 x 60 x 4 cells (230 MB) arrives in 16 ms,
// in 10.6 through the larger slots (130 through host vectors in one thread); a
// context's first read-back of 60 x 45 x 40 x 8 (7 MB) in 0.9 ms (1.7 through
// vectors, 9.2 with the larger slots from the start); the corner fields of a
// 200 x 150 x 40 meteo update go up in 7.6 ms (36 stacked and pageable).
#include "state_io.h"

#include <algorithm>
#include <cstring>
#include <exception>
#include <memory>
#include <new>
#include <thread>

namespace f3d {

// Elements [e0, e0 + cnt) of the array as FP64 values into a page-locked slot.
__global__ void k_rows_out(const double* __restrict__ c64, const float* __restrict__ c32,
                           const float* __restrict__ lo, long long e0, long long cnt,
                           double* __restrict__ out) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
       e += (long long)gridDim.x * blockDim.x) {
    const long long q = e0 + e;
    double v;
    if (c64) v = c64[q];
    else if (lo) v = (double)c32[q] + (double)lo[q];
    else v = (double)c32[q];
    out[e] = v;
  }
}

cudaError_t StateIO::reserve(size_t total, size_t unit) {
  moved_ += std::min(total, kLargeFrom);  // no overflow in the longest run
  moved_ = std::min(moved_, kLargeFrom);
  const bool large = !no_large_ && moved_ >= kLargeFrom && total >= kSlots * kLargeSlotBytes;
  const size_t slot = std::max(unit, std::min(large ? kLargeSlotBytes : kSlotBytes, total));
  const int n = (int)std::min<size_t>(kSlots, (total + slot - 1) / slot);
  if (slot <= slot_bytes_ && n <= nslots_) return cudaSuccess;
  release();
  cudaError_t e = cudaMallocHost((void**)&pin_, slot * n);
  if (e != cudaSuccess) {
    pin_ = nullptr;
    if (!large) return e;
    cudaGetLastError();
    no_large_ = true;
    return reserve(total, unit);
  }
  for (int s = 0; s < n; ++s)
    if ((e = cudaEventCreateWithFlags(&ev_[s], cudaEventDisableTiming)) != cudaSuccess) {
      release();
      return e;
    }
  slot_bytes_ = slot;
  nslots_ = n;
  return cudaSuccess;
}

void StateIO::release() {
  if (pin_) cudaFreeHost(pin_);
  for (auto& e : ev_) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  pin_ = nullptr;
  slot_bytes_ = 0;
  nslots_ = 0;
}

// Runs work(t, nthreads) on the calling thread and nthreads - 1 others; a
// thread that cannot be started leaves its share to the calling thread.
template <class W>
static cudaError_t on_threads(int nthreads, W work) {
  cudaError_t err[8];
  std::thread th[8];
  std::fill(err, err + 8, cudaSuccess);
  bool here[8] = {};
  for (int t = 1; t < nthreads; ++t) {
    try {
      th[t] = std::thread([&err, &work, t, nthreads] { err[t] = work(t, nthreads); });
    } catch (const std::exception&) {  // no thread, or no memory for one
      here[t] = true;
    }
  }
  err[0] = work(0, nthreads);
  for (int t = 1; t < nthreads; ++t) {
    if (here[t]) err[t] = work(t, nthreads);
    else th[t].join();
  }
  for (int t = 0; t < nthreads; ++t)
    if (err[t] != cudaSuccess) return err[t];
  return cudaSuccess;
}

// Rows [r0, r1) from a slot into the caller's array, with the face ghosts.
static void place_rows(const RowsOut& r, const double* src, long long r0, long long r1) {
  const size_t nx = (size_t)r.nx;
  if (!r.faces && r.X == r.nx && r.Y == r.ny && r.Z == r.nz) {  // no halo: one run
    memcpy(r.host + r.off + r0 * r.nx, src, nx * 8 * (size_t)(r1 - r0));
    return;
  }
  for (long long q = r0; q < r1; ++q, src += nx) {
    const long long j = q % r.ny, k = (q / r.ny) % r.nz, b = q / (r.ny * r.nz);
    double* dst = r.host + r.off + r.X * (j + r.Y * (k + r.Z * b));
    memcpy(dst, src, nx * 8);
    if (!r.faces) continue;
    dst[-1] = dst[-2] = src[0];
    dst[nx] = dst[nx + 1] = src[nx - 1];
    for (int g = 1; g <= 2; ++g) {
      if (j == 0) memcpy(dst - g * r.X, src, nx * 8);
      if (j == r.ny - 1) memcpy(dst + g * r.X, src, nx * 8);
      if (k == 0) memcpy(dst - g * r.X * r.Y, src, nx * 8);
      if (k == r.nz - 1) memcpy(dst + g * r.X * r.Y, src, nx * 8);
    }
  }
}

// The same rows through ordinary memory, a megabyte at a time on the calling
// thread: what is left where page-locked memory cannot be had.
static cudaError_t download_pageable(const RowsOut& r, cudaStream_t st) {
  const long long rows = r.ny * r.nz * r.nb;
  const long long per = std::max<long long>(1, (1 << 17) / r.nx), most = std::min(rows, per) * r.nx;
  std::unique_ptr<double[]> v(new (std::nothrow) double[most]);
  std::unique_ptr<float[]> f(r.c64 ? nullptr : new (std::nothrow) float[2 * most]);
  if (!v || (!r.c64 && !f)) return cudaErrorMemoryAllocation;
  for (long long r0 = 0; r0 < rows; r0 += per) {
    const long long r1 = std::min(rows, r0 + per), e0 = r0 * r.nx, cnt = (r1 - r0) * r.nx;
    cudaError_t e;
    if (r.c64) {
      e = cudaMemcpyAsync(v.get(), r.c64 + e0, cnt * 8, cudaMemcpyDeviceToHost, st);
    } else {
      e = cudaMemcpyAsync(f.get(), r.c32 + e0, cnt * 4, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess && r.lo)
        e = cudaMemcpyAsync(f.get() + most, r.lo + e0, cnt * 4, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    if (!r.c64)
      for (long long q = 0; q < cnt; ++q) v[q] = r.lo ? (double)f[q] + (double)f[most + q] : (double)f[q];
    place_rows(r, v.get(), r0, r1);
  }
  return cudaSuccess;
}

cudaError_t StateIO::download(const RowsOut& r, int device, cudaStream_t st) {
  const long long rows = r.ny * r.nz * r.nb;
  const size_t row = (size_t)r.nx * 8;
  if (reserve(row * (size_t)rows, row) != cudaSuccess) {
    cudaGetLastError();
    return download_pageable(r, st);
  }
  const long long per = std::max<long long>(1, (long long)(slot_bytes_ / row));
  const long long chunks = (rows + per - 1) / per;
  // two slots a thread; a single thread below 8 MB, where starting others
  // (~30 us each) costs what they save
  const int nth = (row * (size_t)rows < (8u << 20) || nslots_ < 4) ? 1 : nslots_ / 2;
  const int own = nth > 1 ? 2 : nslots_;  // slots of a thread
  return on_threads(nth, [&](int t, int n) -> cudaError_t {
    cudaError_t err = cudaSetDevice(device);
    if (err != cudaSuccess) return err;
    auto fill = [&](long long i) -> cudaError_t {  // the thread's i-th chunk
      const long long ch = t + i * n, r0 = ch * per, r1 = std::min(rows, r0 + per);
      const int s = t * own + (int)(i % own);
      const long long cnt = (r1 - r0) * r.nx;
      const int blocks = (int)std::min<long long>(148, (cnt + 511) / 512);
      k_rows_out<<<blocks, 512, 0, st>>>(r.c64, r.c32, r.lo, r0 * r.nx, cnt,
                                         (double*)(pin_ + s * slot_bytes_));
      cudaError_t q = cudaGetLastError();
      return q != cudaSuccess ? q : cudaEventRecord(ev_[s], st);
    };
    const long long mine = chunks > t ? (chunks - t + n - 1) / n : 0;
    for (long long i = 0; i < own && i < mine; ++i)
      if ((err = fill(i)) != cudaSuccess) return err;
    for (long long i = 0; i < mine; ++i) {
      const long long ch = t + i * n, r0 = ch * per, r1 = std::min(rows, r0 + per);
      const int s = t * own + (int)(i % own);
      if ((err = cudaEventSynchronize(ev_[s])) != cudaSuccess) return err;
      place_rows(r, (const double*)(pin_ + s * slot_bytes_), r0, r1);
      if (i + own < mine && (err = fill(i + own)) != cudaSuccess) return err;
    }
    return cudaSuccess;
  });
}

static bool page_locked(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeHost;
  cudaGetLastError();
  return false;
}

cudaError_t StateIO::upload(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
  // small ones take the driver's own staging, which does as well there; so do
  // all where page-locked memory cannot be had, and a caller's page-locked
  // array needs none
  bool slots = bytes >= (4u << 20) && !page_locked(src);
  if (slots && reserve(bytes, 1) != cudaSuccess) {
    cudaGetLastError();
    slots = false;
  }
  if (!slots) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  const long long per = (long long)slot_bytes_, chunks = ((long long)bytes + per - 1) / per;
  const int nth = (bytes < (8u << 20) || nslots_ < 4) ? 1 : nslots_ / 2;
  const int own = nth > 1 ? 2 : nslots_;
  const cudaError_t e = on_threads(nth, [&](int t, int n) -> cudaError_t {
    cudaError_t err = cudaSetDevice(device);
    if (err != cudaSuccess) return err;
    for (long long i = 0; t + i * n < chunks; ++i) {
      const long long o = (t + i * n) * per;
      const size_t cnt = (size_t)std::min<long long>(per, (long long)bytes - o);
      const int s = t * own + (int)(i % own);
      if (i >= own && (err = cudaEventSynchronize(ev_[s])) != cudaSuccess) return err;
      memcpy(pin_ + s * slot_bytes_, (const char*)src + o, cnt);
      if ((err = cudaMemcpyAsync((char*)dst + o, pin_ + s * slot_bytes_, cnt, cudaMemcpyHostToDevice,
                                 st)) != cudaSuccess)
        return err;
      if ((err = cudaEventRecord(ev_[s], st)) != cudaSuccess) return err;
    }
    return cudaSuccess;
  });
  const cudaError_t w = cudaStreamSynchronize(st);  // the slots are free again
  return e != cudaSuccess ? e : w;
}

}  // namespace f3d
