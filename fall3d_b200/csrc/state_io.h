// state_io.h -- host <-> device transfers of the large arrays.
//
// The reference arrays live in pageable host memory and hold FP64 values with
// two halo cells around each plane; the device keeps interior cells in the
// form it steps.  A StateIO moves them through a few page-locked slots: on
// the way out a kernel writes the FP64 values of a range of rows straight
// into a slot over PCIe, and a few host threads copy finished slots into the
// caller's array while later ones fill.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "f3d_common.cuh"

namespace f3d {

// Rows of a device array [b][k][j][i] and where they go in the host array:
// row (b, k, j) starts at host[off + X * (j + Y * (k + Z * b))].  Exactly one
// of c64, c32 is set; lo adds to c32 when given.
struct RowsOut {
  const double* c64;
  const float* c32;
  const float* lo;
  long long nx, ny, nz, nb;
  double* host;
  long long off, X, Y, Z;
  bool faces;  // also the zero-gradient face ghosts, two cells deep (needs the halo pitches)
};

// A member's concentration into my_c(ips-2:ipe+2, jps-2:jpe+2, kps-2:kpe+2, nbins).
inline RowsOut rows3d(const MemberDev& m, double* my_c, bool faces) {
  const long long X = m.nx + 4, Y = m.ny + 4, Z = m.nz + 4;
  return RowsOut{m.c64, m.c32, m.c32lo, m.nx, m.ny, m.nz, m.nb, my_c, 2 + X * (2 + Y * 2), X, Y, Z, faces};
}
// A deposit [b][j][i] into my_acum(ips-2:ipe+2, jps-2:jpe+2, nbins).
inline RowsOut rows2d(const double* a, long long nx, long long ny, long long nb, double* host) {
  return RowsOut{a, nullptr, nullptr, nx, ny, 1, nb, host, 2 + (nx + 4) * 2, nx + 4, ny + 4, 1, false};
}

class StateIO {
 public:
  ~StateIO() { release(); }
  // A download returns once the host array is complete.  An uploaded array may
  // change again, and the device side is complete, once the stream has been
  // waited for, as after cudaMemcpyAsync.  Work already on the stream comes
  // first.  Without page-locked memory both go through ordinary memory.
  cudaError_t download(const RowsOut& r, int device, cudaStream_t st);
  cudaError_t upload(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);
  void release();

 private:
  static constexpr int kSlots = 8;  // two per host thread
  // Eight slots of 192 KB come with the 2 MB that the driver page-locks for
  // the context's first small allocation, so that the first transfer of a
  // context takes no longer than the later ones.  Slots of 1 MB take 5-9 ms to
  // page-lock and save 2-3 ms per 100 MB (512 KB as much on the way out, but a
  // 200 x 150 x 40 x 8 meteo update takes 19.1 ms with them against 17.7), so
  // they are taken once a context has moved 128 MB.
  static constexpr size_t kSlotBytes = 192 << 10, kLargeSlotBytes = 1 << 20;
  static constexpr size_t kLargeFrom = 128 << 20;
  cudaError_t reserve(size_t total, size_t unit);
  char* pin_ = nullptr;
  size_t slot_bytes_ = 0;
  int nslots_ = 0;
  size_t moved_ = 0;  // bytes that went through reserve(), up to kLargeFrom
  bool no_large_ = false;  // the large slots could not be had
  cudaEvent_t ev_[kSlots] = {};
};

}  // namespace f3d
