// active.cuh -- the part of the domain that a step can change.
//
// A cell's new value depends on its old one and eight neighbours on either
// side (four RK stages of two cells), so cells more than eight positions away
// from every non-zero value of their pencil keep the +0 they hold: every flux
// there is 0 times a finite face value, and +0 + dt (+-0) = +0.  Before the
// sweeps one pass over the state takes the box of non-zero cells of every
// level (MemberDev::box; -0 and NaN count as non-zero, and a level is full
// when the step's fields are not bounded, MemberDev::wild).  From the boxes,
// widened by the eight cells of each direction swept in between, every work
// item of a sweep gets its range: a block outside the boxes does nothing, the
// others march from eight cells before the box to eight after, and the zeros
// around act as the ghost cells do (frozen values, no right-hand side).
//
// The host asks for all this only where it pays (box_gate.h): a sweep without
// ranges marches whole pencils.  An eruption's plume fills a small part of its
// domain for most of a run.  On the B200 the three compensated sweeps of a
// plume in 400 x 300 x 60 x 8 cells went from 1.38 to 0.35 ms a step, with 0.08
// ms for the boxes and ranges (with ash everywhere they take 14 us and save
// nothing).  Measured against it and left: looking at the pencils from both
// ends in each sweep (0.50 ms on the plume, a memory latency ahead of every
// short march) and testing every block of the march (0.56 ms; the dense plain
// FP32 y and z sweeps 25% slower: registers).
#pragma once
#include "f3d_common.cuh"

namespace f3d {

constexpr int kReach = 8;  // cells a sweep carries values along its pencils

// Whether the step's fields are bounded, so that zeros stay zero.
__device__ __forceinline__ bool fields_calm(const MemberDev& m) {
  return m.wild && *m.wild == 0 && !m.gc_cur && fabs(m.dt) < kCalm && fabs(m.stime) < 1e6 &&
         fabs(m.wfacd) < 1e6;
}

// Widens {x0, x1} by the non-zero columns of row[from, to), read by a full
// warp 256 at a time; returns whether there are any.
__device__ __forceinline__ bool row_extent(const unsigned int* row, int from, int to, int& x0, int& x1) {
  const int lane = threadIdx.x & 31;
  bool found = false;
  for (int p = from; p < to; p += 256) {
    unsigned int v[8], any = 0u;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = p + 32 * u + lane;
      v[u] = i < to ? row[i] : 0u;
      any |= v[u];
    }
    if (!__any_sync(0xffffffffu, any != 0u)) continue;
    found = true;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const unsigned int w = __ballot_sync(0xffffffffu, v[u] != 0u);
      if (w) {
        x0 = min(x0, p + 32 * u + __ffs(w) - 1);
        x1 = max(x1, p + 32 * u + 31 - __clz(w));
      }
    }
  }
  return found;
}

// Box {x0, x1, y0, y1} (inclusive; x1 < x0 when empty) of the non-zero cells of
// level blockIdx.x (bin nz + k) of member blockIdx.y, 256 threads.  Each warp
// takes every eighth row: whole rows from both ends until one is not empty,
// then only the columns outside its box so far.  A level of zeros is read
// once (the plume's 230 MB of levels in 69 us, 3.3 TB/s); one full of ash ends
// after a few rows (46 MB in 6 us).
__global__ void __launch_bounds__(256) k_boxes32(const MemberDev* __restrict__ members) {
  const MemberDev& m = members[blockIdx.y];
  const int nx = m.nx, ny = m.ny, lev = blockIdx.x;
  if (lev >= m.nb * m.nz) return;
  if (!fields_calm(m)) {
    if (threadIdx.x == 0) m.box[lev] = make_int4(0, nx - 1, 0, ny - 1);
    return;
  }
  const unsigned int* c = reinterpret_cast<const unsigned int*>(m.c32) + (long long)lev * nx * ny;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x0 = nx, x1 = -1, y0 = ny, y1 = -1;
  int a = warp;  // rows a, a + 8, ...
  for (; a < ny; a += 8)
    if (row_extent(c + a * nx, 0, nx, x0, x1)) break;
  if (a < ny) {
    y0 = y1 = a;
    int z = warp + ((ny - 1 - warp) & ~7);
    for (; z > a; z -= 8)
      if (row_extent(c + z * nx, 0, nx, x0, x1)) break;
    y1 = z;
    for (int j = a + 8; j < z && (x0 > 0 || x1 < nx - 1); j += 8) {
      const int l = x0, r = x1 + 1;
      row_extent(c + j * nx, 0, l, x0, x1);
      row_extent(c + j * nx, r, nx, x0, x1);
    }
  }
  __shared__ int4 part[8];
  if (lane == 0) part[warp] = make_int4(x0, x1, y0, y1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int4 q = part[0];
    for (int w = 1; w < 8; ++w) {
      q.x = min(q.x, part[w].x);
      q.y = max(q.y, part[w].y);
      q.z = min(q.z, part[w].z);
      q.w = max(q.w, part[w].w);
    }
    m.box[lev] = q;
  }
}

// The cells [lo, hi) of one warp's 32 pencils, pen0.. of bin b, that a sweep
// in direction dir has to march over (lo >= hi: none).
__device__ __forceinline__ int2 box_range(const MemberDev& m, int dir, int b, int pen0, int grown) {
  const int nx = m.nx, ny = m.ny, nz = m.nz, lane = threadIdx.x & 31;
  const int n = (dir == DIR_X) ? nx : (dir == DIR_Y) ? ny : nz;
  const int nsp = (dir == DIR_X) ? ny * nz : (dir == DIR_Y) ? nx * nz : nx * ny;
  if (b >= m.nb || pen0 >= nsp) return make_int2(n, 0);
  const int gx = (grown & 1 << DIR_X) ? kReach : 0, gy = (grown & 1 << DIR_Y) ? kReach : 0;
  const int4* box = m.box + b * nz;
  int lo = n, hi = 0;
  if (dir == DIR_Z) {
    // the warp's columns: part of a row, or whole rows
    const int last = min(pen0 + 31, nsp - 1), j0 = pen0 / nx, j1 = last / nx;
    const int i0 = j0 == j1 ? pen0 - j0 * nx : 0, i1 = j0 == j1 ? last - j0 * nx : nx - 1;
    for (int q = lane; q < nz; q += 32) {
      const int4 r = box[q];
      if (r.x <= r.y && i0 <= r.y + gx && i1 >= r.x - gx && j0 <= r.w + gy && j1 >= r.z - gy) {
        lo = min(lo, q);
        hi = max(hi, q + 1);
      }
    }
  } else {
    const int pen = min(pen0 + lane, nsp - 1), ni = (dir == DIR_X) ? ny : nx, k = pen / ni, in = pen - k * ni;
    const int4 r = box[k];
    const int a0 = (dir == DIR_X) ? r.z - gy : r.x - gx, a1 = (dir == DIR_X) ? r.w + gy : r.y + gx;
    if (r.x <= r.y && in >= a0 && in <= a1) {
      lo = (dir == DIR_X) ? r.x : r.z;
      hi = ((dir == DIR_X) ? r.y : r.w) + 1;
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (hi <= lo) return make_int2(n, 0);
  lo = max(0, lo - kReach);
  return make_int2((dir == DIR_X) ? lo & ~7 : lo, min(n, hi + kReach));
}

// The range of every work item of the sweeps in dirs (a bit mask), the union
// over its four warps: one for the block, at an address that does not depend
// on the thread, so that the march keeps its length and positions in uniform
// registers (with a length of their own in every warp the y and z sweeps
// spill 150-330 bytes and take up to 25% longer).  grown[d]: the directions
// swept between the boxes and the sweep in d.  A warp per item.
__global__ void __launch_bounds__(256) k_ranges32(const MemberDev* __restrict__ members, RangeArgs a) {
  __shared__ unsigned int most[3], sum[3];
  if (threadIdx.x < 3) most[threadIdx.x] = sum[threadIdx.x] = 0u;
  __syncthreads();
  int q = blockIdx.x * 8 + (threadIdx.x >> 5), d = 0;
  for (; d < 3; ++d) {
    const int n = (a.dirs >> d & 1) ? a.nwork[d] : 0;
    if (q < n) break;
    q -= n;
  }
  if (d < 3) {
    const WorkItem w = a.work[d][q];
    int lo = 0x7fffffff, hi = 0;
    for (int s = 0; s < 4; ++s) {
      const int2 r = box_range(members[w.member], d, w.bin0 + s % a.bpb, w.pen0 + 32 * (s / a.bpb), a.grown[d]);
      lo = min(lo, r.x);
      hi = max(hi, r.y);
    }
    if ((threadIdx.x & 31) == 0) {
      a.range[d][q] = lo < hi ? make_int2(lo, hi) : make_int2(0, 0);
      if (lo < hi) {
        atomicMax(&most[d], (unsigned int)(hi - lo));
        atomicAdd(&sum[d], (unsigned int)(hi - lo));
      }
    }
  }
  __syncthreads();
  // the lengths of all items for the host (box_gate.h); k_flux_reduce passes
  // them on at the end of the step, beside work that takes longer (here, with
  // a ticket and a write to the host, they cost 6 us a step)
  if (threadIdx.x < 3 && sum[threadIdx.x]) {
    atomicMax(a.acc + threadIdx.x, most[threadIdx.x]);
    atomicAdd(a.acc + 3 + threadIdx.x, sum[threadIdx.x]);
  }
}

}  // namespace f3d
