// f3d_common.cuh -- device-side data layout shared by all FALL3D ADS kernels.
//
// One "member" is one model domain (a serial FALL3D run, or one ensemble
// member).  Every kernel takes a table of members plus a work list, so the
// single-domain drop-in and the batched ensemble run the same code.
//
// HBM layout of a member (interior cells only; ghost cells are rebuilt by
// the free-flow boundary condition inside each sweep, exactly where the
// reference writes them before reading them, mod_ADS.F90:269-271):
//   c     [bin][k][j][i]                     concentration (FP64 or FP32)
//   acum  [bin][j][i]                        ground deposit, FP64 always
//   ux    [snap][k][f=0..nx][j]              x-face wind, j fastest so a warp
//                                            of x-pencils reads it coalesced
//   vy    [snap][k][f=0..ny][i]              y-face wind
//   wz    [snap][f=0..nz][j][i]              z-face wind
//   k1x   [k][p=-1..nx][j]   k2y [k][p=-1..ny][i]   k3z [p=-1..nz][j][i]
//   vs    [bin][f=0..nz][j][i]               settling velocity (scaled)
// Pencils: x-pencil (j,k,bin) lanes over j; y-pencil (i,k,bin) and
// z-pencil (i,j,bin) lanes over i, so y/z loads are fully coalesced.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

namespace f3d {

constexpr double kCalm = 1e12;  // bound of the face data for MemberDev::wild
constexpr double kEps = 1e-12;  // EPSILON, mod_KindType.F90:42

// The precision form's sweeps address a member's cells and faces within one
// bin by 32-bit element offsets: (nx+1)(ny+1)(nz+1) must stay below this.
constexpr long long kMaxPencilSpan = 1LL << 31;
__host__ __device__ inline bool pencil_span_ok(long long nx, long long ny, long long nz) {
  return (nx + 1) * (ny + 1) * (nz + 1) < kMaxPencilSpan;
}

enum Dir { DIR_X = 0, DIR_Y = 1, DIR_Z = 2 };

struct MemberDev {
  int nx, ny, nz, nb;
  // state
  double* c64;
  float* c32;
  double* acum;
  // meteo snapshots (FP64 copies, used by the exact path and the CFL)
  const double* ux[2];
  const double* vy[2];
  const double* wz[2];
  const double* k1x;
  const double* k2y;
  const double* k3z;
  const double* vs;
  // FP64 face data of the exact form, per direction (0 x, 1 y, 2 z):
  //   geo[d][p+1] = {dxp(p), 1/dxp(p), dxb(p), 1/dxb(p)} for p = -1..n-1,
  //   geo[d][n+1].x = div_small() of them
  //   kkf[d] = 0.5 (k(f) + k(f-1)) at every face, laid out like the winds
  const double4* geo[3];
  const double* kkf[3];
  // FP32 face data of the precision form (null when unused), one float4 per
  // face and direction, laid out like the winds (x [k][f][j], y [k][f][i],
  // z [f][j][i]): {velocity at its, velocity at ite, 0.5 (k(f) + k(f-1)) /
  // dxp(f-1), 1/dxb(f-1) (0 at f = 0)}, so that a sweep reads a face with a
  // single 16-byte load
  const float4* f4[3];
  const float* vs32;  // [bin][f][j][i]
  // per-step current winds (written by the prep kernel)
  double* ucur;  // [k][f][j]
  double* vcur;  // [k][f][i]
  double* wcur;  // [f][j][i]
  float4* gc4[2];  // precision form with the gravity current: x and y face
                   // data with this step's winds in both velocity slots
  float wfac;       // per-member multiplicative factor on u,v (ensemble), FP32 form
  double wfacd;     // the same factor for the FP64 form and the CFL reduction
  // grid metrics (reference arrays with their halos)
  const double* dx1p;  // (nx+4)   ips-2..ipe+2
  const double* dx1b;  // (nx+3)   ibs-1..ibe+1
  const double* dx2p;
  const double* dx2b;
  const double* dx3p;
  const double* dx3b;
  const double* hm1;  // ny
  const double* hm2;  // ny+4
  const double* hm3;  // nx*ny
  const float* rdx1b32;  // 1/dx_b per axis, FP32 form
  const float* rdx2b32;
  const float* rdx3b32;
  // sparse source: cell index (i + nx*(j + ny*k)), my_s values per bin,
  // cell volume dX dY dZ Hm1 Hm2 Hm3
  int nsrc;
  const int* src_cell;
  const double* src_s;  // [q][bin]
  const double* src_vol;
  // step parameters (device resident so a step can run inside a graph)
  double dt;
  double stime;
  double time;
  double t_its, t_ite;
  int iiter;
  int gc_cur;  // precision form: the x and y sweeps read gc4 (this step's
               // winds with the gravity current) instead of f4
  // flux bookkeeping
  double* flux_part;  // per-block partial sums, [slot][2]
  int part_base[3];   // first partial slot of this member for x, y, z
  int part_count[3];  // number of partial slots (blocks) per direction
  double* flux_tot;   // running totals {W,E,S,N,U,D} and compensations [12]
  double* flux_step;  // this step's increments {W,E,S,N,U,D}
  // boundary halo layers (null unless kept): the free-flow ghost value each
  // sweep puts in the first halo cell at both ends of its pencils, laid out
  // per bin as gh_offset() gives (exact form gh64, precision form gh32)
  double* gh64;
  float* gh32;
  // compensated precision form (null otherwise): the low part of the state,
  // laid out like c32, so that the concentration is c32 + c32lo (about 48
  // bits), and 1/dxb per axis in FP64 ([cell], n entries) for the
  // conservative final update of the sweeps
  float* c32lo;
  const double* rdxb64[3];
  const float2* rdxb2[3];  // the same 1/dxb as an FP32 pair {hi, lo} (~48 bits)
  // Wet deposition and radioactive decay as the z sweep's epilogue
  // (mod_F3D.F90:1493-1520; z is the last sweep of a step): as each cell's
  // final value leaves the march it is scavenged (bins of wet_mask, cells
  // below the column's ktop) and decayed (radionuclide bins), and the
  // column's wet and dry deposits are updated by the thread that owns them.
  // epi_on = 0 leaves both processes to the separate kernels.
  int epi_on;
  unsigned long long wet_mask;       // bins that take wet deposition (0: none)
  double wet_a;                      // lambda = min(1, dt wet_a P^b)
  const double* powpb;               // P^b per column [j][i]
  const int* ktop;                   // cells k < ktop of the column are below the PBL top
  double* awet;                      // wet deposit [bin][j][i] (null without wet deposition)
  const double* radf;                // this step's {exp(-kn dt)[nr], parent's [nr]}, or null
  signed char rad_r[64];             // radionuclide index of each bin, -1 for none
  unsigned long long daughter_mask;  // bins set from their parent after the sweep (Y90)
  // *wild != 0 unless every wind, diffusion, settling velocity and spacing
  // (and its reciprocal) is below kCalm in magnitude; null counts as wild
  const int* wild;
  int4* box;  // precision form: non-zero box of every level [bin][k] (active.cuh)
};

// Host: whether steps run wet deposition and decay as the z sweep's
// epilogue (f3d_set_zsweep_epilogue; on by default).
int zsweep_epilogue();

// The epilogue's per-cell arithmetic, in the order of the separate kernels
// (phys_wet_deposition, then phys_radionuclides): a cell below the PBL top
// adds (dX3_p lambda) c to the column's wet deposit and keeps (1 - lambda) c;
// a radionuclide bin then takes c f.  Every operation is explicitly rounded
// (no contraction), so the fused and the separate paths agree bit for bit.
struct ZEpi {
  double lam;          // wet: min(1, dt a P^b) of the column
  int kt;              // wet: cells below the PBL top (0: no wet deposition)
  const double* dx3p;  // dX3_p with the reference offset (kps-2)
  double aw;           // wet deposit of the column, accumulated in k order
  double f;            // decay factor of the bin
  bool dec;            // the bin decays in the epilogue
  __device__ __forceinline__ double apply(int k, double c) {
    if (k < kt) {
      aw = __dadd_rn(aw, __dmul_rn(__dmul_rn(dx3p[k + 2], lam), c));
      c = __dmul_rn(c, __dsub_rn(1.0, lam));
    }
    return dec ? __dmul_rn(c, f) : c;
  }
  // the FP32 state: each process rounds its result to FP32, as the separate
  // kernels store it
  __device__ __forceinline__ float apply32(int k, float v) {
    if (k < kt) {
      const double c = (double)v;
      aw = __dadd_rn(aw, __dmul_rn(__dmul_rn(dx3p[k + 2], lam), c));
      v = __double2float_rn(__dmul_rn(c, __dsub_rn(1.0, lam)));
    }
    return dec ? __double2float_rn(__dmul_rn((double)v, f)) : v;
  }
};

struct NoEpi {};

// Epilogue parameters of bin b of member m for the column at ij (z sweep).
// A daughter bin (Y90) is overwritten from its parent after the sweep, so its
// epilogue does nothing.
__device__ __forceinline__ ZEpi zepi_setup(const MemberDev& m, int b, long long ij) {
  ZEpi e;
  e.lam = 0.0;
  e.kt = 0;
  e.dx3p = m.dx3p;
  e.aw = 0.0;
  e.f = 1.0;
  e.dec = false;
  const bool daughter = (m.daughter_mask >> b) & 1ull;
  if (((m.wet_mask >> b) & 1ull) && !daughter) {
    const double lam = __dmul_rn(__dmul_rn(m.dt, m.wet_a), m.powpb[ij]);
    e.lam = lam > 1.0 ? 1.0 : lam;
    e.kt = m.ktop[ij];
    e.aw = m.awet[(long long)b * m.nx * m.ny + ij];  // the sum starts from the deposit
  }
  const int r = m.rad_r[b];
  if (m.radf && r >= 0 && !daughter) {
    e.f = m.radf[r];
    e.dec = true;
  }
  return e;
}

// The column's deposits after the march: the wet deposit takes the
// scavenged sum, then both deposits decay with the bin (the dry deposit has
// already taken this step's flux).
__device__ __forceinline__ void zepi_finish(const MemberDev& m, const ZEpi& e, int b, long long ij) {
  const long long q = (long long)b * m.nx * m.ny + ij;
  if (m.awet && (e.kt > 0 || e.dec)) {
    const double w = (e.kt > 0) ? e.aw : m.awet[q];
    m.awet[q] = e.dec ? __dmul_rn(w, e.f) : w;
  }
  if (e.dec) m.acum[q] = __dmul_rn(m.acum[q], e.f);
}

// Precision-form state value of element at (c32, plus c32lo when kept).
__host__ __device__ __forceinline__ double state32(const MemberDev& m, long long at) {
  return m.c32lo ? (double)m.c32[at] + (double)m.c32lo[at] : (double)m.c32[at];
}
// Store v into the precision-form state: rounded to FP32, or split into the
// FP32 pair c32 + c32lo when the compensated state is kept.
__device__ __forceinline__ void set_state32(const MemberDev& m, long long at, double v) {
  const float hi = __double2float_rn(v);
  m.c32[at] = hi;
  if (m.c32lo) m.c32lo[at] = __double2float_rn(v - (double)hi);
}
// Add inc to the precision-form state element at (FP64 add, one rounding).
__device__ __forceinline__ void add_to_state32(const MemberDev& m, long long at, double inc) {
  set_state32(m, at, state32(m, at) + inc);
}

// Boundary halo layers of one bin: x sweep W, E [k][j]; y sweep S, N [k][i];
// z sweep D, U [j][i].  Element of pencil pen (the sweep's spatial pencil
// index) on side s (0 low, 1 high) of direction dir:
__host__ __device__ __forceinline__ long long gh_per_bin(int nx, int ny, int nz) {
  return 2LL * ((long long)ny * nz + (long long)nx * nz + (long long)nx * ny);
}
__host__ __device__ __forceinline__ long long gh_offset(int dir, int side, long long pen, int nx, int ny,
                                                        int nz) {
  const long long ax = (long long)ny * nz, ay = (long long)nx * nz, az = (long long)nx * ny;
  const long long base = (dir == 0) ? 0 : (dir == 1) ? 2 * ax : 2 * (ax + ay);
  const long long n = (dir == 0) ? ax : (dir == 1) ? ay : az;
  return base + side * n + pen;
}

// A block of one sweep: 32 consecutive spatial pencils [pen0, pen0+32) of
// one member, one warp per bin [bin0, bin0 + blockDim/32).  Spatial pencil
// index: x (j + ny k), y (i + nx k), z (i + nx j).  Blocks of the same
// spatial tile are adjacent in the work list, so the face data they share
// is served from L1/L2 instead of DRAM once per bin.
struct WorkItem {
  int member;
  int pen0;
  int bin0;
  int slot;  // flux partial slot
};

// Arguments of the precision form's range kernel (active.cuh).
struct RangeArgs {
  const WorkItem* work[3];
  int2* range[3];
  int nwork[3], grown[3];
  int dirs, bpb;
  unsigned int* acc;  // BoxGate's words in device memory
};
// What k_flux_reduce passes on to the host after a step with ranges over dirs
// (box_gate.h); null otherwise.
struct GatePub {
  unsigned int* acc;  // zero between steps but for the last word, the count of runs
  unsigned int* pub;  // page-locked
  int dirs;
};

// Host: bins per sweep block (its four warps take that many bins of one tile
// of 32 pencils, or as many more tiles).  Bins of a tile share its face data
// in L1, but a bin group that nb does not fill leaves warps idle that the
// block's registers pay for: 4, 2 or 1, the largest that divides nb.  A step of
// 201 x 147 x 43 cells full of ash with 1, 2 and 4 bins a block, us:
//   bins                7               9              11              14              15
//   compensated  337  351  350   444  450  531   477  524  559   608  603  663   634  650  673
//   FP64        2026 2108 2076  2449 2599 3119  2820 3142 3184  3638 3634 3733  3762 3780 3751
// (FP32 goes with the compensated form; the most the rule loses is 2%, FP64 100
// x 80 x 40 x 15).  Eight bins by ones instead of fours would cost 24%.  The
// boundary fluxes are sums over the blocks, so their last bits go with it.
inline int bins_per_block(int nb) { return nb % 4 == 0 ? 4 : nb % 2 == 0 ? 2 : 1; }

// Correctly rounded a/b for a divisor with precomputed y = RN(1/b)
// (Markstein's correction, applied twice so that the second correction
// starts from a faithful quotient; P. Markstein, IBM J. Res. Dev. 34(1),
// 1990).  Numerators below 2^-800 are first scaled by 2^400 (exact) so no
// intermediate is subnormal, and zero numerators return the correctly
// signed zero a*y.  For |b| in [2^-100, 2^100] this is IEEE round-to-nearest
// a/b.  A quotient in the subnormal range (numerators below ~2^-900 only, the
// far fringe of a plume) is rounded a second time by the scaling back; that
// double rounding differs from a single one only when the scaled quotient q
// lies exactly halfway between two subnormals, and then the exact remainder
// sa - q b (one FMA) tells on which side the true quotient lies, so the tie
// is resolved by one subnormal ulp.  No division and no call on any path.
__device__ __forceinline__ double div_rn_recip(double a, double b, double y) {
  const bool tiny = fabs(a) < 0x1p-800;
  const double sa = tiny ? a * 0x1p400 : a;
  double q = sa * y;
  double r = fma(-q, b, sa);
  q = fma(r, y, q);
  r = fma(-q, b, sa);
  q = fma(r, y, q);
  double res = tiny ? q * 0x1p-400 : q;
#ifndef F3D_DIV_TIE
#define F3D_DIV_TIE 1
#endif
  if (F3D_DIV_TIE && tiny) {
    const double rem = fma(-q, b, sa);     // exact: the true quotient is q + rem / b
    const double d = q - res * 0x1p400;    // exact: q's distance from the rounded result
    if (fabs(d) == 0x1p-675 && rem != 0.0 && ((d > 0.0) == ((rem > 0.0) == (b > 0.0))))
      res = res + copysign(0x1p-1074, d);  // a tie the true quotient lies beyond
  }
  return (a == 0.0) ? a * y : res;
}

// Non-zero and below the power of two whose high word is `hi`.  On the integer pipe.
__device__ __forceinline__ bool below_nonzero(double a, unsigned int hi) {
  const unsigned int m = (unsigned int)__double2hiint(a) & 0x7fffffffu;
  return m < hi && (m | (unsigned int)__double2loint(a)) != 0u;
}

// a/b as in div_rn_recip for |a| < 2^500, scaled whatever its size: no select,
// and a branch for the tie alone (one for every subnormal result makes the
// sweeps of a wide plume 10% slower: they are frequent and diverge).
__device__ __forceinline__ double div_rn_scaled(double a, double b, double y) {
  const double sa = a * 0x1p400;
  double q = sa * y;
  double r = fma(-q, b, sa);
  q = fma(r, y, q);
  r = fma(-q, b, sa);
  q = fma(r, y, q);
  double res = q * 0x1p-400;
  const double d = fma(-res, 0x1p400, q);  // exact; 0 where the result is normal
  if (fabs(d) == 0x1p-675) {
    const double rem = fma(-q, b, sa);  // exact
    if (rem != 0.0 && ((d > 0.0) == ((rem > 0.0) == (b > 0.0)))) res = res + copysign(0x1p-1074, d);
  }
  return res;
}

// The quotient with the rare numerators out of the way: q = a y and
// Markstein's two corrections, five operations where the selects, scalings
// and the tie of div_rn_recip make it ten to sixteen.  Correctly rounded while
// nothing leaves the normal range: |a| not below div_small(...) of the
// spacings, or zero.  A zero numerator gives a zero of either sign, which no
// sum of the sweeps tells apart.
__device__ __forceinline__ double div_rn_geo(double a, double b, double y) {
  double q = a * y;
  double r = fma(-q, b, a);
  q = fma(r, y, q);
  r = fma(-q, b, a);
  return fma(r, y, q);
}
// Host: the numerators div_rn_geo can take for spacings of at most `most`.
// The quotient is normal from 2^-1022 on, and the remainder, a multiple of
// ulp(q) ulp(b) >= 2^-106 |a|, is representable while that is 2^-1074 or more:
// |a| >= 2^-966 for |b| <= 2^50, 2^-920 for |b| <= 2^100 (the largest taken).
inline double div_small(double most) { return most <= 0x1p50 ? 0x1p-966 : 0x1p-920; }

// A cell's diffusive flux P0 = n / dxp and right-hand side (P0 - P1) / dxb -
// dF / dxb where one of the three numerators is small: one call for the three
// divisions.  The fringe of a wide plume is full of such values; a step of
// 301 x 227 x 37 x 4 cells takes 3.66 ms there (4.31 with a call for each
// division, 3.53 with div_rn_recip everywhere) and 1.97 without a fringe (2.50
// with div_rn_recip).  Inline in each place it costs 255 registers and 7
// minutes of compiling for no gain; a warp-wide mode that follows the last
// block's values makes every sweep 10% slower.
static __device__ __noinline__ double2 rhs_small(double n, double P1, double dF, double dxp, double rdxp, double dxb,
                                                 double rdxb) {
  // the scaled quotients stay below 2^1001
  if (fabs(n) < 0x1p400 && fabs(P1) < 0x1p499 && fabs(dF) < 0x1p500) {
    const double P0 = div_rn_scaled(n, dxp, rdxp);
    return make_double2(P0, div_rn_scaled(P0 - P1, dxb, rdxb) - div_rn_scaled(dF, dxb, rdxb));
  }
  const double P0 = div_rn_recip(n, dxp, rdxp);
  return make_double2(P0, div_rn_recip(P0 - P1, dxb, rdxb) - div_rn_recip(dF, dxb, rdxb));
}

// Correctly rounded a / 3 and a / 6 in two operations: a z + (a z') with z + z'
// = 1/3 to 2^-108 (N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 53(8), 2004).  z = RN(1/3) has 3 z = 1 -
// 2^-54, so 1/3 - z = 2^-54 / 3 and z' = RN of that = 2^-54 z.  Before its
// rounding the sum is off by less than 2^-105 |a|, and by 2^-1075 more where a
// z' is subnormal; a / 3 is a multiple of 1/3 of half an ulp of the quotient
// and no midpoint itself, so it is 1/6 ulp or more away from every midpoint,
// and the rounding falls on its side while an ulp of the quotient is 2^-1072
// or more: |a| >= 2^-1010 is.  Dividing by 2 is exact.
constexpr unsigned int kSmall36 = (1023u - 1010u) << 20;
static __device__ __noinline__ double div_rn_small(double a, double b, double y) { return div_rn_scaled(a, b, y); }
__device__ __forceinline__ double div_rn_3(double a) {
  constexpr double z = 0x1.5555555555555p-2;
  const double q = fma(a, z, a * (z * 0x1p-54));
  return below_nonzero(a, kSmall36) ? div_rn_small(a, 3.0, 1.0 / 3.0) : q;
}
__device__ __forceinline__ double div_rn_6(double a) {
  constexpr double z = 0x1.5555555555555p-3;
  const double q = fma(a, z, a * (z * 0x1p-54));
  return below_nonzero(a, kSmall36) ? div_rn_small(a, 6.0, 1.0 / 6.0) : q;
}

}  // namespace f3d
