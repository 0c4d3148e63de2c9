// sph_device.cuh -- device helpers shared by the per-particle and the per-cell kernels:
// the SPH kernel, minimum image, cell checks, neighbour records, Morris ghost velocities
// and the pair arithmetic of the velocity-gradient / force pass.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include <type_traits>

#include "sph_internal.h"

namespace sph {
#define SPH_FULL 0xffffffffu

__device__ __forceinline__ int type_of(int t) { return t & kTypeMask; }
__device__ __forceinline__ int box_of(int t) { return t >> kTypeBits; }

template <typename T> struct V4;
template <> struct V4<double> { using type = double4; };
template <> struct V4<float> { using type = float4; };

template <typename T, int DIM> struct RecFor;
template <> struct RecFor<double, 3> { using type = RecD; };
template <> struct RecFor<float, 3> { using type = RecF; };
template <> struct RecFor<double, 2> { using type = RecD2; };
template <> struct RecFor<float, 2> { using type = RecF2; };

// Fields a 2D record does not carry read as zero.
template <int DIM, typename R>
__device__ __forceinline__ auto rec_z(const R& r) -> decltype(r.x) {
  if constexpr (DIM == 3) return r.z; else return decltype(r.x)(0);
}
template <int DIM, typename R>
__device__ __forceinline__ auto rec_vz(const R& r) -> decltype(r.x) {
  if constexpr (DIM == 3) return r.vz; else return decltype(r.x)(0);
}
template <int DIM, typename R>
__device__ __forceinline__ auto rec_P(const R& r, int q) -> decltype(r.x) {
  if constexpr (DIM == 3) return r.P[q]; else return q < 3 ? r.P[q] : decltype(r.x)(0);
}

// Explicitly rounded operations: the pair sums must give the same bits in every kernel that
// takes them (one box or many, with or without the minimum image, one or two particles per
// lane), and the compiler may contract a plain expression differently in each.
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// 1 / sqrt(x) of a positive normal x.  FP64: the hardware's seed and one third-order
// Householder step, y (1 + e (1/2 + 3/8 e)) with e = 1 - x y^2 (the Taylor series of
// (1 - e)^(-1/2) to second order: the error is 5/16 e^3), without the special cases of the
// library function: below the smallest normal number the result is not finite.
__device__ __forceinline__ double inv_sqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = __fma_rn(-__dmul_rn(x, y), y, 1.0);
  return __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
}
constexpr double kMinNormal = 0x1p-1022;
// sqrt(x) of x >= 0 as x times that; 0 below the smallest normal number.
__device__ __forceinline__ double length_of(double x, double inv) {
  return x >= kMinNormal ? __dmul_rn(x, inv) : 0.0;
}

// a / b.  FP64: a times the hardware's reciprocal seed after one third-order step,
// y (1 + e + e^2) with e = 1 - b y (the series of 1 / (1 - e)), without the library's special
// cases; b is a distance from a wall or a colloid's surface.
__device__ __forceinline__ double quotient(double a, double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  const double e = __fma_rn(-b, y, 1.0);
  return __dmul_rn(a, __fma_rn(y, __fma_rn(e, e, e), y));
}
__device__ __forceinline__ float quotient(float a, float b) { return a / b; }

// c where t >= 0, else 0 (a test of the sign bit; the constant's low word is zero)
template <int C>
__device__ __forceinline__ double where_pos(double t) {
  return __hiloint2double(__double2hiint(t) < 0 ? 0 : __double2hiint((double)C), 0);
}
// SPH kernel (kernel_W.cu:13-59; its radial derivative, kernel_gradW.cu:13-53, is in
// PairRadial): cw ((3 - q)^5 - 6 (2 - q)^5 [q < 2] + 15 (1 - q)^5 [q < 1]), q = 3 r / rcut.
// Branch-free: the clamped terms are exact zeros where the reference skips them, so the value
// is that of the branchy form.  FP64: without cw, which the density sum is multiplied by.
__device__ __forceinline__ double sph_w(double r, double rcut_inv3) {
  const double t1 = xfma(-rcut_inv3, r, 3.0), t2 = xfma(-rcut_inv3, r, 2.0),
               t3 = xfma(-rcut_inv3, r, 1.0);
  const double a1 = xmul(t1, t1), a2 = xmul(t2, t2), a3 = xmul(t3, t3);
  return xfma(xmul(where_pos<15>(t3), t3), xmul(a3, a3),
              xfma(xmul(where_pos<-6>(t2), t2), xmul(a2, a2), xmul(xmul(a1, a1), t1)));
}
__device__ __forceinline__ float sph_w(float r, float rcut_inv, float cw) {
  float q3 = (r * rcut_inv) * 3.0f;
  float t1 = 3.0f - q3, t2 = 2.0f - q3, t3 = 1.0f - q3;
  float a1 = t1 * t1, a2 = t2 * t2, a3 = t3 * t3;
  float w = (a1 * a1) * t1;
  if (q3 < 2.0f) w = w - 6.0f * ((a2 * a2) * t2);
  if (q3 < 1.0f) w = w + 15.0f * ((a3 * a3) * t3);
  return cw * w;
}
__device__ __forceinline__ float sph_gradw(float r, float rcut_inv, float c_gradw) {
  float q3 = 3.0f * (r * rcut_inv);
  float t1 = 3.0f - q3, t2 = 2.0f - q3, t3 = 1.0f - q3;
  float a1 = t1 * t1, a2 = t2 * t2, a3 = t3 * t3;
  float g = a1 * a1;
  if (q3 < 2.0f) g = g - 6.0f * (a2 * a2);
  if (q3 < 1.0f) g = g + 15.0f * (a3 * a3);
  return c_gradw * g;
}

// Minimum image as the reference writes it: subtract L above L/2, add L below -L/2
// (kernel_densities.cu:90-110).  y is periodic only without walls; z only in 3D.
// WRAP false: the separation is taken as it is (for particles clear of the periodic faces,
// see clear_of_faces, where the shifts change no pair inside the cutoff).
template <typename T, int DIM, bool WRAP = true>
__device__ __forceinline__ void min_image(T& rx, T& ry, T& rz, const T L[3], const T h[3],
                                          int wall) {
  if constexpr (!WRAP) return;
  if (rx > h[0]) rx -= L[0];
  if (rx < -h[0]) rx += L[0];
  if (!wall) {
    if (ry > h[1]) ry -= L[1];
    if (ry < -h[1]) ry += L[1];
  }
  if (DIM == 3) {
    if (rz > h[2]) rz -= L[2];
    if (rz < -h[2]) rz += L[2];
  }
}

// |r|^2 with explicit roundings, rx^2 then + ry^2 then + rz^2 by fused multiply-adds: the
// compiler may contract a plain expression differently in each pass that inlines it, and
// the passes with and without the minimum image (and the density's two forms) must agree
// bit for bit.
__device__ __forceinline__ double norm2(double rx, double ry, double rz, bool three) {
  const double s = __fma_rn(ry, ry, __dmul_rn(rx, rx));
  return three ? __fma_rn(rz, rz, s) : s;
}
__device__ __forceinline__ float norm2(float rx, float ry, float rz, bool three) {
  const float s = __fmaf_rn(ry, ry, __fmul_rn(rx, rx));
  return three ? __fmaf_rn(rz, rz, s) : s;
}

// Cell of a position as kernel_cell_list.cu:15-63 computes it (with its clamp rules).
// Returns the box-local linear cell, or -1 when the reference would assert
// (kernel_cell_ranges.cu:20-23) or the position is not finite.
__device__ __forceinline__ int hash_cell(const BoxParams& p, double x, double y, double z) {
  if (!isfinite(x) || !isfinite(y) || (p.dim == 3 && !isfinite(z))) return -2;
  const double fx = floor(x / p.cell_size[0]);
  const double fy = p.wall == 0 ? floor(y / p.cell_size[1])
                                : floor((y + p.wall_width) / p.cell_size[1]);
  const double fz = p.dim == 3 ? floor(z / p.cell_size[2]) : 0.0;
  // far outside the grid: the linear index below would overflow int
  const double big = 1 << 20;
  if (fabs(fx) > big || fabs(fy) > big || fabs(fz) > big) return -1;
  int cx = (int)fx;
  if (cx == p.Ncells[0]) cx = cx - 1;
  int cy = (int)fy;
  if (p.wall == 0 && cy == p.Ncells[1]) cy = cy - 1;
  long long c;
  if (p.dim == 3) {
    int cz = (int)fz;
    if (cz == p.Ncells[2]) cz = cz - 1;
    c = (long long)cz * p.Ncells[0] * p.Ncells[1] + (long long)cy * p.Ncells[0] + cx;
  } else {
    c = (long long)cy * p.Ncells[0] + cx;
  }
  if (c < 0 || c > p.Ntotal_cells - 1) return -1;
  return (int)c;
}

// The cell the pair kernels of the reference iterate around: unclamped floor
// (kernel_densities.cu:52-60).  Returns false, leaving the outputs untouched, when the
// position is not finite or so far outside the box that one periodic wrap of the
// neighbour cells cannot bring them back into the grid; every cell index derived from a
// true result is in range.
__device__ __forceinline__ bool own_cell(const BoxParams& p, double x, double y, double z,
                                         int& cx, int& cy, int& cz) {
  const double fx = floor(x / p.cell_size[0]);
  const double fy = p.wall == 0 ? floor(y / p.cell_size[1])
                                : floor((y + p.wall_width) / p.cell_size[1]);
  const double fz = p.dim == 3 ? floor(z / p.cell_size[2]) : 0.0;
  // comparisons with NaN are false, so NaN fails every range test
  if (!(fx >= 1.0 - p.Ncells[0] && fx <= 2.0 * p.Ncells[0] - 2.0)) return false;
  if (p.wall == 0) {
    if (!(fy >= 1.0 - p.Ncells[1] && fy <= 2.0 * p.Ncells[1] - 2.0)) return false;
  } else if (!(fy >= -2.0 * p.Ncells[1] && fy <= 3.0 * p.Ncells[1])) {
    return false;  // wall axis: out-of-grid rows are skipped, only int overflow matters
  }
  if (p.dim == 3 && !(fz >= 1.0 - p.Ncells[2] && fz <= 2.0 * p.Ncells[2] - 2.0)) return false;
  cx = (int)fx;
  cy = (int)fy;
  cz = (int)fz;
  return true;
}

// Reports a failure (WORD 1: found by the hash).  The first report of any kind also records the
// step counter and the phase; the first report of a bad position records the particle's global
// id.
template <int WORD = 0>
__device__ __forceinline__ void raise_status(const Dev& d, unsigned bit, int info, int phase) {
  const unsigned old = atomicOr(d.status + WORD, bit);
  if (!(old & bit) && bit != kStatCapacity) atomicExch(&d.err_info[kErrBadId], info);
  if (!(old & kStatAbortMask)) {
    const long long s = *d.step;
    d.err_info[kErrStepLo] = (int)(s & 0xffffffffLL);
    d.err_info[kErrStepHi] = (int)(s >> 32);
    d.err_info[kErrPhase] = phase;
  }
}

// One particle's neighbour candidates in list order, decoded from the chunk entries the list
// build writes: nchunk[k * Npad + i] = (first slot, hit mask) of the particle's k-th chunk
// with hits, bit 31 - q of the mask meaning slot first + q (the first candidate in the highest
// bit, so that a count of leading zeros gives its offset).  Candidates come chunk by chunk and,
// inside a chunk, by increasing slot.
//
// next() may be called nbr_cnt[i] times: that many bits are set in the entries stored, every
// one of which has a hit, so that moving to the next entry never loops and needs no test for the
// last.  Entries are loaded one ahead; the row past the last stored one is read (the array has
// one more than the entries a particle can store) and not used.  There is no branch: the
// lanes of a warp move to their next chunks at different positions, and a branch taken by
// any lane would cost every lane the move (branch-free: 128^3 pair pass 4.03 -> 3.82 ms).
// Against tests for the last entry in each step (a count of entries, a row index): density pass
// 0.671 -> 0.624 ms (128^3 mixed), 0.707 -> 0.658 (512 2D boxes, FP64); pair pass 2.50 -> 2.46
// (128^3 FP64), 2.05 -> 2.01 (mixed), 2.58 -> 2.47 (512 boxes, FP64).
struct NbrIter {
  const int2* pn;  // the entry after nxt
  int np;          // entries are np apart
  unsigned mk;     // the current chunk's bits not yet taken
  int base;
  int2 nxt;        // the next chunk's entry
  __device__ __forceinline__ void init(const Dev& d, int i) {
    np = d.Npad;
    const int2* col = d.nchunk + i;
    const int2 e0 = __ldg(col);
    base = e0.x;
    mk = (unsigned)e0.y;
    nxt = __ldg(col + (size_t)np);
    pn = col + 2 * (size_t)np;
  }
  __device__ __forceinline__ int next() {
    const bool r = mk == 0u;
    base = r ? nxt.x : base;
    mk = r ? (unsigned)nxt.y : mk;
    if (r) {
      nxt = __ldg(pn);
      pn += np;
    }
    const int q = __clz(mk);
    mk ^= 0x80000000u >> q;
    return base + q;
  }
};

// True once a kernel before this one reported a failure: the step's state-changing kernels
// then return at entry.  The flag words are read past L1 (they are written by atomics in L2).
// In kernels whose warps cooperate, lane 0's reading is taken by the whole warp.
// step_stopped: before this step's hash (see StatusBits).
__device__ __forceinline__ bool step_stopped(const Dev& d) {
  return (*(volatile const unsigned*)d.status & kStatAbortMask) != 0u;
}
__device__ __forceinline__ bool step_aborted(const Dev& d) {
  const volatile unsigned* s = d.status;
  return ((s[0] | s[1]) & kStatAbortMask) != 0u;
}
__device__ __forceinline__ bool step_aborted_warp(const Dev& d) {
  unsigned v = 0u;
  if ((threadIdx.x & 31) < 2) v = ((volatile const unsigned*)d.status)[threadIdx.x & 31];
  return __any_sync(0xffffffffu, (v & kStatAbortMask) != 0u);
}

// A position outside [0, L] along a periodic axis of its box (or not finite).
__device__ __forceinline__ bool outside_periodic(const BoxParams& p, double x, double y,
                                                 double z) {
  return !(x >= 0.0 && x <= p.L[0]) || (p.wall == 0 && !(y >= 0.0 && y <= p.L[1])) ||
         (p.dim == 3 && !(z >= 0.0 && z <= p.L[2]));
}
__device__ __forceinline__ void mark_outside(const Dev& d, int parity) {
  d.err_info[kPosOutside + parity] = 1;
}
__device__ __forceinline__ void mark_outside(const Dev& d) { mark_outside(d, d.parity); }

// A particle at least 1.0625 rcut from every periodic face of its box.  While every position
// lies in [0, L] along the periodic axes (err_info[kPosOutside] clear), the minimum image
// changes no pair of such a particle that the sums take: a neighbour within the cutoff is
// never across a face, and a pair whose plain separation along an axis exceeds L/2 fails the
// cutoff both unshifted (L/2 > rcut) and shifted (then at least the margin, more than rcut,
// since the particle is that far from the face).  The pair passes take the separations of
// warps of such particles without the shifts: the same bits, fewer dependent operations.
template <typename T, int DIM>
__device__ __forceinline__ bool clear_of_faces(const BoxParams& p, T x, T y, T z) {
  const T m = (T)(1.0625 * p.rcut);
  bool in = x >= m && x <= (T)p.L[0] - m;
  if (DIM == 3) in = in && z >= m && z <= (T)p.L[2] - m;
  if (!p.wall) in = in && y >= m && y <= (T)p.L[1] - m;
  return in;
}
// Whether a whole warp may drop the minimum image (every lane passes `clear`); lane 0's
// reading of the flag is taken by the whole warp.
__device__ __forceinline__ bool warp_plain_image(const Dev& d, bool clear) {
  int v = 0;
  if ((threadIdx.x & 31) == 0) v = *(volatile const int*)(d.err_info + kPosOutside + d.parity);
  v = __shfl_sync(0xffffffffu, v, 0);
  return __all_sync(0xffffffffu, clear) && v == 0;
}


template <typename T, int DIM>
__device__ __forceinline__ void write_record(const Dev& d, int i, const BoxParams& p, int ti,
                                             double dens, double press) {
  using Rec = typename RecFor<T, DIM>::type;
  constexpr int kP = DIM == 3 ? 6 : 3;  // stress components carried
  Rec* rec = reinterpret_cast<Rec*>(d.rec);
  const int Np = d.Npad;
  const double4 x = d.pos[i];
  const double4 v = d.vel[i];
  Rec r;
  r.x = x.x; r.y = x.y;
  r.vx = v.x; r.vy = v.y;
  if constexpr (DIM == 3) {
    r.z = x.z;
    r.vz = v.z;
    r.tinfo = ti;
  }
  const double nkT = p.nkT;
  double c[6];
#pragma unroll
  for (int q = 0; q < kP; ++q) c[q] = d.conf[q * Np + i];
  const double dinv = 1.0 / dens;
  if (type_of(ti) == 0) {
    // Pi / d^2 with Pi = p I - nkT c (kernel_forces.cu:62-88); diagonal: xx, yy, zz
    const double dsq = dinv * dinv;
#pragma unroll
    for (int q = 0; q < kP; ++q) {
      const bool diag = q == 0 || q == 2 || q == 5;
      r.P[q] = diag ? (T)((press - nkT * c[q]) * dsq) : (T)((-nkT * c[q]) * dsq);
    }
  } else {
    // walls / colloid particles: -nkT c, completed with the fluid partner's p and d
#pragma unroll
    for (int q = 0; q < kP; ++q) r.P[q] = (T)(-nkT * c[q]);
  }
  r.invd = (T)dinv;
  rec[i] = r;
}


struct CollView {
  const double* cs;
  int nc;
};

// ---------------------------------------------------------------------------------
// Pair pass arithmetic: velocity gradient (kernel_vel_gradients.cu:15-662), forces
// (kernel_forces.cu:15-865), external force (kernel_ext_force.cu:13-73), dc/dt
// (kernel_dcdt.cu:15-104).  One function for one (i, j) pair, used by every pair kernel.
// ---------------------------------------------------------------------------------
// Read-only position loads.  In 3D a double4 is read as one 256-bit access (the vector
// width of sm_100 global loads): one L1 request per lane instead of two 128-bit ones.  In
// 2D only x and y are read (one 128-bit access; z and the mass come back zero).  Position
// arrays are 32-byte aligned (cudaMalloc base, 32-byte elements).
template <int DIM>
__device__ __forceinline__ double4 ld_pos(const double4* a) {
  double4 v;
  if (DIM == 3) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
        : "l"(a));
  } else {
    const double2 xy = __ldg(reinterpret_cast<const double2*>(a));
    v = make_double4(xy.x, xy.y, 0.0, 0.0);
  }
  return v;
}
template <int DIM>
__device__ __forceinline__ float4 ld_pos(const float4* a) {
  return __ldg(a);
}

template <typename T, int DIM>
struct PairParams {
  T L[3], h[3], rcutsq, rcut_inv, rcut_inv3, c_gradw, a, b;  // rcut_inv3 = 3 / rcut
  __device__ __forceinline__ void load(const BoxParams& p) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      L[q] = (T)p.L[q];
      h[q] = (T)p.halfL[q];
    }
    rcutsq = (T)p.rcutsq;
    rcut_inv = (T)p.rcut_inv;
    rcut_inv3 = (T)(3.0 * p.rcut_inv);
    c_gradw = (T)p.c_gradw;
    a = (T)p.a;
    b = (T)p.b;
  }
};

// the target particle i of the pass
template <typename T, int DIM>
struct PairOwn {
  T x, y, z, v[3], invd, press;
  float P[6];  // mixed precision: the particle's stress term (FP64 applies it to the sums)
  int t;
  bool fluid, do_grad, do_force;
};

// Sums of a pass over one particle's list, in FP64 accumulators.
// FP64: what is common to every term is left out of the terms and applied when the sums are
// stored (pair_store): the kernel's factor c_gradw, the particle's own stress term P_i (its
// part of the force is P_i times the sum s of gw e) and the gradient's -1/d_i.
// Mixed precision: whole terms, evaluated in float (more accurate than compensated float
// sums, and the conversions and FP64 adds run on the otherwise idle FP64 pipe).
template <typename T, int DIM>
struct PairAcc {
  double g[DIM][DIM];  // FP64: sum of gw e_a v_c; mixed: the gradient
  double f[DIM];       // the force (FP64: but the particle's own stress)
  double s[DIM];       // FP64: sum of gw e
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
#pragma unroll
      for (int c = 0; c < DIM; ++c) g[a][c] = 0.0;
      f[a] = s[a] = 0.0;
    }
  }
};

// ti: the particle's type word (from the type array)
template <typename T, int DIM, int MODE, typename Rec>
__device__ __forceinline__ void load_own(const Dev& d, int i, int ti, const Rec& ri,
                                         PairOwn<T, DIM>& o) {
  o.x = (T)ri.x;
  o.y = (T)ri.y;
  o.z = (T)rec_z<DIM>(ri);
  o.v[0] = (T)ri.vx;
  o.v[1] = (T)ri.vy;
  o.v[2] = (T)rec_vz<DIM>(ri);
  o.invd = ri.invd;
  o.press = (T)d.press[i];
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int q = 0; q < 6; ++q) o.P[q] = rec_P<DIM>(ri, q);
  }
  o.t = type_of(ti);
  o.fluid = o.t == 0;
  // gradient: every particle in kPairGradvAll; in the fused pass fluid particles (whose
  // dc/dt needs it), or every particle when the caller stores the whole field
  o.do_grad = (MODE == kPairGradvAll) || (MODE == kPairFused && (o.fluid || d.grad_all));
  o.do_force = MODE != kPairGradvAll;
}

// Separation r = x_i - x_j under the minimum image; returns |r|^2.
template <typename T, int DIM, bool WRAP, typename Rec>
__device__ __forceinline__ T pair_sep(const PairParams<T, DIM>& pp, int wall,
                                      const PairOwn<T, DIM>& o, const Rec& rj, T r[3]) {
  r[0] = o.x - (T)rj.x;
  r[1] = o.y - (T)rj.y;
  r[2] = DIM == 3 ? o.z - (T)rec_z<DIM>(rj) : T(0);
  min_image<T, DIM, WRAP>(r[0], r[1], r[2], pp.L, pp.h, wall);
  return norm2(r[0], r[1], r[2], DIM == 3);
}

// Morris ghost velocity difference of a fluid particle and a wall or colloid particle
// (kernel_forces.cu:234-418, 590-821; kernel_vel_gradients.cu:162-331, 421-630), seen from the
// target i: o is the target, rj its partner, r = x_i - x_j.  The fluid particle's velocity
// relative to the boundary is extrapolated to the solid particle, beta = 1 + (the solid
// particle's distance from the boundary) / (the fluid one's); whichever of the two the target
// is, the difference is that of the same two particles, and the lanes of a warp that hold one
// and the other take the same path.
template <typename T, int DIM, typename Rec>
__device__ __forceinline__ void ghost_velocity(const BoxParams& p, const PairParams<T, DIM>& pp,
                                               const CollView& cv, const PairOwn<T, DIM>& o,
                                               const Rec& rj, int tj, const T r[3], T v[3]) {
  const bool own = o.fluid;        // the target is the fluid particle
  const int ts = own ? tj : o.t;   // the solid particle's type
  const T vq[3] = {own ? o.v[0] : (T)rj.vx, own ? o.v[1] : (T)rj.vy,
                   DIM == 3 ? (own ? o.v[2] : (T)rec_vz<DIM>(rj)) : T(0)};
  const T yq = own ? o.y : (T)rj.y;
  const T beta_max = (T)p.beta_max;
  if (ts == 1 || ts == 2) {
    const T ys = own ? (T)rj.y : o.y;
    T dq, ds, Vw;
    if (ts == 1) {
      dq = yq - (T)p.y_bottom;
      ds = (T)p.y_bottom - ys;
      Vw = (T)p.V_bottom;
    } else {
      dq = (T)p.y_top - yq;
      ds = ys - (T)p.y_top;
      Vw = (T)p.V_top;
    }
    T beta = T(1) + quotient(ds, dq);
    beta = beta <= beta_max ? beta : beta_max;
    beta = dq > T(0) ? beta : T(1);
    v[0] = beta * (vq[0] - Vw);
    v[1] = beta * vq[1];
    v[2] = beta * vq[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = own ? v[a] : -v[a];
    return;
  }
  const int c = p.coll0 + ts - 3, nc = cv.nc;
  const T xq = own ? o.x : (T)rj.x, zq = DIM == 3 ? (own ? o.z : (T)rec_z<DIM>(rj)) : T(0);
  T rc[3] = {xq - (T)cv.cs[CS_X * nc + c], yq - (T)cv.cs[CS_Y * nc + c],
             DIM == 3 ? zq - (T)cv.cs[CS_Z * nc + c] : T(0)};
  min_image<T, DIM>(rc[0], rc[1], rc[2], pp.L, pp.h, p.wall);
  const T d2 = DIM == 3 ? rc[0] * rc[0] + rc[1] * rc[1] + rc[2] * rc[2]
                        : rc[0] * rc[0] + rc[1] * rc[1];
  const T R = (T)p.coll_R;
  T dc, n[3];  // distance from the centre and its direction
  if constexpr (sizeof(T) == 8) {
    const T inv = inv_sqrt(d2);
    dc = d2 * inv;
#pragma unroll
    for (int a = 0; a < 3; ++a) n[a] = rc[a] * inv;
  } else {
    dc = sqrt(d2);
#pragma unroll
    for (int a = 0; a < 3; ++a) n[a] = a < DIM ? rc[a] / dc : T(0);
  }
  const T dq = dc - R;  // the fluid particle's distance from the surface
  const T cvel[3] = {(T)cv.cs[CS_VX * nc + c], (T)cv.cs[CS_VY * nc + c],
                     DIM == 3 ? (T)cv.cs[CS_VZ * nc + c] : T(0)};
  const T xs = n[0] * R, ys = n[1] * R, zs = n[2] * R;
  T vr[3];
  const T wz = (T)cv.cs[CS_OZ * nc + c];
  if (DIM == 2) {
    vr[0] = -wz * ys;
    vr[1] = wz * xs;
    vr[2] = T(0);
  } else {
    const T wx = (T)cv.cs[CS_OX * nc + c], wy = (T)cv.cs[CS_OY * nc + c];
    vr[0] = wy * zs - wz * ys;
    vr[1] = wz * xs - wx * zs;
    vr[2] = wx * ys - wy * xs;
  }
  // the separation along the normal, from the solid particle to the fluid one
  const T along = DIM == 3 ? r[0] * n[0] + r[1] * n[1] + r[2] * n[2] : r[0] * n[0] + r[1] * n[1];
  const T ds = (own ? along : -along) - dq;
  T beta = T(1) + quotient(ds, dq);
  beta = beta <= beta_max ? beta : beta_max;
  // Inside the colloid: not extrapolated, and without the rotation.  A particle in the centre
  // (FP64: d2 is no normal number, and dc has no value) is inside too; the test of the exponent
  // bits costs nothing measurable (512 boxes 2.073 / 2.060 ms without / with it).
  bool inside = dq < T(0);
  if constexpr (sizeof(T) == 8) inside = inside || __double2hiint(d2) < 0x00100000;
  beta = inside ? T(1) : beta;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const T w = inside ? T(0) : vr[a];
    // (v_q - V) - w, or (V + w) - v_q
    v[a] = beta * (own ? (vq[a] - cvel[a]) - w : (cvel[a] + w) - vq[a]);
  }
}

// The radial part of a pair's terms.  FP64: 1/|r| and the vector s = (dW/dr / c_gradw) r / |r|,
// w = |s| / |r|.  Mixed: 1/|r|, the slope gw = dW/dr and the unit vector e = r / |r|.
template <typename T, int DIM>
struct PairRadial;
template <int DIM>
struct PairRadial<double, DIM> {
  double rinv, w, s[DIM];
  __device__ __forceinline__ void eval(const PairParams<double, DIM>& pp, double r2,
                                       const double r[3]) {
    rinv = inv_sqrt(r2);
    const double rr = xmul(r2, rinv);
    // (3 - q)^4 - 6 (2 - q)^4 [q < 2] + 15 (1 - q)^4 [q < 1], q = 3 |r| / rcut
    const double t1 = xfma(-pp.rcut_inv3, rr, 3.0), t2 = xfma(-pp.rcut_inv3, rr, 2.0),
                 t3 = xfma(-pp.rcut_inv3, rr, 1.0);
    const double a1 = xmul(t1, t1), a2 = xmul(t2, t2), a3 = xmul(t3, t3);
    const double gw = xfma(xmul(where_pos<15>(t3), a3), a3,
                           xfma(xmul(where_pos<-6>(t2), a2), a2, xmul(a1, a1)));
    w = xmul(gw, rinv);
#pragma unroll
    for (int a = 0; a < DIM; ++a) s[a] = xmul(w, r[a]);
  }
};
template <int DIM>
struct PairRadial<float, DIM> {
  float rinv, gw, e[3];
  __device__ __forceinline__ void eval(const PairParams<float, DIM>& pp, float r2,
                                       const float r[3]) {
    rinv = rsqrt(r2);  // r and 1/r from one reciprocal square root
    const float rr = r2 * rinv;
    gw = sph_gradw(rr, pp.rcut_inv, pp.c_gradw);
    e[0] = r[0] * rinv;
    e[1] = r[1] * rinv;
    e[2] = DIM == 3 ? r[2] * rinv : 0.0f;
  }
};

// Velocity-gradient term (kernel_vel_gradients.cu:334-337, 632-640): FP64 g_ac += gw e_a v_c,
// mixed g_ac += -(1/d_i) gw e_a v_c.
template <int DIM>
__device__ __forceinline__ void pair_grad_add(const PairOwn<double, DIM>&,
                                              const PairRadial<double, DIM>& g, const double v[3],
                                              PairAcc<double, DIM>& acc) {
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc.g[a][c] = xfma(g.s[a], v[c], acc.g[a][c]);
}
template <int DIM>
__device__ __forceinline__ void pair_grad_add(const PairOwn<float, DIM>& o,
                                              const PairRadial<float, DIM>& g, const float v[3],
                                              PairAcc<float, DIM>& acc) {
  const float s = -o.invd * g.gw;
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const float se = s * g.e[a];
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc.g[a][c] += (double)(se * v[c]);
  }
}

// Force term (kernel_forces.cu:426-440, 826-850) from the partners' stress terms Pi, Pj
// (P/d^2 - nkT c/d^2) and inverse densities di, dj: the reversible part -gw (Pi + Pj).e and the
// viscous part a gw/(di dj r) v + b gw/(di dj r) (e.v) e.  FP64: without Pi (see PairAcc).
template <int DIM>
__device__ __forceinline__ void pair_force_add(const PairParams<double, DIM>& pp,
                                               const PairRadial<double, DIM>& g,
                                               const double r[3], const double v[3],
                                               const double*, const double Pj[6], double di,
                                               double dj, PairAcc<double, DIM>& acc) {
  const double m = xmul(g.w, xmul(di, dj));
  const double aux1 = xmul(pp.a, m);
  double rv = xfma(r[1], v[1], xmul(r[0], v[0]));
  if (DIM == 3) rv = xfma(r[2], v[2], rv);
  const double aux2 = xmul(xmul(xmul(pp.b, m), rv), xmul(g.rinv, g.rinv));
  // rows of the symmetric stress: xx xy xz, xy yy yz, xz yz zz
  constexpr int kRow[3][3] = {{0, 1, 3}, {1, 2, 4}, {3, 4, 5}};
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    double f = acc.f[a];
#pragma unroll
    for (int c = 0; c < DIM; ++c) f = xfma(-Pj[kRow[a][c]], g.s[c], f);
    acc.f[a] = xfma(aux2, r[a], xfma(aux1, v[a], f));
    acc.s[a] = xadd(acc.s[a], g.s[a]);
  }
}
template <int DIM>
__device__ __forceinline__ void pair_force_add(const PairParams<float, DIM>& pp,
                                               const PairRadial<float, DIM>& g, const float*,
                                               const float v[3], const float Pi[6],
                                               const float Pj[6], float di, float dj,
                                               PairAcc<float, DIM>& acc) {
  const float gw = g.gw;
  const float* e = g.e;
  const float aux = gw * di * dj * g.rinv;
  const float aux1 = pp.a * aux;
  // the pair's force as one float term per component, then one FP64 add
  const float axx = -gw * (Pi[0] + Pj[0]);
  const float axy = -gw * (Pi[1] + Pj[1]);
  const float ayy = -gw * (Pi[2] + Pj[2]);
  float ev = e[0] * v[0] + e[1] * v[1];
  float t0 = axx * e[0] + axy * e[1], t1 = axy * e[0] + ayy * e[1], t2 = 0.0f;
  if (DIM == 3) {
    const float axz = -gw * (Pi[3] + Pj[3]);
    const float ayz = -gw * (Pi[4] + Pj[4]);
    const float azz = -gw * (Pi[5] + Pj[5]);
    ev += e[2] * v[2];
    t0 += axz * e[2];
    t1 += ayz * e[2];
    t2 = axz * e[0] + ayz * e[1] + azz * e[2];
  }
  const float aux2 = pp.b * aux * ev;
  acc.f[0] += (double)(t0 + (aux1 * v[0] + aux2 * e[0]));
  acc.f[1] += (double)(t1 + (aux1 * v[1] + aux2 * e[1]));
  if constexpr (DIM == 3) acc.f[2] += (double)(t2 + (aux1 * v[2] + aux2 * e[2]));
}

// One (i, j) pair.  tj: the neighbour's particle type.  WRAP: see min_image.
template <typename T, int DIM, bool WRAP, typename Rec>
__device__ __forceinline__ void pair_term(const BoxParams& p, const PairParams<T, DIM>& pp,
                                          const CollView& cv, const PairOwn<T, DIM>& o,
                                          const Rec& rj, int tj, PairAcc<T, DIM>& acc) {
  const bool fluid_j = tj == 0;
  // skip rules: gradient kernel_vel_gradients.cu:126-127, forces kernel_forces.cu:157-158
  const bool pair_grad = o.do_grad && !(o.t == tj && !o.fluid);
  const bool pair_force = o.do_force && (o.fluid || fluid_j);
  if (!pair_grad && !pair_force) return;
  T r[3];
  const T r2 = pair_sep<T, DIM, WRAP>(pp, p.wall, o, rj, r);
  if (!(r2 < pp.rcutsq)) return;
  T v[3] = {o.v[0] - (T)rj.vx, o.v[1] - (T)rj.vy, o.v[2] - (T)rec_vz<DIM>(rj)};
  if (o.t != tj) ghost_velocity<T, DIM>(p, pp, cv, o, rj, tj, r, v);
  PairRadial<T, DIM> g;
  g.eval(pp, r2, r);
  if (pair_grad) pair_grad_add<DIM>(o, g, v, acc);
  if (pair_force) {
    // The partner's stress term, by the two particles' kinds: fluid and fluid: its own; fluid i,
    // solid j: j mirrors i's density and pressure and keeps its own c (kernel_forces.cu:217-233);
    // solid i: i takes j's density, pressure and c (kernel_forces.cu:320-336; FP64: twice j's
    // stress, and none of its own at the end of the pass).
    const bool mirrors = o.fluid && !fluid_j;
    const T diag = mirrors ? o.press : T(0);
    const T scale = mirrors ? o.invd * o.invd : (sizeof(T) == 8 && !o.fluid ? T(2) : T(1));
    T Pi[6], Pj[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const T P = rec_P<DIM>(rj, q);
      Pi[q] = o.fluid ? (T)o.P[q] : P;
      Pj[q] = ((q == 0 || q == 2 || q == 5) ? diag + P : P) * scale;
    }
    const T di = o.fluid ? o.invd : (T)rj.invd, dj = fluid_j ? (T)rj.invd : o.invd;
    pair_force_add<DIM>(pp, g, r, v, Pi, Pj, di, dj, acc);
  }
}

// One list position of a fluid particle whose partner there is a fluid particle (or is
// absent: valid false): pair_term's fluid-fluid term without its type tests, for warps whose
// every lane has such a position (fewer branches, longer blocks for the scheduler).  For a
// fluid particle the terms taken follow from MODE alone (load_own's do_grad, do_force).
template <int MODE>
struct FluidTerms {
  static constexpr bool kGrad = MODE != kPairForcesOnly;
  static constexpr bool kForce = MODE != kPairGradvAll;
};
template <typename T, int DIM, bool WRAP, int MODE, typename Rec>
__device__ __forceinline__ void pair_fluid_x1(const BoxParams& p, const PairParams<T, DIM>& pp,
                                              const PairOwn<T, DIM>& o, const Rec& rj,
                                              bool valid, PairAcc<T, DIM>& acc) {
  T r[3];
  const T r2 = pair_sep<T, DIM, WRAP>(pp, p.wall, o, rj, r);
  if (!(valid && r2 < pp.rcutsq)) return;
  const T v[3] = {o.v[0] - (T)rj.vx, o.v[1] - (T)rj.vy, o.v[2] - (T)rec_vz<DIM>(rj)};
  PairRadial<T, DIM> g;
  g.eval(pp, r2, r);
  if constexpr (FluidTerms<MODE>::kGrad) pair_grad_add<DIM>(o, g, v, acc);
  if constexpr (FluidTerms<MODE>::kForce) {
    T Pi[6], Pj[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      Pi[q] = o.P[q];
      Pj[q] = rec_P<DIM>(rj, q);
    }
    pair_force_add<DIM>(pp, g, r, v, Pi, Pj, o.invd, (T)rj.invd, acc);
  }
}

// Second half-kick of a fluid particle's velocity, v += (dt / 2) f / m
// (kernel_move_sys_VV_part2.cu:13-58), as explicit fused multiply-adds so that the step's
// fused form and the standalone V_Verlet_step2 give the same bits.
template <int DIM>
__device__ __forceinline__ void vv2_fluid(const BoxParams& p, double mass, double fx, double fy,
                                          double fz, double4& v) {
  const double hm = 0.5 * p.dt / mass;
  v.x = __fma_rn(hm, fx, v.x);
  v.y = __fma_rn(hm, fy, v.y);
  if (DIM == 3) v.z = __fma_rn(hm, fz, v.z);
}

// stored gradient, forces with the body force, and dc/dt of particle i, from the pass's sums
// and the factors left out of them (see PairAcc)
template <typename T, int DIM, int MODE, bool EXT>
__device__ __forceinline__ void pair_store(const Dev& d, int i, const BoxParams& p,
                                           const PairOwn<T, DIM>& o,
                                           const PairAcc<T, DIM>& acc) {
  using Rec = typename RecFor<T, DIM>::type;
  const int Np2 = d.Npad;
  const double cg = sizeof(T) == 8 ? -(o.invd * p.c_gradw) : 1.0;
  double G[DIM][DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int c = 0; c < DIM; ++c) G[a][c] = cg * acc.g[a][c];
  if (MODE == kPairGradvAll || (MODE == kPairFused && d.gradv != nullptr && o.do_grad)) {
    // storage order xx xy xz yx yy yz zx zy zz
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int c = 0; c < DIM; ++c) d.gradv[(3 * a + c) * Np2 + i] = G[a][c];
  }
  if (MODE == kPairGradvAll) return;
  double F[3] = {acc.f[0], acc.f[1], DIM == 3 ? acc.f[DIM - 1] : 0.0};
  if (sizeof(T) == 8 && o.fluid) {
    const Rec* rec = reinterpret_cast<const Rec*>(d.rec);
    const double Pxx = rec[i].P[0], Pxy = rec[i].P[1], Pyy = rec[i].P[2];
    F[0] = __fma_rn(-Pxy, acc.s[1], __fma_rn(-Pxx, acc.s[0], F[0]));
    F[1] = __fma_rn(-Pyy, acc.s[1], __fma_rn(-Pxy, acc.s[0], F[1]));
    if constexpr (DIM == 3) {
      const double Pxz = rec[i].P[3], Pyz = rec[i].P[4], Pzz = rec[i].P[5];
      F[0] = __fma_rn(-Pxz, acc.s[2], F[0]);
      F[1] = __fma_rn(-Pyz, acc.s[2], F[1]);
      F[2] = __fma_rn(-Pzz, acc.s[2],
                      __fma_rn(-Pyz, acc.s[1], __fma_rn(-Pxz, acc.s[0], F[2])));
    }
  }
  const double cf = sizeof(T) == 8 ? p.c_gradw : 1.0;
  double fx = __dmul_rn(cf, F[0]), fy = __dmul_rn(cf, F[1]), fz = __dmul_rn(cf, F[2]);
  if (EXT && o.fluid) {
    const double4 xd = d.pos[i];
    const double m = xd.w;
    if (p.ext_force_type == 1) {
      fx += m * p.ext_force[0];
      fy += m * p.ext_force[1];
      if (DIM == 3) fz += m * p.ext_force[2];
    } else if (p.ext_force_type == 2) {
      fx += m * p.ext_force[0] * sin(p.ky * xd.y);
      fy += 0.0;
      if (DIM == 3) fz += 0.0;
    } else if (p.ext_force_type == 3) {
      fx += (xd.y < 0.5 * p.L[1]) ? m * p.ext_force[0] : -(m * p.ext_force[0]);
      fy += 0.0;
      if (DIM == 3) fz += 0.0;
    }
  }
  d.f[i] = fx;
  d.f[Np2 + i] = fy;
  if (DIM == 3) d.f[2 * Np2 + i] = fz;
  if (MODE == kPairFused && !o.fluid) {
    // kernel_dcdt.cu:39 leaves dc/dt of walls and colloids at its initial zero
#pragma unroll
    for (int q = 0; q < 6; ++q) d.dcdt[q * Np2 + i] = 0.0;
  }
  if (MODE == kPairFused && o.fluid) {
    // dc/dt = c.g + (c.g)^T + (I - c)/tau  (kernel_dcdt.cu:76-102)
    const double tinv = 1.0 / p.tau;
    double dc[6];
    const double cxx = d.conf[i], cxy = d.conf[Np2 + i], cyy = d.conf[2 * Np2 + i];
    if (DIM == 2) {
      const double gxx = G[0][0], gxy = G[0][1], gyx = G[1][0],
                   gyy = G[1][1];
      const double Axx = cxx * gxx + cxy * gyx, Axy = cxx * gxy + cxy * gyy;
      const double Ayx = cxy * gxx + cyy * gyx, Ayy = cxy * gxy + cyy * gyy;
      dc[0] = 2.0 * Axx + tinv * (1.0 - cxx);
      dc[1] = Axy + Ayx - tinv * cxy;
      dc[2] = 2.0 * Ayy + tinv * (1.0 - cyy);
      // the z components stay zero in 2D
      dc[3] = 0.0;
      dc[4] = 0.0;
      dc[5] = 0.0;
    } else {
      const double cxz = d.conf[3 * Np2 + i], cyz = d.conf[4 * Np2 + i], czz = d.conf[5 * Np2 + i];
      const double gxx = G[0][0], gxy = G[0][1], gxz = G[0][DIM - 1];
      const double gyx = G[1][0], gyy = G[1][1], gyz = G[1][DIM - 1];
      const double gzx = G[DIM - 1][0], gzy = G[DIM - 1][1],
                   gzz = G[DIM - 1][DIM - 1];
      const double Axx = cxx * gxx + cxy * gyx + cxz * gzx;
      const double Axy = cxx * gxy + cxy * gyy + cxz * gzy;
      const double Axz = cxx * gxz + cxy * gyz + cxz * gzz;
      const double Ayx = cxy * gxx + cyy * gyx + cyz * gzx;
      const double Ayy = cxy * gxy + cyy * gyy + cyz * gzy;
      const double Ayz = cxy * gxz + cyy * gyz + cyz * gzz;
      const double Azx = cxz * gxx + cyz * gyx + czz * gzx;
      const double Azy = cxz * gxy + cyz * gyy + czz * gzy;
      const double Azz = cxz * gxz + cyz * gyz + czz * gzz;
      dc[0] = 2.0 * Axx + tinv * (1.0 - cxx);
      dc[1] = Axy + Ayx - tinv * cxy;
      dc[2] = 2.0 * Ayy + tinv * (1.0 - cyy);
      dc[3] = Axz + Azx - tinv * cxz;
      dc[4] = Ayz + Azy - tinv * cyz;
      dc[5] = 2.0 * Azz + tinv * (1.0 - czz);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) d.dcdt[q * Np2 + i] = dc[q];
    if (d.fold_vv2) {
      // the step's second half-kick of this fluid particle (kernel_move_sys_VV_part2.cu:13-58),
      // the same operations as vv2_fluid, on the force and rate just stored
      double4 v = d.vel[i];
      vv2_fluid<DIM>(p, d.pos[i].w, fx, fy, fz, v);
      d.vel[i] = v;
#pragma unroll
      for (int q = 0; q < (DIM == 3 ? 6 : 3); ++q)
        d.conf[q * Np2 + i] = __fma_rn(0.5 * p.dt, dc[q], d.conf[q * Np2 + i]);
    }
  }
}

}  // namespace sph
