// sph_kernels.cu -- device kernels of the SPH step for sm_100a.
//
// Layout: particles live in "slot" order, the stable (cell, id) order of the last
// neighbour search, so that every cell's particles are contiguous in HBM.  State is SoA /
// packed AoS (pos = double4 x,y,z,mass; vel = double4) and is permuted into the new order
// once per search (k_reorder).  The pair phases read per-particle neighbour lists built by
// a warp-per-cell kernel (k_build_lists) that walks the 3^d neighbour cells (y slowest, then
// z, then x), so each particle's sums run over the same neighbours as the reference's gather
// loops (kernel_densities.cu:52-163), rows of cells along x one after the other.  All sums are
// gathers (no atomics), so results are bit-reproducible run to run.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "sph_device.cuh"
#include "sph_internal.h"

namespace sph {

// ---------------------------------------------------------------------------------
// Velocity Verlet, particles (kernel_move_sys_VV_part1.cu:13-114, ..._part2.cu:13-58)
// ---------------------------------------------------------------------------------
// Half-kick and drift of slot i (type word ti); returns its new position.  The particles of
// colloids are placed by k_vv1_colloids.
__device__ __forceinline__ double4 vv1_particle(const Dev& d, int i, int ti, const BoxParams& p) {
  const int t = type_of(ti);
  double4 x = d.pos[i];
  if (t > 2) return x;
  const double dt = p.dt;
  double4 v = d.vel[i];
  const int Np = d.Npad;
  if (t == 0) {
    double h = 0.5 * dt;
    double hm = h / x.w;
    v.x = v.x + hm * d.f[i];
    v.y = v.y + hm * d.f[Np + i];
    d.conf[i] = d.conf[i] + h * d.dcdt[i];
    d.conf[Np + i] = d.conf[Np + i] + h * d.dcdt[Np + i];
    d.conf[2 * Np + i] = d.conf[2 * Np + i] + h * d.dcdt[2 * Np + i];
    if (p.dim == 3) {
      v.z = v.z + hm * d.f[2 * Np + i];
      d.conf[3 * Np + i] = d.conf[3 * Np + i] + h * d.dcdt[3 * Np + i];
      d.conf[4 * Np + i] = d.conf[4 * Np + i] + h * d.dcdt[4 * Np + i];
      d.conf[5 * Np + i] = d.conf[5 * Np + i] + h * d.dcdt[5 * Np + i];
    }
  } else {
    v.x = (t == 1) ? p.V_bottom : p.V_top;
    v.y = 0.0;
    if (p.dim == 3) v.z = 0.0;
  }
  double xi = x.x + v.x * dt;
  double yi = x.y + v.y * dt;
  double zi = x.z;
  if (p.dim == 3) zi = x.z + v.z * dt;
  if (xi < 0) xi = xi + p.L[0];
  if (p.wall == 0 && yi < 0) yi = yi + p.L[1];
  if (p.dim == 3 && zi < 0) zi = zi + p.L[2];
  if (xi > p.L[0]) xi = xi - p.L[0];
  if (p.wall == 0 && yi > p.L[1]) yi = yi - p.L[1];
  if (p.dim == 3 && zi > p.L[2]) zi = zi - p.L[2];
  x.x = xi;
  x.y = yi;
  x.z = zi;
  d.pos[i] = x;
  d.vel[i] = v;
  return x;
}

__global__ void k_vv1_particles(Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  const int ti = d.tinfo[i];
  const BoxParams& p = d.box[box_of(ti)];
  const double4 x = vv1_particle(d, i, ti, p);
  // moved more than a box length
  if (type_of(ti) <= 2 && outside_periodic(p, x.x, x.y, x.z)) mark_outside(d);
}

__global__ void k_vv2_particles(Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  int ti = d.tinfo[i];
  if (type_of(ti) != 0) return;
  const BoxParams& p = d.box[box_of(ti)];
  const int Np = d.Npad;
  const double h = 0.5 * p.dt;
  double4 v = d.vel[i];
  const int nc = p.dim == 3 ? 6 : 3;
  if (p.dim == 3)
    vv2_fluid<3>(p, d.pos[i].w, d.f[i], d.f[Np + i], d.f[2 * Np + i], v);
  else
    vv2_fluid<2>(p, d.pos[i].w, d.f[i], d.f[Np + i], 0.0, v);
  for (int q = 0; q < nc; ++q) d.conf[q * Np + i] = __fma_rn(h, d.dcdt[q * Np + i], d.conf[q * Np + i]);
  d.vel[i] = v;
}

// Hamilton product (kernel_quaternion_product.cu:15-31)
__device__ __forceinline__ void qmul(const double* c, const double* e, double* r) {
  r[0] = c[0] * e[0] - c[1] * e[1] - c[2] * e[2] - c[3] * e[3];
  r[1] = c[0] * e[1] + c[1] * e[0] + c[2] * e[3] - c[3] * e[2];
  r[2] = c[0] * e[2] - c[1] * e[3] + c[2] * e[0] + c[3] * e[1];
  r[3] = c[0] * e[3] + c[1] * e[2] - c[2] * e[1] + c[3] * e[0];
}

// Rigid colloid half-kick, drift, rotation and re-placement of its boundary particles
// (kernel_move_colloids_VV_part1.cu:15-204).  One block per colloid.
__global__ void k_vv1_colloids(Dev d) {
  const int c = blockIdx.x;
  if (c >= d.ncoll) return;
  if (step_aborted(d)) return;
  const BoxParams& p = d.box[d.coll_box[c]];
  if (p.coll_move != 0) return;
  __shared__ double rot[4];  // 2D: cos, sin; 3D: quaternion
  __shared__ double ctr[3];
  const int nc = d.ncoll;
  double* cs = d.cs;
  const double dt = p.dt;
  if (threadIdx.x == 0) {
    double hm = 0.5 * dt / p.coll_mass, hI = 0.5 * dt / p.coll_I;
    double cx = cs[CS_X * nc + c], cy = cs[CS_Y * nc + c], cz = cs[CS_Z * nc + c];
    cs[CS_VX * nc + c] += hm * cs[CS_FX * nc + c];
    cs[CS_VY * nc + c] += hm * cs[CS_FY * nc + c];
    if (p.dim == 3) cs[CS_VZ * nc + c] += hm * cs[CS_FZ * nc + c];
    cs[CS_OZ * nc + c] += hI * cs[CS_TZ * nc + c];
    double omega;
    if (p.dim == 2) {
      omega = cs[CS_OZ * nc + c];
    } else {
      cs[CS_OX * nc + c] += hI * cs[CS_TX * nc + c];
      cs[CS_OY * nc + c] += hI * cs[CS_TY * nc + c];
      double ox = cs[CS_OX * nc + c], oy = cs[CS_OY * nc + c], oz = cs[CS_OZ * nc + c];
      omega = sqrt(ox * ox + oy * oy + oz * oz);
    }
    cx = cx + cs[CS_VX * nc + c] * dt;
    cy = cy + cs[CS_VY * nc + c] * dt;
    if (p.dim == 3) cz = cz + cs[CS_VZ * nc + c] * dt;
    if (cx < 0) cx = cx + p.L[0];
    if (cx > p.L[0]) cx = cx - p.L[0];
    if (p.wall == 0) {
      if (cy < 0) cy = cy + p.L[1];
      if (cy > p.L[1]) cy = cy - p.L[1];
    }
    if (p.dim == 3) {
      if (cz < 0) cz = cz + p.L[2];
      if (cz > p.L[2]) cz = cz - p.L[2];
    }
    cs[CS_X * nc + c] = cx;
    cs[CS_Y * nc + c] = cy;
    if (p.dim == 3) cs[CS_Z * nc + c] = cz;
    ctr[0] = cx;
    ctr[1] = cy;
    ctr[2] = cz;
    if (p.dim == 2) {
      double th = cs[CS_THETA * nc + c] + cs[CS_OZ * nc + c] * dt;
      rot[1] = sin(th);
      rot[0] = cos(th);
      cs[CS_THETA * nc + c] = th;
    } else {
      // omega = 0 gives a NaN axis, as in the reference (:123-125); the NaN positions are
      // then reported as SPH_ERR_NAN by the hash instead of trapping.
      double half = 0.5 * omega * dt;
      double ax = cs[CS_OX * nc + c] / omega, ay = cs[CS_OY * nc + c] / omega,
             az = cs[CS_OZ * nc + c] / omega;
      double sh = sin(half);
      double dq[4] = {cos(half), sh * ax, sh * ay, sh * az};
      double q[4] = {cs[CS_Q0 * nc + c], cs[CS_QX * nc + c], cs[CS_QY * nc + c],
                     cs[CS_QZ * nc + c]};
      double r[4];
      qmul(dq, q, r);
      cs[CS_Q0 * nc + c] = r[0];
      cs[CS_QX * nc + c] = r[1];
      cs[CS_QY * nc + c] = r[2];
      cs[CS_QZ * nc + c] = r[3];
      rot[0] = r[0];
      rot[1] = r[1];
      rot[2] = r[2];
      rot[3] = r[3];
    }
  }
  __syncthreads();
  const int j0 = d.coll_seg[c], j1 = d.coll_seg[c + 1];
  const int NL = d.Nlist_coll;
  for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const int slot = d.inv[d.colloids_list[j]];
    double px, py, pz = 0.0;
    if (p.dim == 2) {
      double x0 = d.xc[j], y0 = d.xc[NL + j];
      px = x0 * rot[0] - y0 * rot[1];
      py = x0 * rot[1] + y0 * rot[0];
    } else {
      double q[4] = {rot[0], rot[1], rot[2], rot[3]};
      double qi[4] = {rot[0], -rot[1], -rot[2], -rot[3]};
      double pt[4] = {0.0, d.xc[j], d.xc[NL + j], d.xc[2 * NL + j]};
      double t1[4], t2[4];
      qmul(q, pt, t1);
      qmul(t1, qi, t2);
      px = t2[1];
      py = t2[2];
      pz = t2[3];
    }
    double4 x = d.pos[slot];
    x.x = px + ctr[0];
    x.y = py + ctr[1];
    if (p.dim == 3) x.z = pz + ctr[2];
    if (x.x < 0) x.x = x.x + p.L[0];
    if (x.x > p.L[0]) x.x = x.x - p.L[0];
    if (p.wall == 0) {
      if (x.y < 0) x.y = x.y + p.L[1];
      if (x.y > p.L[1]) x.y = x.y - p.L[1];
    }
    if (p.dim == 3) {
      if (x.z < 0) x.z = x.z + p.L[2];
      if (x.z > p.L[2]) x.z = x.z - p.L[2];
    }
    if (outside_periodic(p, x.x, x.y, x.z)) mark_outside(d);
    d.pos[slot] = x;
  }
}

// Second half-kick of colloid c (kernel_move_colloids_VV_part2.cu:14-46)
__device__ __forceinline__ void vv2_colloid(const Dev& d, const BoxParams& p, int c) {
  if (p.coll_move != 0) return;
  const int nc = d.ncoll;
  double* cs = d.cs;
  double hm = 0.5 * p.dt / p.coll_mass, hI = 0.5 * p.dt / p.coll_I;
  cs[CS_VX * nc + c] += hm * cs[CS_FX * nc + c];
  cs[CS_VY * nc + c] += hm * cs[CS_FY * nc + c];
  if (p.dim == 3) cs[CS_VZ * nc + c] += hm * cs[CS_FZ * nc + c];
  cs[CS_OZ * nc + c] += hI * cs[CS_TZ * nc + c];
  if (p.dim == 3) {
    cs[CS_OX * nc + c] += hI * cs[CS_TX * nc + c];
    cs[CS_OY * nc + c] += hI * cs[CS_TY * nc + c];
  }
}

__global__ void k_vv2_colloids(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.ncoll) return;
  if (step_aborted(d)) return;
  vv2_colloid(d, d.box[d.coll_box[c]], c);
}

// ---------------------------------------------------------------------------------
// Neighbour search: hash and count -> cell ranges -> buckets -> reorder -> lists.
// The order is the reference's stable sort by cell, (cell, id) (thrust::sort_by_key,
// src/system_neighbours_search.cu:56-58): a particle's cell bounds its new slot to the cell's
// range, and its slot there is the number of the cell's particles with smaller ids, which the
// reorder counts directly (a cell holds 10 to 60 of them).  Against a two-pass radix sort of
// the keys and a separate kernel for the half-kick (8 or 13 launches from half-kick to reorder, 4
// so): a 64^2 box's step 98 -> 77 us (with the step count and the moments in other kernels too),
// half-kick to reorder at 128^3 0.35 -> 0.30 ms.
// ---------------------------------------------------------------------------------
// Magnetic moment of box b at a step (main.cu:395-400): m = (cos w t, sin w t, 0), t = t0 + dt *
// step.
__device__ __forceinline__ void set_moment(const Dev& d, int b, long long step) {
  const BoxParams& p = d.box[b];
  const double ang = p.omega_magnet * (p.t0 + p.dt * (double)step);
  d.mag[3 * b + 0] = cos(ang);
  d.mag[3 * b + 1] = sin(ang);
  d.mag[3 * b + 2] = 0.0;
}

// Cell of slot i at position x, counted; every thread of the warp calls it (active: has a
// particle).  The lanes of a cell take their places in its count by one atomic.
__device__ __forceinline__ void hash_count(const Dev& d, int i, bool active, const BoxParams& p,
                                           const double4& x) {
  int key = -1;
  if (active) {
    if (outside_periodic(p, x.x, x.y, x.z)) mark_outside(d, d.parity ^ 1);
    int c = hash_cell(p, x.x, x.y, x.z);
    if (c < 0) {
      raise_status<1>(d, c == -2 ? kStatNaN : kStatCellRange, d.gid[i], kPhaseHash);
      c = 0;  // keep the count in bounds; the step is reported as failed
    }
    key = p.cell0 + c;
  }
  const unsigned peers = __match_any_sync(SPH_FULL, key);
  const int lane = threadIdx.x & 31, lead = __ffs(peers) - 1;
  int base = 0;
  if (active && lane == lead) base = atomicAdd(&d.cell_count[key], __popc(peers));
  base = __shfl_sync(SPH_FULL, base, lead);
  if (active) d.moved[i] = make_int2(key, base + __popc(peers & ((1u << lane) - 1u)));
}

// MOVE: with the half-kick and drift before it.  Whole warps.
template <bool MOVE>
__global__ void k_hash(Dev d) {
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 - (int)(threadIdx.x & 31) >= d.Ntot) return;
  // the hash reports into the second word, so all warps of this launch decide alike
  if (step_stopped(d)) return;
  const bool active = i0 < d.Ntot;
  const int i = active ? i0 : d.Ntot - 1;
  const int ti = d.tinfo[i];
  const BoxParams& p = d.box[box_of(ti)];
  double4 x = make_double4(0.0, 0.0, 0.0, 0.0);
  if (active) x = MOVE ? vv1_particle(d, i, ti, p) : d.pos[i];
  hash_count(d, i, active, p, x);
}

// Exclusive scan over the block (kScanThreads threads); *total: the block's sum.
constexpr int kScanThreads = 1024, kScanItems = 4, kScanSpan = kScanThreads * kScanItems;
__device__ __forceinline__ int block_scan(int v, int* sh, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(SPH_FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  int u = sh[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(SPH_FULL, u, o);
    if (lane >= o) u += y;
  }
  *total = __shfl_sync(SPH_FULL, u, 31);
  const int before = __shfl_sync(SPH_FULL, u, w > 0 ? w - 1 : 0);
  __syncthreads();
  return x - v + (w > 0 ? before : 0);
}

// Sums of the spans of kScanSpan cells, for grids of more than one block.
__global__ void __launch_bounds__(kScanThreads) k_cell_sums(Dev d) {
  __shared__ int sh[32];
  if (step_stopped(d)) return;
  int v = 0;
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) {
    const int c = blockIdx.x * kScanSpan + q * kScanThreads + threadIdx.x;
    if (c < d.Ctot) v += d.cell_count[c];
  }
  int total;
  block_scan(v, sh, &total);
  if (threadIdx.x == 0) d.scan_sums[blockIdx.x] = total;
}

// cell_begin (dense, all cells) from the counts, which are zeroed for the next search; `spans`
// spans per block (more than one only in a grid of one block).  Also clears the outside flag of
// the next search and, with `advance`, sets the magnetic moments of the step being taken.
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(Dev d, int spans, int advance) {
  __shared__ int sh[32];
  if (step_stopped(d)) return;
  int carry = 0;
  if (gridDim.x > 1) {
    int v = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanThreads) v += d.scan_sums[k];
    block_scan(v, sh, &carry);
  }
  for (int s = 0; s < spans; ++s) {
    const int c0 = ((int)blockIdx.x * spans + s) * kScanSpan + (int)threadIdx.x * kScanItems;
    int n[kScanItems], v = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
      n[q] = c0 + q < d.Ctot ? d.cell_count[c0 + q] : 0;
      v += n[q];
    }
    int total;
    int at = carry + block_scan(v, sh, &total);
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
      if (c0 + q < d.Ctot) {
        d.cell_begin[c0 + q] = at;
        d.cell_count[c0 + q] = 0;
      }
      at += n[q];
    }
    carry += total;
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      d.cell_begin[d.Ctot] = d.Ntot;
      d.err_info[kPosOutside + d.parity] = 0;
    }
    if (advance && !step_aborted(d))
      for (int b = threadIdx.x; b < d.nboxes; b += kScanThreads)
        set_moment(d, b, *d.step + 1);
  }
}

// Each particle into its cell's range.
__global__ void k_bucket(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  const int2 m = d.moved[i];
  d.bucket[d.cell_begin[m.x] + m.y] = make_int2(d.gid[i], i);
}

// Gathers the state into the new slot order and records the reference's cell ranges: written
// for occupied cells only, box-local slot numbers (kernel_cell_ranges.cu:13-33).  The lanes of
// a warp hold one or two cells' particles, so the ids they count are read by broadcast.
template <bool MIXED, bool PERMUTE_F>
__global__ void k_reorder(Dev d) {
  const int at = blockIdx.x * blockDim.x + threadIdx.x;
  if (at >= d.Ntot) return;
  if (step_aborted(d)) {
    // the hash's flags, for the kernels of later steps that look at the first word alone
    if (at == 0) atomicOr(d.status, d.status[1]);
    return;
  }
  const int2 me = d.bucket[at];
  const int g = me.x, o = me.y;
  const int key = d.moved[o].x;
  const int b = d.cell_begin[key], e = d.cell_begin[key + 1];
  int rank = 0;
#pragma unroll 4
  for (int m = b; m < e; ++m) rank += d.bucket[m].x < g ? 1 : 0;
  const int k = b + rank;
  const int Np = d.Npad;
  const double4 x = d.pos[o];
  d.pos_b[k] = x;
  d.vel_b[k] = d.vel[o];
#pragma unroll
  for (int q = 0; q < 6; ++q) d.conf_b[q * Np + k] = d.conf[q * Np + o];
  if (PERMUTE_F) {
#pragma unroll
    for (int q = 0; q < 3; ++q) d.f_b[q * Np + k] = d.f[q * Np + o];
#pragma unroll
    for (int q = 0; q < 6; ++q) d.dcdt_b[q * Np + k] = d.dcdt[q * Np + o];
  }
  const int ti = d.tinfo[o];
  d.tinfo_b[k] = ti;
  d.gid_b[k] = g;
  d.inv[g] = k;
  d.keys[k] = key;
  d.vals[k] = g;
  if (MIXED) d.pos_f[k] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
  if (rank == 0) {
    const int slot0 = d.box[box_of(ti)].slot0;
    d.cell_start[key] = b - slot0;
    d.cell_end[key] = e - 1 - slot0;
  }
}

// Density contribution of one list entry (kernel_densities.cu:52-163 with kernel_W.cu): the
// exact distance test, then W(r) with r from one reciprocal square root; the particle itself
// (r2 = 0) contributes W(0).  FP64: over cw, and rcut_inv is 3 / rcut.  WRAP: see min_image.
// SELECT: without a branch.
template <typename T, int DIM, bool WRAP = true, bool SELECT = false>
__device__ __forceinline__ T density_term(const typename V4<T>::type& xi,
                                          const typename V4<T>::type& xj, const T L[3],
                                          const T h[3], int wall, T rcutsq, T rcut_inv, T cw) {
  T rx = xi.x - xj.x, ry = xi.y - xj.y, rz = DIM == 3 ? xi.z - xj.z : T(0);
  min_image<T, DIM, WRAP>(rx, ry, rz, L, h, wall);
  const T r2 = norm2(rx, ry, rz, DIM == 3);
  const bool in = r2 < rcutsq;
  if (!SELECT && !in) return T(0);
  T w;
  if constexpr (sizeof(T) == 8) {
    // r is 0 where r2 has no reciprocal root, chosen after it, or before it with SELECT (ms, before /
    // after: 128^3 0.935 / 0.921, 512 2D boxes 0.658 / 0.644; with SELECT, 64^2, 0.0221 / 0.0230)
    double r;
    if constexpr (SELECT)
      r = r2 >= kMinNormal ? xmul(r2, inv_sqrt(r2)) : 0.0;
    else
      r = length_of(r2, inv_sqrt(r2));
    w = sph_w(r, rcut_inv);
  } else {
    w = sph_w(r2 > 0.0f ? r2 * rsqrt(r2) : 0.0f, rcut_inv, cw);
  }
  return in ? w : T(0);
}

// Density, pressure (kernel_pressures.cu:13-23) and the neighbour record of slot i.
template <typename T, int DIM>
__device__ __forceinline__ void density_epilogue(const Dev& d, int i, const BoxParams& p,
                                                 double dens) {
  d.dens[i] = dens;
  const double press = p.csq * (d.pos[i].w * dens - p.rho0);
  d.press[i] = press;
  write_record<T, DIM>(d, i, p, d.tinfo[i], dens, press);
}

// One warp per cell: the cell's particles (<= 32 per round) test the candidates of the
// 3^d neighbour cells, staged 32 at a time in shared memory as offsets from the cell.
// Candidate ranges are those of the reference-semantics cell_start / cell_end, so the
// candidates are the reference's (kernel_densities.cu:52-163), stale
// ranges included.  The test uses a slightly enlarged cutoff; consumers apply the
// exact test.
//
// The lists are chunks with hit masks, not indices.  Candidates come in chunks of up to 32
// consecutive slots of one range; for every chunk in which it has a hit, a particle
// stores one 8-byte entry (the chunk's first slot, a 32-bit mask whose bit 31 - q means slot
// first + q is a candidate), chunk-major: nchunk[k * Npad + i], so that consumers walking
// their lists in step read neighbouring words.  Decoding the entries in order, bit by bit,
// gives the neighbours in the order of an index list (the candidate order), at
// 8 bytes per chunk with hits (about 20 in 3D) instead of 4 bytes per neighbour (about
// 108), and the build needs no per-lane append loop: a chunk's hits are one store.
//
// A particle whose own (unclamped) cell differs from its sort cell (x exactly at L) has
// other neighbour cells; its whole warp tests its candidates with ballots.
//
// (Summing the density over the hits inside this kernel was measured slower than the
// separate k_density pass: the per-lane hit loops diverge and the warp runs the FP64
// kernel evaluation for its busiest lane.)
//
// With 16 threads per cell (k_build_lists_half) each half-warp works on its own cell, chunks are
// 16 slots long and the test is in packed float.  The neighbours are the same either way (same
// candidates, same order).  It is a choice of the tuning, the faster build of large 2D boxes with
// 16 particles a cell only.  Measured (us, a warp per cell / a half): 2D, overlap 4, 64^2 12.0 /
// 14.8, 256^2 16.2 / 17.1, 512^2 35.0 / 34.8, 600^2 46.8 / 44.0 (its pair pass 151.6 / 155.1, over
// longer lists); overlap 3, 512^2 45.2 / 53.2; 512 boxes 446 / 660; 3D, 48^3 40.6 / 98.3.
//
// Blocks of 4 warps, measured against 8 (128^3 list build 1.66 vs 1.88 ms; 2D ensemble
// 1.15 vs 1.19 ms, with the test loop not unrolled).
constexpr int kListWarps = 4;

// Packed FP32 pairs (the f32x2 arithmetic of sm_100): two candidates per instruction.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float lo, float hi) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Candidate test of two staged candidates (a: their x pair, b: y, c: z, as loaded from the
// stage) against one particle: the sign bit of rx^2 + ry^2 + rz^2 - cut2, accumulated by fused
// multiply-adds from -cut2, funnel-shifted into `hits` first candidate first (one shift per
// candidate).  The rounding of the chain can only move candidates within a few float ulps of
// the list cutoff, which lies 5e-5 of rcut beyond the cutoff every consumer applies exactly,
// so the neighbours found are the same.  Staged padding at 1e30 gives +inf and no hit.
// (Against a separate subtract and a shift-and-or per candidate: 128^3 list build 1.04 ->
// 0.95 ms.)
template <int DIM>
__device__ __forceinline__ unsigned list_test2(unsigned hits, f32x2 xi, f32x2 yi, f32x2 zi,
                                               f32x2 ncut2, f32x2 a, f32x2 b, f32x2 c) {
  const f32x2 rx = f2_sub(xi, a), ry = f2_sub(yi, b);
  f32x2 s = f2_fma(ry, ry, f2_fma(rx, rx, ncut2));
  if (DIM == 3) {
    const f32x2 rz = f2_sub(zi, c);
    s = f2_fma(rz, rz, s);
  }
  unsigned lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(s));
  hits = __funnelshift_l(lo, hits, 1);
  return __funnelshift_l(hi, hits, 1);
}

// Candidate placement.  A candidate of a neighbour cell's range is staged with that cell's
// periodic shift, except in two cases where it must be placed at its minimum image about the
// centre of the listing cell:
//  - a stale range: an emptied cell keeps the range of the search that last saw it occupied
//    (kernel_cell_ranges.cu:13-33); after the sort those slots hold whatever particles, from
//    anywhere in the box, and the consumers take them by the minimum image as the reference
//    does (kernel_densities.cu:90-110), so some are neighbours through another face;
//  - a position outside the box (err_info[kPosOutside]): the hash's linear cell index runs
//    on into the next row, so a particle can sit in a range far from its position.
// With at least 3 cells per axis (cell >= rcut) the image about the centre is the one within
// the cutoff of every particle of the cell, if any is.  A warp with a stale neighbour range,
// or every warp while a position is outside, places all its candidates so; the others keep
// the per-cell shift, which needs no test per candidate.
//
// v: a candidate's unshifted offset from the cell's corner along one axis; c the cell's
// width, L the box's.
__device__ __forceinline__ float stale_offset(float v, double c, double L) {
  const float r = v - (float)(0.5 * c), hl = (float)(0.5 * L);
  return r > hl ? v - (float)L : (r < -hl ? v + (float)L : v);
}
// The same with the bounds precomputed (lo = c/2 - L/2, hi = c/2 + L/2; an axis that does
// not wrap has infinite bounds).
__device__ __forceinline__ float frame_offset(float v, const float* lo, const float* hi,
                                              const float* L, int q) {
  v = v > hi[q] ? v - L[q] : v;
  return v < lo[q] ? v + L[q] : v;
}

// Neighbour cell q (0 .. 3^d - 1: dy slowest, then dz, then dx) of cell (cx, cy, cz) of box p
// with the periodic wrap; false where the row does not exist (beyond a wall).  The three cells
// of a row lie one after the other in memory, up to the wrap.
template <int DIM>
__device__ __forceinline__ bool neighbour_cell(const BoxParams& p, int cx, int cy, int cz,
                                               int q, int& nc) {
  constexpr int kNZ = DIM == 3 ? 3 : 1;
  const int N0 = p.Ncells[0], N1 = p.Ncells[1], N2 = p.Ncells[2];
  int nx = cx + q % 3 - 1, ny = cy + q / (3 * kNZ) - 1;
  int nz = DIM == 3 ? cz + (q / 3) % 3 - 1 : 0;
  if (nx < 0) nx += N0;
  if (nx >= N0) nx -= N0;
  if (DIM == 3) {
    if (nz < 0) nz += N2;
    if (nz >= N2) nz -= N2;
  }
  if (!p.wall) {
    if (ny < 0) ny += N1;
    if (ny >= N1) ny -= N1;
  }
  if (ny < 0 || ny >= N1) return false;
  nc = p.cell0 + (DIM == 3 ? (nz * N1 + ny) * N0 + nx : ny * N0 + nx);
  return true;
}

// An emptied cell whose reference range still lists slots.
__device__ __forceinline__ bool stale_cell(const Dev& d, int nc) {
  return d.cell_end[nc] >= d.cell_start[nc] && d.cell_begin[nc] == d.cell_begin[nc + 1];
}

// A particle exactly on the upper box edge: its own neighbour cells, the whole warp testing its
// candidates.  ti, tb: its slot and box (uniform).  Returns its chunks with hits.
template <int DIM>
__device__ __forceinline__ int list_odd_particle(const Dev& d, int ti, int tb) {
  constexpr int kNZ = DIM == 3 ? 3 : 1;
  const int lane = threadIdx.x & 31, cap = d.cap;
  const size_t Np = d.Npad;
  const BoxParams& tp = d.box[tb];
  const double4 xt = d.pos[ti];
  int ax = 0, ay = 0, az = 0;
  own_cell(tp, xt.x, xt.y, xt.z, ax, ay, az);  // checked above: cannot fail
  const double tox = ax * tp.cell_size[0];
  const double toy = ay * tp.cell_size[1] - (tp.wall ? tp.wall_width : 0.0);
  const double toz = DIM == 3 ? az * tp.cell_size[2] : 0.0;
  const float tcut2 = (float)tp.list_cut2;
  const float txi = (float)(xt.x - tox), tyi = (float)(xt.y - toy), tzi = (float)(xt.z - toz);
  int tcnt = 0, tk = 0;
  for (int q = 0; q < 9 * kNZ; ++q) {
    int nc;
    if (!neighbour_cell<DIM>(tp, ax, ay, az, q, nc)) continue;
    const int s = d.cell_start[nc] + tp.slot0, e = d.cell_end[nc] + tp.slot0;
    for (int c0 = s; c0 <= e; c0 += 32) {
      const int j = c0 + lane;
      bool hit = false;
      if (j <= e) {
        // rare: every candidate at its minimum image about the particle's own cell
        double4 xj = d.pos[j];
        const float vx = stale_offset((float)(xj.x - tox), tp.cell_size[0], tp.L[0]);
        float vy = (float)(xj.y - toy);
        if (!tp.wall) vy = stale_offset(vy, tp.cell_size[1], tp.L[1]);
        float vz = (float)(xj.z - toz);
        if (DIM == 3) vz = stale_offset(vz, tp.cell_size[2], tp.L[2]);
        const float rx = txi - vx;
        const float ry = tyi - vy;
        float r2 = rx * rx + ry * ry;
        if (DIM == 3) {
          const float rz = tzi - vz;
          r2 += rz * rz;
        }
        hit = r2 < tcut2;
      }
      const unsigned hits = __brev(__ballot_sync(SPH_FULL, hit));
      if (hits != 0u) {
        if (lane == 0 && tk < cap) d.nchunk[(size_t)tk * Np + ti] = make_int2(c0, (int)hits);
        tcnt += __popc(hits);
        ++tk;
      }
    }
  }
  if (lane == 0) d.nbr_cnt[ti] = tk <= cap ? tcnt : 0;
  return tk;
}

// ---- a warp per cell: the candidate test on the tensor cores ----
//
// r_ij^2 - cut^2 = |x_i|^2 - cut^2 + |x_j|^2 - 2 x_i.x_j for a round of 32 particles (rows) and a
// chunk of 32 candidates (columns) is a matrix product with few terms: mma.m16n8k16, float16
// operands and float accumulators, the sign of an accumulator being the hit.  Coordinates are
// offsets from the cell's centre over rcut, each split into two float16 (the second holds what
// the first rounds away), so that a candidate is eight float16, four words:
//     (x y) (z n) (x' y') (z' n')         n + n' = |x_j|^2, primes: the second parts
// A particle's row multiplies them by (-2x -2y) (-2z 1) (-2x -2y) (-2z 1) and, in the upper half
// of K, the same words once more by (-2x' -2y') (-2z' 0) (-2x' -2y') (-2z' 0); the accumulators
// start from |x_i|^2 - cut^2.  Offsets are below 2 (cells are at most 4/3 rcut wide), so a split
// coordinate is within 5e-7 and the square within 1.5e-5 of its value.  The products are exact.
// Their sum, if the matrix unit cuts each of the 17 addends to 24 bits of the largest (below 8 for
// a pair within reach: n, (1.16 + 1)^2 at most), is off by 17 x 2^-21, 1e-5, at most.  list_cut2
// exceeds the cutoff that every consumer applies exactly by 1e-4: no neighbour is missed.
// Candidates further off (minimum-image placement) only have to be outside: held within 200 rcut,
// and n below what a float16 holds.
//
// What bounds it: instruction issue (67 % at 96^3).  The packed float test (k_build_lists_half),
// whose operands and subtractions each lane repeats for every candidate, took most of a chunk's
// instructions; with the matrix product about 110 are left, for staging (FP64 positions to four
// words), eight matrix instructions and the masks, and as many as 15 chunks take for a cell's
// ranges and rows.  A row of three neighbour cells is one range of slots, since their particles
// follow one another in memory, so chunks are nearly full: cells of 16 particles took 9 chunks,
// their rows take 6, and the consumers' lists are shorter as well.
// Sign bits are shifted into one byte per row and lane, and two exchanges with byte selections
// turn a quad's bytes into its rows' masks; candidates are staged in the columns that make their
// order come out right.  The largest chunk count goes to memory only where it is larger than the
// one there: an atomic from every cell's warp was what the 2D grids waited for.
// Measured (ms; packed float test cell by cell / matrix product cell by cell / by rows / and with
// the byte masks and the filtered count): 128^3 0.857 / 0.641 / 0.599 / 0.564, 96^3 with colloids
// 0.346 / 0.265 / 0.258 / 0.244, 61 x 53 x 67 0.129 / 0.099 / 0.097 / 0.089, 512 2D boxes 0.657 /
// 0.683 / 0.616 / 0.447, one 64^2 box 0.0140 / 0.0127 / 0.0119 / 0.0113.  64 rows a round, for
// cells of more than 32, were slower (128^3 0.577 -> 0.629: registers).
__device__ __forceinline__ unsigned pack_h2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}
__device__ __forceinline__ float2 unpack_h2(unsigned u) {
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}
// B's two registers hold the same word, C's four two start values; they are passed one by one,
// from loads and shuffles of their own, because the instruction takes them from neighbouring
// registers and equal ones would be copied there before each.
__device__ __forceinline__ void mma_16x8x16(unsigned (&d)[4], const unsigned (&a)[4], unsigned b0,
                                            unsigned b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%11,%12,%13};\n"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
        "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], unsigned at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
// The sign bits of a lane's accumulators against TILES tiles of 8 candidates, one byte (two tiles:
// nibble) for each of its two rows, g in the upper one: columns 2 t and 2 t + 1 of tile 0 first.
template <int TILES>
__device__ __forceinline__ unsigned hit_bits(const unsigned (&a)[4], const unsigned (&b)[8],
                                             const float (&c)[4]) {
  unsigned d[TILES][4];
#pragma unroll
  for (int u = 0; u < TILES; ++u) mma_16x8x16(d[u], a, b[2 * u], b[2 * u + 1], c);
  unsigned m[2] = {0u, 0u};
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int u = 0; u < TILES; ++u) {
      m[h] = __funnelshift_l(d[u][2 * h], m[h], 1);
      m[h] = __funnelshift_l(d[u][2 * h + 1], m[h], 1);
    }
  return m[0] << 8 | m[1];
}
// The four words of a candidate at (x, y, z); keep: it exists.
__device__ __forceinline__ uint4 candidate_words(float x, float y, float z, bool keep) {
  constexpr float kFar = 60000.0f;
  float n = fminf(fmaf(z, z, fmaf(y, y, x * x)), kFar);
  n = keep ? n : kFar;
  uint4 w;
  w.x = pack_h2(x, y);
  w.y = pack_h2(z, n);
  const float2 a = unpack_h2(w.x), c = unpack_h2(w.y);
  w.z = pack_h2(x - a.x, y - a.y);
  w.w = pack_h2(z - c.x, n - c.y);
  return w;
}

template <int DIM>
// Blocks per SM the registers are held to, measured (ms, 6 / 7 / 8): 128^3 0.596 / 0.574 / 0.564,
// 512 2D boxes 0.512 / 0.473 / 0.447.
__global__ void __launch_bounds__(kListWarps * 32, 8)
    k_build_lists(Dev d, int split) {
  constexpr int kNZ = DIM == 3 ? 3 : 1;
  // the chunk's candidates, 16 bytes each, tiles of 8 rows two rows apart (a round of stores then
  // meets no bank twice)
  __shared__ uint4 stage[kListWarps][40];
  __shared__ float frame[kListWarps][9];   // lo[3], hi[3], L[3] (frame_offset)
  // the candidates as ranges of consecutive slots (a row of three neighbour cells is one, or two
  // at the periodic wrap), and what takes their positions to offsets from this cell's centre
  __shared__ int2 range[kListWarps][9 * kNZ];
  __shared__ double shift[kListWarps][9 * kNZ][DIM];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (step_aborted_warp(d)) return;
  // a position outside the box (the hash's flag) may be sorted into a cell other than its
  // own (the linear cell index runs on into the next row): then every candidate is placed
  // by its minimum image, as in a stale range
  int out_flag = 0;
  if (lane == 0) out_flag = *(volatile const int*)(d.err_info + kPosOutside + d.parity);
  const bool any_out = __shfl_sync(SPH_FULL, out_flag, 0) != 0;
  // `split` warps per cell, warp `part` of them taking every split-th round of particles
  const int part = (blockIdx.x * kListWarps + w) % split;
  const int cell = (blockIdx.x * kListWarps + w) / split;
  if (cell >= d.Ctot) return;  // whole warps
  const int b = d.cell_box[cell];
  const BoxParams& p = d.box[b];
  const int N0 = p.Ncells[0], N1 = p.Ncells[1], N2 = p.Ncells[2];
  const int lc = cell - p.cell0;
  const int row = lc / N0, cx = lc - row * N0;
  const int cz = DIM == 3 ? row / N1 : 0, cy = row - cz * N1;
  const int beg = d.cell_begin[cell], end = d.cell_begin[cell + 1];
  const double ox = cx * p.cell_size[0];
  const double oy = cy * p.cell_size[1] - (p.wall ? p.wall_width : 0.0);
  const double oz = DIM == 3 ? cz * p.cell_size[2] : 0.0;
  // the cell's centre; offsets from it in units of rcut
  const double mx = ox + 0.5 * p.cell_size[0], my = oy + 0.5 * p.cell_size[1];
  const double mz = DIM == 3 ? oz + 0.5 * p.cell_size[2] : 0.0;
  const float inv = (float)p.rcut_inv;
  // offsets up to these are inside the cell whatever the rounding of its bounds
  constexpr float kIn = 0.5f - 1e-5f;
  const float inx = kIn * (float)p.cell_size[0] * inv, iny = kIn * (float)p.cell_size[1] * inv;
  const float inz = kIn * (float)p.cell_size[2] * inv;
  const float cut2 = (float)(p.list_cut2 * p.rcut_inv * p.rcut_inv);
  const int cap = d.cap;  // chunks with hits a particle can store
  const size_t Np = d.Npad;
  const int span = end - beg;
  int maxch = 0;  // the most chunks with hits any particle of this warp had
  // lane q looks up neighbour cell q (all 3^d loads in flight at once)
  int rs = 0, re = -1, nb = 0, ne = -1;  // the recorded range, the range of this search
  if (lane < 9 * kNZ) {
    int nc;
    if (neighbour_cell<DIM>(p, cx, cy, cz, lane, nc)) {
      rs = d.cell_start[nc] + p.slot0;
      re = d.cell_end[nc] + p.slot0;
      nb = d.cell_begin[nc];
      ne = d.cell_begin[nc + 1] - 1;
    }
  }
  // a stale range, or a position outside the box: minimum-image placement for the whole warp
  // (see stale_offset)
  const bool mi = any_out || __any_sync(SPH_FULL, re >= rs && ne < nb);
  // Otherwise the recorded ranges are this search's, and the cells of a row that follow one
  // another in x do so in memory: the first of them takes the others' slots.
  const int ne1 = __shfl_down_sync(SPH_FULL, ne, 1), ne2 = __shfl_down_sync(SPH_FULL, ne, 2);
  if (!mi) {
    const int dx = lane % 3;  // cell cx - 1, cx or cx + 1 of the row
    rs = nb;
    re = ne;
    if (dx == 0 && cx > 0) re = cx < N0 - 1 ? ne2 : ne1;
    if (dx == 1) re = cx == 0 ? ne1 : rs - 1;
    if (dx == 2 && cx < N0 - 1) re = rs - 1;
  }
  const unsigned filled = __ballot_sync(SPH_FULL, lane < 9 * kNZ && re >= rs);
  const int nseg = __popc(filled);
  if ((filled >> lane) & 1u) {
    const int at = __popc(filled & ((1u << lane) - 1u));
    range[w][at] = make_int2(rs, re);
    const int nx = cx + lane % 3 - 1, ny = cy + lane / (3 * kNZ) - 1;
    shift[w][at][0] = (nx < 0 ? -p.L[0] : nx >= N0 ? p.L[0] : 0.0) - mx;
    shift[w][at][1] = (p.wall ? 0.0 : ny < 0 ? -p.L[1] : ny >= N1 ? p.L[1] : 0.0) - my;
    if (DIM == 3) {
      const int nz = cz + (lane / 3) % 3 - 1;
      shift[w][at][DIM - 1] = (nz < 0 ? -p.L[2] : nz >= N2 ? p.L[2] : 0.0) - mz;
    }
  }
  if (mi && lane == 0) {
    for (int q = 0; q < 3; ++q) {
      const bool wraps = q == 0 || (q == 1 && !p.wall) || (q == 2 && DIM == 3);
      const float c = (float)(0.5 * p.cell_size[q]), h = (float)(0.5 * p.L[q]);
      frame[w][q] = wraps ? c - h : -3.0e38f;
      frame[w][3 + q] = wraps ? c + h : 3.0e38f;
      frame[w][6 + q] = (float)p.L[q];
    }
  }
  __syncwarp();
  const float* flo = frame[w];
  const float* fhi = flo + 3;
  const float* fL = flo + 6;
  const int g = lane >> 2, t = lane & 3;  // this lane's part of the fragments
  // Candidate k of a chunk is staged in the column whose sign bits end up in bit 31 - k of the
  // masks: column 2 t + c of tile u for k = 8 t + 2 u + c, in chunks of at most 16 (two tiles)
  // k = 4 t + 2 u + c.
  const int col_long = 10 * ((lane >> 1) & 3) + 2 * (lane >> 3) + (lane & 1);
  const int col_short =
      lane < 16 ? 10 * ((lane >> 1) & 1) + 2 * (lane >> 2) + (lane & 1) : 20 + (lane & 15);
  // each tile's rows twice, for the two words of B
  const unsigned srow =
      (unsigned)__cvta_generic_to_shared(&stage[w][10 * (lane >> 4) + (lane & 7)]);
  // byte selectors of the quad's 4 x 4 transposition
  const unsigned sel1 = (t & 1) ? 0x6240u : 0x3715u, sel2 = (t & 2) ? 0x5410u : 0x3276u;
  // the particle loop, in the cheap form (per-cell shifts) or the minimum-image one
  auto walk = [&](auto mi_tag) {
    constexpr bool kMI = decltype(mi_tag)::value;
    for (int t0 = part * 32; t0 < span; t0 += split * 32) {
      // lane 4 g + t holds row g + 8 t: the quad of lanes that gets row g's accumulators in its
      // four fragments also holds the particles of those four rows
      const int i = beg + t0 + g + 8 * t;
      const bool active = i < end;
      float xi = 0.f, yi = 0.f, zi = 0.f;
      bool odd = false, lost = false;
      if (active) {
        const double4 x = ld_pos<DIM>(d.pos + i);
        xi = (float)(x.x - mx) * inv;
        yi = (float)(x.y - my) * inv;
        zi = DIM == 3 ? (float)(x.z - mz) * inv : 0.f;
        int ax = 0, ay = 0, az = 0;
        if (fabsf(xi) < inx && fabsf(yi) < iny && (DIM == 2 || fabsf(zi) < inz)) {
          // inside its sort cell, without own_cell's divisions
        } else if (own_cell(p, x.x, x.y, x.z, ax, ay, az)) {
          odd = (ax != cx) || (ay != cy) || (DIM == 3 && az != cz);
        } else {
          // not finite or far outside the box: already reported by the hash; no neighbours
          lost = true;
          const bool finite = isfinite(x.x) && isfinite(x.y) && isfinite(x.z);
          raise_status(d, finite ? kStatCellRange : kStatNaN, d.gid[i], kPhaseLists);
        }
      }
      const bool listed = active && !odd && !lost;
      // A row without a particle is zero but for its start value, and has no hits; a position
      // too far out for a float16 would make it infinities times zero.
      if (!listed) xi = yi = zi = 0.f;
      // this particle's row: words of the lower and the upper half of K, start value
      const uint4 cw = candidate_words(xi, yi, zi, true);
      const float2 h01 = unpack_h2(cw.x), h23 = unpack_h2(cw.y), l01 = unpack_h2(cw.z),
                   l23 = unpack_h2(cw.w);
      const float s = listed ? -2.0f : 0.0f;
      const unsigned lo0 = pack_h2(s * h01.x, s * h01.y), lo1 = pack_h2(s * h23.x, listed ? 1.f : 0.f);
      const unsigned up0 = pack_h2(s * l01.x, s * l01.y), up1 = pack_h2(s * l23.x, 0.f);
      const float start = listed ? fmaf(zi, zi, fmaf(yi, yi, xi * xi)) - cut2 : 1.0f;
      // fragments: word t (of the four) of rows g, g + 8 and of rows g + 16, g + 24
      unsigned fa[2][4];
      float fc[2][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int from = 4 * g + q;  // the lane that holds row g + 8 q
        const unsigned a0 = __shfl_sync(SPH_FULL, lo0, from), a1 = __shfl_sync(SPH_FULL, lo1, from);
        const unsigned b0 = __shfl_sync(SPH_FULL, up0, from), b1 = __shfl_sync(SPH_FULL, up1, from);
        fa[q >> 1][q & 1] = (t & 1) ? a1 : a0;
        fa[q >> 1][2 + (q & 1)] = (t & 1) ? b1 : b0;
        fc[q >> 1][2 * (q & 1)] = __shfl_sync(SPH_FULL, start, from);
        fc[q >> 1][2 * (q & 1) + 1] = __shfl_sync(SPH_FULL, start, from);
      }
      const bool two = span - t0 > 16;             // rows 16 .. 31 are in use
      int2* col = d.nchunk + (listed ? i : 0);     // this particle's chunks, stride Npad
      int cnt = 0;                                 // its candidates
      int kc = 0;                                  // its chunks with hits
      for (int q = 0; q < nseg; ++q) {
        const int cs = range[w][q].x, ce = range[w][q].y;
        const double sx = shift[w][q][0], sy = shift[w][q][1], sz = shift[w][q][DIM - 1];
        for (int c0 = cs; c0 <= ce; c0 += 32) {
          const int j = c0 + lane;
          float vx = 0.f, vy = 0.f, vz = 0.f;
          if (j <= ce) {
            const double4 xj = ld_pos<DIM>(d.pos + j);
            if constexpr (kMI) {
              vx = frame_offset((float)(xj.x - ox), flo, fhi, fL, 0) - (float)(mx - ox);
              vy = frame_offset((float)(xj.y - oy), flo, fhi, fL, 1) - (float)(my - oy);
              if (DIM == 3) vz = frame_offset((float)(xj.z - oz), flo, fhi, fL, 2) - (float)(mz - oz);
            } else {
              vx = (float)(xj.x + sx);
              vy = (float)(xj.y + sy);
              if (DIM == 3) vz = (float)(xj.z + sz);
            }
          }
          vx *= inv;
          vy *= inv;
          vz *= inv;
          if constexpr (kMI) {  // no further than float16 reaches
            vx = fminf(fmaxf(vx, -200.f), 200.f);
            vy = fminf(fmaxf(vy, -200.f), 200.f);
            vz = fminf(fmaxf(vz, -200.f), 200.f);
          }
          const bool wide = ce - c0 >= 16;
          stage[w][wide ? col_long : col_short] = candidate_words(vx, vy, vz, j <= ce);
          __syncwarp();
          unsigned fb[8];  // word t of candidate g of tile u in fb[2 u] and fb[2 u + 1]
          ldmatrix_x4(*reinterpret_cast<unsigned(*)[4]>(&fb[0]), srow);
          // rows g and g + 8 in bytes 3 and 2, g + 16 and g + 24 in bytes 1 and 0
          unsigned m;
          if (wide) {
            ldmatrix_x4(*reinterpret_cast<unsigned(*)[4]>(&fb[4]), srow + 20 * 16);
            __syncwarp();  // the stage is refilled by the next chunk
            m = hit_bits<4>(fa[0], fb, fc[0]) << 16;
            if (two) m |= hit_bits<4>(fa[1], fb, fc[1]);
          } else {
            __syncwarp();
            m = hit_bits<2>(fa[0], fb, fc[0]) << 16;
            if (two) m |= hit_bits<2>(fa[1], fb, fc[1]);
          }
          // the quad's bytes of row g + 8 r to the lane that holds the row (t = r), t = 0 first: bit
          // 31 - k of `hits` is then candidate k, the consumers' order of leading zeros
          m = __byte_perm(m, __shfl_xor_sync(SPH_FULL, m, 1), sel1);
          unsigned hits = __byte_perm(m, __shfl_xor_sync(SPH_FULL, m, 2), sel2);
          if (!wide) {  // nibbles: together, and to the top
            hits = __byte_perm(hits << 4 | hits << 8, 0u, 0x3144u);
          }
          if (hits != 0u) {  // a chunk with hits: (first slot, mask) in the next entry
            if (kc < cap) col[(size_t)kc * Np] = make_int2(c0, (int)hits);
            cnt += __popc(hits);
            ++kc;
          }
        }
      }
      if (active && !odd) d.nbr_cnt[i] = kc <= cap ? cnt : 0;  // 0: the step stops here
      maxch = max(maxch, kc);
      // particles exactly on the upper box edge: their own neighbour cells
      unsigned odd_mask = __ballot_sync(SPH_FULL, active && odd);
      while (odd_mask) {
        const int l = __ffs(odd_mask) - 1;
        odd_mask &= odd_mask - 1;
        const int ti = __shfl_sync(SPH_FULL, i, l), tb = __shfl_sync(SPH_FULL, b, l);
        maxch = max(maxch, list_odd_particle<DIM>(d, ti, tb));
      }
    }
  };
  if (mi)
    walk(std::true_type{});
  else
    walk(std::false_type{});
  // warp max of the chunk counts -> capacity check
  maxch = __reduce_max_sync(SPH_FULL, maxch);
  if (lane == 0) {
    if (maxch > *(volatile const int*)(d.err_info + kErrMaxCount))
      atomicMax(&d.err_info[kErrMaxCount], maxch);
    if (maxch > cap) raise_status(d, kStatCapacity, 0, kPhaseLists);
  }
}

// ---- a half warp per cell: packed float test ----
template <int DIM>
__global__ void __launch_bounds__(kListWarps * 32) k_build_lists_half(Dev d, int split) {
  constexpr int TPC = 16;
  // candidates staged as three float rows per warp, read four at a time
  __shared__ __align__(16) float stage_x[kListWarps][32];
  __shared__ __align__(16) float stage_y[kListWarps][32];
  __shared__ __align__(16) float stage_z[kListWarps][32];
  __shared__ float frame[kListWarps][2][9];  // per group: lo[3], hi[3], L[3] (frame_offset)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (step_aborted_warp(d)) return;
  // a position outside the box (the hash's flag) may be sorted into a cell other than its
  // own (the linear cell index runs on into the next row): then every candidate is placed
  // by its minimum image, as in a stale range
  int out_flag = 0;
  if (lane == 0) out_flag = *(volatile const int*)(d.err_info + kPosOutside + d.parity);
  const bool any_out = __shfl_sync(SPH_FULL, out_flag, 0) != 0;
  const int sub = lane / TPC, gl = lane % TPC;  // group within the warp, lane within the group
  float* stx = &stage_x[w][sub * TPC];
  float* sty = &stage_y[w][sub * TPC];
  float* stz = &stage_z[w][sub * TPC];
  // `split` warps per cell, warp `part` of them taking every split-th round of particles
  const int part = (blockIdx.x * kListWarps + w) % split;
  const int cell = (blockIdx.x * kListWarps + w) / split * (32 / TPC) + sub;
  // both groups of a warp walk the same loop structure in lockstep (divergent halves would
  // run one after the other): trip counts are warp maxima, a group past its own range idles
  const bool live = cell < d.Ctot;
  if (!__any_sync(SPH_FULL, live)) return;
  const int cl = live ? cell : 0;
  const int b = d.cell_box[cl];
  const BoxParams& p = d.box[b];
  const int N0 = p.Ncells[0], N1 = p.Ncells[1], N2 = p.Ncells[2];
  const int lc = cl - p.cell0;
  const int cx = lc % N0, cy = (lc / N0) % N1, cz = DIM == 3 ? lc / (N0 * N1) : 0;
  const int beg = live ? d.cell_begin[cl] : 0, end = live ? d.cell_begin[cl + 1] : 0;
  const double ox = cx * p.cell_size[0];
  const double oy = cy * p.cell_size[1] - (p.wall ? p.wall_width : 0.0);
  const double oz = DIM == 3 ? cz * p.cell_size[2] : 0.0;
  const float cut2 = (float)p.list_cut2;
  const int cap = d.cap;  // chunks with hits a particle can store
  const size_t Np = d.Npad;
  auto warp_max = [](int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(SPH_FULL, v, o));
    return v;
  };
  const int span = warp_max(end - beg);
  int maxch = 0;  // the most chunks with hits any particle of this warp had
  constexpr int kNZ = DIM == 3 ? 3 : 1;
  bool found = false;  // a stale neighbour range
  if (live) {
    for (int q = gl; q < 9 * kNZ; q += TPC) {
      int nc;
      if (neighbour_cell<DIM>(p, cx, cy, cz, q, nc)) found = found || stale_cell(d, nc);
    }
  }
  // minimum-image placement for the whole warp (see stale_offset)
  const bool mi = any_out || __any_sync(SPH_FULL, found);
  if (mi && gl == 0) {
    float* f = frame[w][sub];
    for (int q = 0; q < 3; ++q) {
      const bool wraps = q == 0 || (q == 1 && !p.wall) || (q == 2 && DIM == 3);
      const float c = (float)(0.5 * p.cell_size[q]), h = (float)(0.5 * p.L[q]);
      f[q] = wraps ? c - h : -3.0e38f;
      f[3 + q] = wraps ? c + h : 3.0e38f;
      f[6 + q] = (float)p.L[q];
    }
  }
  __syncwarp();
  const float* flo = frame[w][sub];
  const float* fhi = flo + 3;
  const float* fL = flo + 6;
  // the particle loop, in the cheap form (per-cell shifts) or the minimum-image one
  auto walk = [&](auto mi_tag) {
    constexpr bool kMI = decltype(mi_tag)::value;
    for (int t0 = part * TPC; t0 < span; t0 += split * TPC) {
      const int i = beg + t0 + gl;
      const bool active = i < end;
      float xi = 0.f, yi = 0.f, zi = 0.f;
      bool odd = false, lost = false;
      if (active) {
        const double4 x = ld_pos<DIM>(d.pos + i);
        xi = (float)(x.x - ox);
        yi = (float)(x.y - oy);
        zi = (float)(x.z - oz);
        int ax = 0, ay = 0, az = 0;
        if (own_cell(p, x.x, x.y, x.z, ax, ay, az)) {
          odd = (ax != cx) || (ay != cy) || (DIM == 3 && az != cz);
        } else {
          // not finite or far outside the box: already reported by the hash; no neighbours
          lost = true;
          const bool finite = isfinite(x.x) && isfinite(x.y) && isfinite(x.z);
          raise_status(d, finite ? kStatCellRange : kStatNaN, d.gid[i], kPhaseLists);
        }
      }
      const bool listed = active && !odd && !lost;
      const f32x2 xi2 = f2_pack(xi, xi), yi2 = f2_pack(yi, yi), zi2 = f2_pack(zi, zi);
      const f32x2 ncut22 = f2_pack(-cut2, -cut2);
      int2* col = d.nchunk + (listed ? i : 0);  // this particle's chunks, stride Npad
      int cnt = 0;                              // this lane's candidates
      int kc = 0;                               // this lane's chunks with hits
      for (int ddy = -1; ddy <= 1; ++ddy)
        for (int ddz = (DIM == 3 ? -1 : 0); ddz <= (DIM == 3 ? 1 : 0); ++ddz)
          for (int ddx = -1; ddx <= 1; ++ddx) {
            int nx = cx + ddx, ny = cy + ddy, nz = cz + ddz;
            double sx = 0.0, sy = 0.0, sz = 0.0;
            if (nx < 0) { nx += N0; sx = -p.L[0]; }
            if (nx >= N0) { nx -= N0; sx = p.L[0]; }
            if (DIM == 3) {
              if (nz < 0) { nz += N2; sz = -p.L[2]; }
              if (nz >= N2) { nz -= N2; sz = p.L[2]; }
            }
            if (!p.wall) {
              if (ny < 0) { ny += N1; sy = -p.L[1]; }
              if (ny >= N1) { ny -= N1; sy = p.L[1]; }
            }
            // an empty range where the neighbour row does not exist (walls) or the group idles
            int s = 0, e = -1;
            if (live && ny >= 0 && ny < N1) {
              const int nc = p.cell0 + (DIM == 3 ? (nz * N1 + ny) * N0 + nx : ny * N0 + nx);
              s = d.cell_start[nc] + p.slot0;
              e = d.cell_end[nc] + p.slot0;
            }
            const int nch = e >= s ? (e - s + TPC) / TPC : 0;
            const int nchw = warp_max(nch);
            for (int k = 0; k < nchw; ++k) {
              const int c0 = s + k * TPC;
              const int j = c0 + gl;
              float vx = 1e30f, vy = 1e30f, vz = 1e30f;  // padding: never a hit
              if (k < nch && j <= e) {
                const double4 xj = ld_pos<DIM>(d.pos + j);
                if constexpr (kMI) {
                  vx = frame_offset((float)(xj.x - ox), flo, fhi, fL, 0);
                  vy = frame_offset((float)(xj.y - oy), flo, fhi, fL, 1);
                  vz = frame_offset((float)(xj.z - oz), flo, fhi, fL, 2);
                } else {
                  vx = (float)(xj.x + sx - ox);
                  vy = (float)(xj.y + sy - oy);
                  vz = (float)(xj.z + sz - oz);
                }
              }
              stx[gl] = vx;
              sty[gl] = vy;
              if (DIM == 3) stz[gl] = vz;
              __syncwarp();
              const int n = k < nch ? min(TPC, e - c0 + 1) : 0;
              // hit mask of this chunk; staged candidate q is slot c0 + q.  Both halves run a
              // fixed trip count, which keeps them on one instruction stream.
              unsigned hits = 0u;
#pragma unroll 1
              for (int q = 0; q < TPC; q += 4) {
                const ulonglong2 cx4 = *reinterpret_cast<const ulonglong2*>(stx + q);
                const ulonglong2 cy4 = *reinterpret_cast<const ulonglong2*>(sty + q);
                const ulonglong2 cz4 = DIM == 3 ? *reinterpret_cast<const ulonglong2*>(stz + q)
                                                : make_ulonglong2(0ull, 0ull);
                hits = list_test2<DIM>(hits, xi2, yi2, zi2, ncut22, cx4.x, cy4.x, cz4.x);
                hits = list_test2<DIM>(hits, xi2, yi2, zi2, ncut22, cx4.y, cy4.y, cz4.y);
              }
              // first candidate was shifted in first: align it to bit 31 (bit 31 - q is
              // candidate q, the consumers' order of leading zeros)
              hits <<= 32 - TPC;
              hits &= (listed && n > 0) ? ~(0xFFFFFFFFu >> n) : 0u;
              if (hits != 0u) {  // a chunk with hits: (first slot, mask) in the next entry
                if (kc < cap) col[(size_t)kc * Np] = make_int2(c0, (int)hits);
                cnt += __popc(hits);
                ++kc;
              }
              __syncwarp();  // the stage is refilled by the next chunk
            }
          }
      if (active && !odd) d.nbr_cnt[i] = kc <= cap ? cnt : 0;  // 0: the step stops here
      maxch = max(maxch, kc);
      // particles exactly on the upper box edge: their own neighbour cells
      unsigned odd_mask = __ballot_sync(SPH_FULL, active && odd);
      while (odd_mask) {
        const int l = __ffs(odd_mask) - 1;
        odd_mask &= odd_mask - 1;
        const int ti = __shfl_sync(SPH_FULL, i, l), tb = __shfl_sync(SPH_FULL, b, l);
        maxch = max(maxch, list_odd_particle<DIM>(d, ti, tb));
      }
    }
  };
  if (mi)
    walk(std::true_type{});
  else
    walk(std::false_type{});
  // warp max of the chunk counts -> capacity check
  maxch = warp_max(maxch);
  if (lane == 0 && maxch > 0) {
    if (maxch > *(volatile const int*)(d.err_info + kErrMaxCount))
      atomicMax(&d.err_info[kErrMaxCount], maxch);
    if (maxch > cap) raise_status(d, kStatCapacity, 0, kPhaseLists);
  }
}

// Colloid coarse grid (kernel_cell_colloids_list.cu, kernel_initialize_cell_colloids.cu,
// kernel_cell_colloids_ranges.cu) with the stable (cell, index) order of thrust's sort.
// One block per box.
__global__ void k_colloid_cells(Dev d, int nboxes) {
  const int b = blockIdx.x;
  if (b >= nboxes) return;
  if (step_aborted(d)) return;
  const BoxParams& p = d.box[b];
  const int n = p.N_colloids;
  if (n < 2) return;
  const int c0 = p.coll0, nc = d.ncoll;
  extern __shared__ int s_cell[];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double x = d.cs[CS_X * nc + c0 + i], y = d.cs[CS_Y * nc + c0 + i];
    int cx = (int)floor(x / p.cell_colloids_size[0]);
    int cy = (int)floor(y / p.cell_colloids_size[1]);
    int c;
    if (p.dim == 3) {
      int cz = (int)floor(d.cs[CS_Z * nc + c0 + i] / p.cell_colloids_size[2]);
      c = cz * p.Ncells_colloids[0] * p.Ncells_colloids[1] + cy * p.Ncells_colloids[0] + cx;
    } else {
      c = cy * p.Ncells_colloids[0] + cx;
    }
    s_cell[i] = c;
  }
  for (int c = threadIdx.x; c < p.Ntotal_cells_colloids; c += blockDim.x) {
    d.ccell_start[p.ccell0 + c] = -1;
    d.ccell_end[p.ccell0 + c] = -2;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int ci = s_cell[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) rank += (s_cell[j] < ci) || (s_cell[j] == ci && j < i);
    d.ccell[c0 + rank] = ci;
    d.cindex[c0 + rank] = i;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int ci = d.ccell[c0 + i];
    if (ci < 0 || ci >= p.Ntotal_cells_colloids) continue;
    if (i == 0 || d.ccell[c0 + i - 1] != ci) d.ccell_start[p.ccell0 + ci] = i;
    if (i == n - 1 || d.ccell[c0 + i + 1] != ci) d.ccell_end[p.ccell0 + ci] = i;
  }
}

// One lane's density sum over its list, in list order.  The positions of kAhead entries are
// loaded before they are summed (each term depends on a gathered position: with one load in
// flight per lane the pass waited on memory, 5 long-scoreboard stalls per instruction).
// Measured at 128^3 (FP64, with the plain separations): 1.16 ms with one entry at a time,
// 1.10 ms with two, 1.21 and 1.22 ms with three and four (registers, fewer warps).
template <typename T, int DIM, bool WRAP, int kAhead>
__device__ __forceinline__ double density_sum(const Dev& d, const typename V4<T>::type* P,
                                              int i, const BoxParams& p) {
  using V = typename V4<T>::type;
  const T L[3] = {(T)p.L[0], (T)p.L[1], (T)p.L[2]};
  const T h[3] = {(T)p.halfL[0], (T)p.halfL[1], (T)p.halfL[2]};
  const T rcutsq = (T)p.rcutsq;
  const T rcut_inv = (T)((sizeof(T) == 8 ? 3.0 : 1.0) * p.rcut_inv), cw = (T)p.cw;
  const V xi = ld_pos<DIM>(P + i);
  const int n = d.nbr_cnt[i];
  NbrIter it;
  it.init(d, i);
  double dens = 0;
  for (int k = 0; k < n; k += kAhead) {
    int j[kAhead];
    V x[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) j[u] = k + u < n ? it.next() : -1;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) x[u] = ld_pos<DIM>(P + (j[u] >= 0 ? j[u] : i));
    if constexpr (kAhead > 2) {
      // the terms side by side, then their sum in order
      T w[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        w[u] = density_term<T, DIM, WRAP, true>(xi, x[u], L, h, p.wall, rcutsq, rcut_inv, cw);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) dens = dens + (j[u] >= 0 ? w[u] : T(0));
    } else {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (j[u] < 0) break;
        const T w = density_term<T, DIM, WRAP>(xi, x[u], L, h, p.wall, rcutsq, rcut_inv, cw);
        dens = dens + w;
      }
    }
  }
  return sizeof(T) == 8 ? __dmul_rn(p.cw, dens) : dens;  // the factor left out of the terms
}

// Whole warps (lanes past the end mirror the last slot and store nothing), so that a warp
// of particles clear of the periodic faces takes the sums without the minimum image.
template <typename T, int DIM, int AHEAD>
__global__ void k_density(Dev d) {
  using V = typename V4<T>::type;
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 - (int)(threadIdx.x & 31) >= d.Ntot) return;  // whole warps only
  if (step_aborted_warp(d)) return;
  const bool active = i0 < d.Ntot;
  const int i = active ? i0 : d.Ntot - 1;
  // positions: the double state itself, or its float copy in mixed precision
  const V* __restrict__ P = sizeof(T) == 8 ? reinterpret_cast<const V*>(d.pos)
                                           : reinterpret_cast<const V*>(d.pos_f);
  const BoxParams& p = d.box[box_of(d.tinfo[i])];
  const V xi = ld_pos<DIM>(P + i);
  double dens;
  if (warp_plain_image(d, clear_of_faces<T, DIM>(p, xi.x, xi.y, xi.z)))
    dens = density_sum<T, DIM, false, AHEAD>(d, P, i, p);
  else
    dens = density_sum<T, DIM, true, AHEAD>(d, P, i, p);
  if (active) density_epilogue<T, DIM>(d, i, p, dens);
}

// Density over neighbour-cell tiles: one warp per cell, as the list build.  The positions
// of the neighbour cells' candidate ranges (the list build's ranges, stale ones included)
// are staged in shared memory by coalesced copies, in phases of 9 cells (the dy = -1, 0, +1
// planes in 3D; all 9 cells at once in 2D), and every lane walks its own list in order,
// reading each neighbour from the tile.  The sums are those of k_density term for term:
// the same list order, the same arithmetic; only where the position is read from differs.
// An entry outside the staged ranges (a tile overflow, or a particle listed from other
// cells because it sits exactly on the upper box edge) reads its position from global
// memory in place, so the order is never changed.
constexpr int kDensWarps = 4;
constexpr int kDensTile = 320;  // staged positions per warp and phase

template <typename T, int DIM>
__global__ void __launch_bounds__(kDensWarps * 32) k_density_cells(Dev d) {
  using V = typename V4<T>::type;
  constexpr int kNZ = DIM == 3 ? 3 : 1;
  constexpr int kNR = 9 * kNZ;               // neighbour cells
  constexpr int kPh = DIM == 3 ? 3 : 1;      // phases
  constexpr int kPerPh = kNR / kPh;          // cells per phase (9)
  __shared__ T tx[kDensWarps][kDensTile], ty[kDensWarps][kDensTile], tz[kDensWarps][kDensTile];
  __shared__ int rtab[kDensWarps][kPerPh][3];  // per phase: first slot, last slot, tile offset
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cell = blockIdx.x * kDensWarps + w;
  if (cell >= d.Ctot) return;  // whole warps only
  if (step_aborted_warp(d)) return;
  const V* __restrict__ P = sizeof(T) == 8 ? reinterpret_cast<const V*>(d.pos)
                                           : reinterpret_cast<const V*>(d.pos_f);
  const int b = d.cell_box[cell];
  const BoxParams& p = d.box[b];
  const int N0 = p.Ncells[0], N1 = p.Ncells[1], N2 = p.Ncells[2];
  const int lc = cell - p.cell0;
  const int cx = lc % N0, cy = (lc / N0) % N1, cz = DIM == 3 ? lc / (N0 * N1) : 0;
  // candidate range of neighbour cell `lane` (the list build's, kernel_densities.cu:52-163)
  int rs = 0, re = -1;
  if (lane < kNR) {
    const int ddx = lane % 3 - 1, ddy = lane / (3 * kNZ) - 1;
    const int ddz = DIM == 3 ? (lane / 3) % 3 - 1 : 0;
    int nx = cx + ddx, ny = cy + ddy, nz = cz + ddz;
    if (nx < 0) nx += N0;
    if (nx >= N0) nx -= N0;
    if (DIM == 3) {
      if (nz < 0) nz += N2;
      if (nz >= N2) nz -= N2;
    }
    if (!p.wall) {
      if (ny < 0) ny += N1;
      if (ny >= N1) ny -= N1;
    }
    if (ny >= 0 && ny < N1) {
      const int nc = p.cell0 + (DIM == 3 ? (nz * N1 + ny) * N0 + nx : ny * N0 + nx);
      rs = d.cell_start[nc] + p.slot0;
      re = d.cell_end[nc] + p.slot0;
    }
  }
  const int rcount = re >= rs ? re - rs + 1 : 0;
  const T L[3] = {(T)p.L[0], (T)p.L[1], (T)p.L[2]};
  const T h[3] = {(T)p.halfL[0], (T)p.halfL[1], (T)p.halfL[2]};
  const T rcutsq = (T)p.rcutsq;
  const T rcut_inv = (T)((sizeof(T) == 8 ? 3.0 : 1.0) * p.rcut_inv), cw = (T)p.cw;
  const int beg = d.cell_begin[cell], end = d.cell_begin[cell + 1];
  for (int t0 = 0; t0 < end - beg; t0 += 32) {
    const int i = beg + t0 + lane;
    const bool active = i < end;
    const V xi = active ? ld_pos<DIM>(P + i) : V{};
    const int n = active ? d.nbr_cnt[i] : 0;
    NbrIter it;
    it.init(d, active ? i : beg);
    // the next list entry not yet summed (-1: none left)
    int jn = n > 0 ? it.next() : -1;
    double dens = 0;
    auto add = [&](const V& xj) {
      const T wv = density_term<T, DIM>(xi, xj, L, h, p.wall, rcutsq, rcut_inv, cw);
      dens = dens + wv;
    };
    int k = 0;
    for (int ph = 0; ph < kPh; ++ph) {
      // tile offsets of this phase's ranges: exclusive prefix over lanes ph*9 .. ph*9+8
      const bool mine = lane >= ph * kPerPh && lane < (ph + 1) * kPerPh;
      int off = mine ? rcount : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(SPH_FULL, off, o);
        if (lane >= o) off += v;
      }
      off -= mine ? rcount : 0;
      if (mine) {
        rtab[w][lane - ph * kPerPh][0] = rs;
        rtab[w][lane - ph * kPerPh][1] = re;
        rtab[w][lane - ph * kPerPh][2] = off;
      }
      // stage the phase's ranges (coalesced), up to the tile capacity
#pragma unroll 1
      for (int q = 0; q < kPerPh; ++q) {
        const int qs = __shfl_sync(SPH_FULL, rs, ph * kPerPh + q);
        const int qn = __shfl_sync(SPH_FULL, rcount, ph * kPerPh + q);
        const int qo = __shfl_sync(SPH_FULL, off, ph * kPerPh + q);
        for (int u = lane; u < qn && qo + u < kDensTile; u += 32) {
          const V x = ld_pos<DIM>(P + qs + u);
          tx[w][qo + u] = x.x;
          ty[w][qo + u] = x.y;
          if (DIM == 3) tz[w][qo + u] = x.z;
        }
      }
      __syncwarp();
      // this lane's list entries that fall in the phase's ranges, in list order
      int qc = 0;
      int qs = rtab[w][0][0], qe = rtab[w][0][1], qo = rtab[w][0][2];
      while (k < n && jn >= 0) {
        const int j = jn;
        while (qc < kPerPh && (j < qs || j > qe)) {
          if (++qc < kPerPh) {
            qs = rtab[w][qc][0];
            qe = rtab[w][qc][1];
            qo = rtab[w][qc][2];
          }
        }
        if (qc == kPerPh) break;  // a later phase's entry
        const int t = qo + (j - qs);
        V xj;
        if (t < kDensTile) {
          xj.x = tx[w][t];
          xj.y = ty[w][t];
          xj.z = DIM == 3 ? tz[w][t] : T(0);
        } else {
          xj = ld_pos<DIM>(P + j);
        }
        add(xj);
        ++k;
        jn = k < n ? it.next() : -1;
      }
      __syncwarp();  // the tile and the range table are refilled by the next phase
    }
    // entries from no staged range: global reads, still in list order
    for (; k < n && jn >= 0; ++k) {
      add(ld_pos<DIM>(P + jn));
      jn = k + 1 < n ? it.next() : -1;
    }
    if (active) density_epilogue<T, DIM>(d, i, p, sizeof(T) == 8 ? __dmul_rn(p.cw, dens) : dens);
  }
}

// kernel_pressures.cu:13-23 (standalone, also refreshes the neighbour record)
template <typename T>
__global__ void k_pressure(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  const int ti = d.tinfo[i];
  const BoxParams& p = d.box[box_of(ti)];
  const double dens = d.dens[i];
  const double press = p.csq * (d.pos[i].w * dens - p.rho0);
  d.press[i] = press;
  if (p.dim == 3)
    write_record<T, 3>(d, i, p, ti, dens, press);
  else
    write_record<T, 2>(d, i, p, ti, dens, press);
}

// Pair pass (kernel_vel_gradients.cu:15-662 and kernel_forces.cu:15-865 in one sweep),
// one lane per particle over its neighbour list.
//
// Gather: at list position k every lane needs one neighbour record (128 B in FP64, 64 B
// in mixed precision), each at its own address.  Loaded lane by lane, one 16-byte piece
// per instruction, that is 32 separate cache lines per instruction.  Instead the warp
// copies the 32 records into shared memory cooperatively: kPieces consecutive lanes move
// the pieces of one record, so one copy instruction covers whole lines of 32 / kPieces
// records.  The copies for the next position are in flight (cp.async, double buffer)
// while the current ones are evaluated.  Each lane then reads its records
// from shared memory (row stride padded by one piece: conflict-free).
//
// What bounds the FP64 3D pass is the load/store pipe all of this goes through (81 % busy at 96^3,
// the FP64 pipe 37 %, issue 51 %): per position of a warp 32 passes for the copies of a record, 28 to
// read it and one for each shuffle or slot.  (FP64 2D, where the general pair term's chains are
// waited for: 65 %, 35 % and 54 %.)  The slots go through shared memory, three passes in place of
// eight shuffles, and records are read 16 bytes at a time: 128^3 pair pass 2.70 -> 2.51 ms FP64,
// 2.12 -> 2.06 mixed; 512 2D boxes, FP64, 2.26 -> 2.17.  With the 32-byte float 2D records the slots
// cost more than two shuffles (512 boxes 1.87 -> 1.91 ms).
//
// Launch shape of the pair pass per precision and dimension, as measured on B200.  Every pass
// evaluates one list position per step: with the fluid-fluid form of that walk, evaluating two
// positions side by side (to overlap their dependency chains) measured slower everywhere
// (float 3D at 128^3 2.41 vs 2.38 ms, FP64 2D on the 512-box ensemble 3.63 vs 3.52 ms, and on one
// 64^2 box, two warps per SM, 31.5 vs 27.9 us).
//  - kWarps: warps per block; kMinBlocks: resident blocks per SM the register allocation is held
//    to.  512 boxes, FP64 2D: 3 / 4 / 5 / 6 blocks 2.29 / 2.26 / 2.47 / 2.90 ms (spills from 5 on).
//    128^3 float 3D: 3 / 4 / 5 blocks 1.994 / 2.004 / 2.037 ms; FP64 3D: 3 (168 registers).  Float
//    2D: 2-warp blocks, 5 to 8 the same.
//  - One-box 3D contexts (k_pairs<..., ONE = true>) read the pair constants from the
//    constant bank (Dev::pc) instead of registers: 128^3 pair pass 3.59 -> 3.55 ms (FP64)
//    and 2.43 -> 2.38 ms (mixed) at the same shape.  The FP64 3D pass then fits 128
//    registers with 32 bytes of spill, but at 16 warps per SM (4 blocks of 4 warps or 8 of
//    2) it took 4.03 and 3.98 ms: the larger shared-memory carve-out leaves L1 too little
//    for the record gathers.
template <typename T, int DIM>
struct PairShape {
  using Rec = typename RecFor<T, DIM>::type;
  static constexpr bool kF64 = sizeof(T) == 8;
  static constexpr bool kF2D = !kF64 && DIM == 2;
  // the float 2D pass runs 2-warp blocks (measured 2.29 vs 2.35 ms on the 512-box ensemble;
  // the float 3D pass was slower with them, the FP64 passes unchanged)
  static constexpr int kWarps = kF2D ? 2 : 4;
  static constexpr int kMinBlocks = kF2D ? 6 : kF64 && DIM == 2 ? 4 : 3;
};

// The pair constants of a one-box context, viewed as PairParams (same layout).
template <typename T, int DIM>
__device__ __forceinline__ const PairParams<T, DIM>& one_box_params(const Dev& d) {
  static_assert(sizeof(PairParams<double, DIM>) == 12 * sizeof(double) &&
                    sizeof(PairParams<float, DIM>) == 12 * sizeof(float),
                "PairParams layout");
  if constexpr (sizeof(T) == 8)
    return *reinterpret_cast<const PairParams<T, DIM>*>(d.pc.L);
  else
    return *reinterpret_cast<const PairParams<T, DIM>*>(d.pc.Lf);
}

template <typename Rec>
struct PairStage {
  static constexpr int kPieces = (int)(sizeof(Rec) / 16);  // 16-byte pieces per record
  static constexpr int kStride = kPieces + 1;               // padded row, in pieces
  static constexpr int kPerCopy = 32 / kPieces;             // records per copy instruction
  static constexpr int kRows = 32 * kStride;                // one position, in pieces
  union Slot {
    int4 v[kPieces];
    Rec r;
  };
};

// L1: the copy allocates in L1 (.ca) or goes through L2 only (.cg).  Records are staged through
// L1, where the neighbouring warps of the SM find them again, except the 32-byte float 2D ones:
// measured, L1 / L2 only, 3.74 / 3.78 ms (FP64 3D), 2.33 / 2.44 (float 3D), 2.14 / 2.17 (FP64 2D,
// 512 boxes) and 2.29 / 2.28 (float 2D, 512 boxes).
template <bool L1>
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (L1)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
template <typename Rec>
constexpr bool kThroughL1 = !std::is_same<Rec, RecF2>::value;
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_prev() {
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
}

// Copies the records the warp's lanes list at one position into row block `buf`, lane `lane`
// one 16-byte piece per copy.  jn: this lane's slot, -1 for none; each copy's slots by a shuffle.
template <typename Rec>
__device__ __forceinline__ void stage_records(int4* buf, const Rec* __restrict__ rec, int jn,
                                              int lane) {
  using St = PairStage<Rec>;
  const int piece = lane % St::kPieces;
#pragma unroll
  for (int t = 0; t < St::kPieces; ++t) {
    const int r = t * St::kPerCopy + lane / St::kPieces;
    const int jr = __shfl_sync(SPH_FULL, jn, r);
    if (jr >= 0)
      cp_async16<kThroughL1<Rec>>(buf + r * St::kStride + piece,
                                  reinterpret_cast<const int4*>(rec + jr) + piece);
  }
}
// The same with the lanes' slots in shared memory (idx): the kPieces lanes that move a record
// move those of kPieces successive rows, whose slots they read in one or two loads.
template <typename Rec>
__device__ __forceinline__ void stage_records(int4* buf, const Rec* __restrict__ rec,
                                              const int* idx, int lane) {
  using St = PairStage<Rec>;
  constexpr int kP = St::kPieces;
  static_assert(kP % 4 == 0, "slots are read four at a time");
  const int piece = lane % kP, r0 = lane - piece;
  int j[kP];
#pragma unroll
  for (int t = 0; t < kP; t += 4) {
    const int4 v = *reinterpret_cast<const int4*>(idx + r0 + t);
    j[t] = v.x;
    j[t + 1] = v.y;
    j[t + 2] = v.z;
    j[t + 3] = v.w;
  }
#pragma unroll
  for (int t = 0; t < kP; ++t) {
    if (j[t] >= 0)
      cp_async16<kThroughL1<Rec>>(buf + (r0 + t) * St::kStride + piece,
                                  reinterpret_cast<const int4*>(rec + j[t]) + piece);
  }
}

// A staged record in a lane's registers, read 16 bytes a load.  FP64: field by field the 3D record
// took 11 loads, the 8-byte ones among them with two-way bank conflicts (pair pass 2.59 -> 2.56 ms
// at 128^3, 2.22 -> 2.17 on the 512 2D boxes).
template <typename T, typename Rec>
struct StagedRec;
template <>
struct StagedRec<double, RecD> {
  RecD r;
  __device__ __forceinline__ explicit StagedRec(const int4* src) {
    const double2* q = reinterpret_cast<const double2*>(src);
    const double2 a = q[0], b = q[1], c = q[2], e = q[3], f = q[4], g = q[5];
    const int4 h = src[6];
    r.x = a.x;
    r.y = a.y;
    r.z = b.x;
    r.vx = b.y;
    r.vy = c.x;
    r.vz = c.y;
    r.P[0] = e.x;
    r.P[1] = e.y;
    r.P[2] = f.x;
    r.P[3] = f.y;
    r.P[4] = g.x;
    r.P[5] = g.y;
    r.invd = __hiloint2double(h.y, h.x);
    r.tinfo = h.z;
  }
};
template <>
struct StagedRec<double, RecD2> {
  RecD2 r;
  __device__ __forceinline__ explicit StagedRec(const int4* src) {
    const double2* q = reinterpret_cast<const double2*>(src);
    const double2 a = q[0], b = q[1], c = q[2], e = q[3];
    r.x = a.x;
    r.y = a.y;
    r.vx = b.x;
    r.vy = b.y;
    r.P[0] = c.x;
    r.P[1] = c.y;
    r.P[2] = e.x;
    r.invd = e.y;
  }
};
template <typename Rec>
struct StagedRec<float, Rec> {
  Rec r;
  __device__ __forceinline__ explicit StagedRec(const int4* src) {
    typename PairStage<Rec>::Slot s;
#pragma unroll
    for (int t = 0; t < PairStage<Rec>::kPieces; ++t) s.v[t] = src[t];
    r = s.r;
  }
};

// Everything a lane's walk over its list needs.
template <typename T, int DIM>
struct PairWalk {
  using Rec = typename RecFor<T, DIM>::type;
  const Dev& d;
  const Rec* __restrict__ rec;
  int4* sb;                      // the warp's staging rows
  int* idx;                      // slots of two positions, 32 each
  int lane, i, n, nmax;
  const BoxParams& p;
  const PairParams<T, DIM>& pp;
  const CollView& cv;
  const PairOwn<T, DIM>& o;
};

// Passes whose slots go through shared memory (see stage_records): all but the float 2D one.
template <typename T, int DIM>
constexpr bool kSlots = DIM == 3 || sizeof(T) == 8;

// A lane's walk over its list, one position per step: the copies for position k + 1 are in
// flight while k is evaluated.  WRAP: see min_image.
template <typename T, int DIM, bool WRAP, int MODE>
__device__ __forceinline__ void pair_walk(const PairWalk<T, DIM>& W, NbrIter& it,
                                           PairAcc<T, DIM>& acc) {
  using Rec = typename RecFor<T, DIM>::type;
  using St = PairStage<Rec>;
  constexpr bool kIdx = kSlots<T, DIM>;  // slots by way of shared memory, two positions ahead
  const int n = W.n, lane = W.lane;
  int jc = n > 0 ? it.next() : -1, jn = -1, j2 = -1;
  // 2D records carry no type word: the neighbour's is read from the type array one
  // position ahead, with its record's copy
  int tc = DIM == 2 && jc >= 0 ? __ldg(&W.d.tinfo[jc]) : 0;
  if constexpr (kIdx) {
    jn = n > 1 ? it.next() : -1;
    W.idx[lane] = jc;
    W.idx[32 + lane] = jn;
    __syncwarp();
    stage_records<Rec>(W.sb, W.rec, W.idx, lane);
    __syncwarp();
  } else {
    stage_records<Rec>(W.sb, W.rec, jc, lane);
  }
  cp_async_commit();
  for (int k = 0; k < W.nmax; ++k) {
    const int k1 = k + 1;
    if constexpr (kIdx) {
      const int b1 = k1 & 1;
      if (k1 < W.nmax) stage_records<Rec>(W.sb + b1 * St::kRows, W.rec, W.idx + b1 * 32, lane);
      j2 = k + 2 < n ? it.next() : -1;
      W.idx[(b1 ^ 1) * 32 + lane] = j2;  // position k's are no longer read, k + 2's after a barrier
    } else {
      jn = k1 < n ? it.next() : -1;
      if (k1 < W.nmax) stage_records<Rec>(W.sb + (k1 & 1) * St::kRows, W.rec, jn, lane);
    }
    const int tn = DIM == 2 && jn >= 0 ? __ldg(&W.d.tinfo[jn]) : 0;
    cp_async_commit();
    cp_async_wait_prev();  // position k has landed (this lane's copies) ...
    __syncwarp();          // ... and every other lane's
    const bool valid = jc >= 0 && jc != W.i;
    const StagedRec<T, Rec> R(W.sb + (k & 1) * St::kRows + lane * St::kStride);
    int tj;
    if constexpr (DIM == 3) tj = type_of(R.r.tinfo); else tj = type_of(tc);
    // the fluid-fluid form where every lane of the warp qualifies (a warp split between the
    // forms would run both)
    if (__all_sync(SPH_FULL, W.o.fluid && (!valid || tj == 0)))
      pair_fluid_x1<T, DIM, WRAP, MODE>(W.p, W.pp, W.o, R.r, valid, acc);
    else if (valid)
      pair_term<T, DIM, WRAP>(W.p, W.pp, W.cv, W.o, R.r, tj, acc);
    __syncwarp();  // buffer k & 1 is refilled at position k + 2
    jc = jn;
    if constexpr (kIdx) jn = j2;
    tc = tn;
  }
}

template <typename T, int DIM, int MODE, bool EXT, bool ONE>
__global__ void __launch_bounds__(PairShape<T, DIM>::kWarps * 32,
                                  PairShape<T, DIM>::kMinBlocks)
    k_pairs(const __grid_constant__ Dev d) {
  using Sh = PairShape<T, DIM>;
  using Rec = typename Sh::Rec;
  using St = PairStage<Rec>;
  // per warp: a double buffer of staged positions
  __shared__ int4 stage[Sh::kWarps][2][St::kRows];
  __shared__ __align__(16) int slots[kSlots<T, DIM> ? Sh::kWarps : 1][2][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wbase = (blockIdx.x * Sh::kWarps + w) * 32;
  if (wbase >= d.Ntot) return;  // whole warps only: the lanes below cooperate
  if (step_aborted_warp(d)) return;
  // the step's count: no kernel from here on in the step looks at it (and here, not at the end,
  // it costs the float 2D pass no registers: 2.25 against 2.62 ms on the 512-box ensemble)
  if (MODE == kPairFused && d.fold_vv2 && blockIdx.x == 0 && threadIdx.x == 0) *d.step += 1;
  const int i = wbase + lane;
  const bool active = i < d.Ntot;
  const int is = active ? i : wbase;  // lanes past the end mirror a valid slot, compute nothing

  const Rec* __restrict__ rec = reinterpret_cast<const Rec*>(d.rec);
  const int ti = d.tinfo[is];
  const BoxParams& p = d.box[box_of(ti)];
  PairParams<T, DIM> ppl;
  if constexpr (!ONE) ppl.load(p);
  const PairParams<T, DIM>& pp = ONE ? one_box_params<T, DIM>(d) : ppl;
  const CollView cv{d.cs, d.ncoll};
  PairOwn<T, DIM> o;
  load_own<T, DIM, MODE>(d, is, ti, rec[is], o);
  PairAcc<T, DIM> acc;
  acc.zero();
  const int n = active ? d.nbr_cnt[i] : 0;
  int nmax = n;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) nmax = max(nmax, __shfl_xor_sync(SPH_FULL, nmax, s));
  NbrIter it;
  it.init(d, is);
  int* const idx = &slots[kSlots<T, DIM> ? w : 0][0][0];
  const PairWalk<T, DIM> W{d, rec, &stage[w][0][0], idx, lane, i, n, nmax, p, pp, cv, o};
  auto walk = [&](auto wrap_tag) {
    pair_walk<T, DIM, decltype(wrap_tag)::value, MODE>(W, it, acc);
  };
  // Warps clear of the periodic faces drop the minimum image.  Not in float 2D, where the second
  // copy of the walk cost more in instruction fetch than the shorter separations saved (small
  // boxes put both kinds of warp on every SM: 512 boxes 2.23 -> 2.38 ms); FP64 2D 2.17 -> 2.09 ms
  // on the 512 boxes, the 3D passes gain 5 %.
  if constexpr (DIM == 3 || sizeof(T) == 8) {
    if (warp_plain_image(d, clear_of_faces<T, DIM>(p, o.x, o.y, o.z)))
      walk(std::false_type{});
    else
      walk(std::true_type{});
  } else {
    walk(std::true_type{});
  }
  if (active) pair_store<T, DIM, MODE, EXT>(d, i, p, o, acc);
}

// kernel_ext_force.cu:13-73 as a separate pass (class_system::calculate_external_forces)
__global__ void k_ext_force(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  const int ti = d.tinfo[i];
  if (type_of(ti) != 0) return;
  const BoxParams& p = d.box[box_of(ti)];
  const int Np = d.Npad;
  const double4 x = d.pos[i];
  const double m = x.w;
  if (p.ext_force_type == 1) {
    d.f[i] += m * p.ext_force[0];
    d.f[Np + i] += m * p.ext_force[1];
    if (p.dim == 3) d.f[2 * Np + i] += m * p.ext_force[2];
  } else if (p.ext_force_type == 2) {
    d.f[i] += m * p.ext_force[0] * sin(p.ky * x.y);
    d.f[Np + i] += 0.0;
    if (p.dim == 3) d.f[2 * Np + i] += 0.0;
  } else if (p.ext_force_type == 3) {
    d.f[i] += (x.y < 0.5 * p.L[1]) ? m * p.ext_force[0] : -(m * p.ext_force[0]);
    d.f[Np + i] += 0.0;
    if (p.dim == 3) d.f[2 * Np + i] += 0.0;
  }
}

// dc/dt from the stored gradient (kernel_dcdt.cu:15-104), used after a standalone
// velocity-gradient pass.
__global__ void k_dcdt(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.Ntot) return;
  if (step_aborted(d)) return;
  const int ti = d.tinfo[i];
  const int Np = d.Npad;
  if (type_of(ti) != 0) {
    // kernel_dcdt.cu:39: walls and colloids keep their initial zero
    for (int q = 0; q < 6; ++q) d.dcdt[q * Np + i] = 0.0;
    return;
  }
  const BoxParams& p = d.box[box_of(ti)];
  const double tinv = 1.0 / p.tau;
  const double* G = d.gradv;
  const double cxx = d.conf[i], cxy = d.conf[Np + i], cyy = d.conf[2 * Np + i];
  const double gxx = G[i], gxy = G[Np + i], gyx = G[3 * Np + i], gyy = G[4 * Np + i];
  if (p.dim == 2) {
    const double Axx = cxx * gxx + cxy * gyx, Axy = cxx * gxy + cxy * gyy;
    const double Ayx = cxy * gxx + cyy * gyx, Ayy = cxy * gxy + cyy * gyy;
    d.dcdt[i] = 2.0 * Axx + tinv * (1.0 - cxx);
    d.dcdt[Np + i] = Axy + Ayx - tinv * cxy;
    d.dcdt[2 * Np + i] = 2.0 * Ayy + tinv * (1.0 - cyy);
    d.dcdt[3 * Np + i] = 0.0;
    d.dcdt[4 * Np + i] = 0.0;
    d.dcdt[5 * Np + i] = 0.0;
    return;
  }
  const double cxz = d.conf[3 * Np + i], cyz = d.conf[4 * Np + i], czz = d.conf[5 * Np + i];
  const double gxz = G[2 * Np + i], gyz = G[5 * Np + i], gzx = G[6 * Np + i],
               gzy = G[7 * Np + i], gzz = G[8 * Np + i];
  const double Axx = cxx * gxx + cxy * gyx + cxz * gzx;
  const double Axy = cxx * gxy + cxy * gyy + cxz * gzy;
  const double Axz = cxx * gxz + cxy * gyz + cxz * gzz;
  const double Ayx = cxy * gxx + cyy * gyx + cyz * gzx;
  const double Ayy = cxy * gxy + cyy * gyy + cyz * gzy;
  const double Ayz = cxy * gxz + cyy * gyz + cyz * gzz;
  const double Azx = cxz * gxx + cyz * gyx + czz * gzx;
  const double Azy = cxz * gxy + cyz * gyy + czz * gzy;
  const double Azz = cxz * gxz + cyz * gyz + czz * gzz;
  d.dcdt[i] = 2.0 * Axx + tinv * (1.0 - cxx);
  d.dcdt[Np + i] = Axy + Ayx - tinv * cxy;
  d.dcdt[2 * Np + i] = 2.0 * Ayy + tinv * (1.0 - cyy);
  d.dcdt[3 * Np + i] = Axz + Azx - tinv * cxz;
  d.dcdt[4 * Np + i] = Ayz + Azy - tinv * cyz;
  d.dcdt[5 * Np + i] = 2.0 * Azz + tinv * (1.0 - czz);
}

// ---------------------------------------------------------------------------------
// Wall forces (kernel_collect_force_walls.cu:15-50) and colloid forces and torques
// (kernel_collect_force_colloids.cu:15-99): one block per wall / colloid, a fixed-order
// FP64 tree reduction in place of the reference's one-thread serial loop.
// ---------------------------------------------------------------------------------
constexpr int kRedThreads = 256;

template <int NV, int NT>
__device__ __forceinline__ void block_reduce(double (&v)[NV], double (*sh)[NT]) {
#pragma unroll
  for (int q = 0; q < NV; ++q) sh[q][threadIdx.x] = v[q];
  __syncthreads();
  for (int s = NT / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s)
#pragma unroll
      for (int q = 0; q < NV; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + s];
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = sh[q][0];
}

// One block per chunk of a wall's list (kWallChunk entries at most); the last block of a wall
// to finish adds the chunks' partial sums in a fixed order.
__global__ void __launch_bounds__(kRedThreads) k_wall_forces(Dev d) {
  __shared__ double sh[3][kRedThreads];
  __shared__ int last;
  const int k = blockIdx.x;
  if (k >= d.nwallchunks) return;
  if (step_aborted(d)) return;
  const int j0 = d.wall_chunk[k], j1 = d.wall_chunk[k + 1];
  const int Np = d.Npad;
  double v[3] = {0.0, 0.0, 0.0};
  for (int j = j0 + threadIdx.x; j < j1; j += kRedThreads) {
    const int s = d.inv[d.walls_list[j]];
    v[0] += d.f[s];
    v[1] += d.f[Np + s];
    v[2] += d.f[2 * Np + s];
  }
  block_reduce<3>(v, sh);
  const int w = d.wall_of_chunk[k];
  const int c0 = d.wall_seg_chunk[w], c1 = d.wall_seg_chunk[w + 1];
  if (threadIdx.x == 0) {
    d.wall_part[3 * k + 0] = v[0];
    d.wall_part[3 * k + 1] = v[1];
    d.wall_part[3 * k + 2] = v[2];
    __threadfence();
    last = atomicAdd(&d.wall_done[w], 1) == c1 - c0 - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  const int lane = threadIdx.x;
  double u[3] = {0.0, 0.0, 0.0};
  for (int c = c0 + lane; c < c1; c += 32)
#pragma unroll
    for (int q = 0; q < 3; ++q) u[q] += __ldcg(&d.wall_part[3 * c + q]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 3; ++q) u[q] += __shfl_xor_sync(SPH_FULL, u[q], o);
  if (lane == 0) {
    d.wall_f[3 * w + 0] = u[0];
    d.wall_f[3 * w + 1] = u[1];
    d.wall_f[3 * w + 2] = u[2];
    d.wall_done[w] = 0;
  }
}

// Colloid-colloid repulsion (kernel_repulsion_force_colloids.cu:21-207, r^2 clamped to the
// cut-on before normalising) then rotating-field dipole force
// (kernel_magnetic_force_colloids.cu:15-203, 3D e scaled to |e| = R), over the coarse
// grid in the reference's order: added to F, the force on colloid c, in lane 0.
//
// A warp per colloid: lane q looks up neighbour cell q, the lanes take 32 of the neighbours in
// order at a time and evaluate their forces together, and the forces are added one by one in
// that order.  (A thread per colloid walking the cells: 0.11 ms per step of the 512-box
// ensemble and 0.079 ms on the 96^3 suspension for the collection, the pairs and the half-kick;
// 0.086 and 0.018 ms in one kernel so.)
template <int PASS>
__device__ __forceinline__ bool colloid_pair_force(const Dev& d, const BoxParams& p, int i, int j,
                                                   double (&f)[3]) {
  const int nc = d.ncoll, c0 = p.coll0;
  const double* cs = d.cs;
  const double L[3] = {p.L[0], p.L[1], p.L[2]};
  const double h[3] = {p.halfL[0], p.halfL[1], p.halfL[2]};
  double r[3] = {cs[CS_X * nc + c0 + i] - cs[CS_X * nc + c0 + j],
                 cs[CS_Y * nc + c0 + i] - cs[CS_Y * nc + c0 + j],
                 p.dim == 3 ? cs[CS_Z * nc + c0 + i] - cs[CS_Z * nc + c0 + j] : 0.0};
  if (p.dim == 3)
    min_image<double, 3>(r[0], r[1], r[2], L, h, p.wall);
  else
    min_image<double, 2>(r[0], r[1], r[2], L, h, p.wall);
  double r2 = p.dim == 3 ? r[0] * r[0] + r[1] * r[1] + r[2] * r[2] : r[0] * r[0] + r[1] * r[1];
  if (PASS == 0) {
    if (r2 < p.rcuton_coll_rep_sq) r2 = p.rcuton_coll_rep_sq;
    if (!(r2 <= p.rcutoff_coll_rep_sq)) return false;
    const double rr = sqrt(r2);
    const double ts = -p.tau_rep * (rr - 2.0 * p.coll_R) / p.coll_R;
    const double ex = exp(ts);
    const double Fm = p.F0_rep * p.tau_rep * ex / (1.0 - ex);
    for (int a = 0; a < 3; ++a) f[a] = a < p.dim ? Fm * (r[a] / rr) : 0.0;
  } else {
    if (!(r2 <= p.r0_magnet_sq)) return false;
    const double* m = d.mag + 3 * d.coll_box[c0 + i];
    const double rr = p.dim == 3 ? sqrt(r2) / p.coll_R : sqrt(r2);
    const double e[3] = {r[0] / rr, r[1] / rr, p.dim == 3 ? r[2] / rr : 0.0};
    const double me = p.dim == 3 ? m[0] * e[0] + m[1] * e[1] + m[2] * e[2]
                                 : m[0] * e[0] + m[1] * e[1];
    const double me2 = me * me;
    const double F0r4 = p.F0_magnet / (r2 * r2);
    for (int a = 0; a < 3; ++a)
      f[a] = a < p.dim ? F0r4 * (2.0 * me * m[a] - (5.0 * me2 - 1.0) * e[a]) : 0.0;
  }
  return true;
}

// Neighbour cell q of a colloid at (x, y, z) in the reference's order; -1: none.
__device__ __forceinline__ int coll_neigh_cell(const BoxParams& p, double x, double y, double z,
                                               int q) {
  const int* Nc = p.Ncells_colloids;
  const double fx = floor(x / p.cell_colloids_size[0]);
  const double fy = floor(y / p.cell_colloids_size[1]);
  const double fz = p.dim == 3 ? floor(z / p.cell_colloids_size[2]) : 0.0;
  // a colloid centre that is not finite or lies beyond one periodic image has no
  // neighbour cells (every index built below then stays inside the coarse grid)
  if (!(fx >= 1.0 - Nc[0] && fx <= 2.0 * Nc[0] - 2.0)) return -1;
  if (!(fy >= -2.0 * Nc[1] && fy <= 3.0 * Nc[1])) return -1;
  if (p.wall == 0 && !(fy >= 1.0 - Nc[1] && fy <= 2.0 * Nc[1] - 2.0)) return -1;
  if (p.dim == 3 && !(fz >= 1.0 - Nc[2] && fz <= 2.0 * Nc[2] - 2.0)) return -1;
  const int nz = p.dim == 3 ? 3 : 1;
  if (q >= 9 * nz) return -1;
  int cx = (int)fx + q / (3 * nz) - 1, cy = (int)fy + (q / nz) % 3 - 1;
  int cz = (int)fz + (p.dim == 3 ? q % 3 - 1 : 0);
  if (cx < 0) cx += Nc[0];
  if (cx >= Nc[0]) cx -= Nc[0];
  if (p.wall == 0) {
    if (cy < 0) cy += Nc[1];
    if (cy >= Nc[1]) cy -= Nc[1];
  }
  if (p.dim == 3) {
    if (cz < 0) cz += Nc[2];
    if (cz >= Nc[2]) cz -= Nc[2];
  }
  if (cy < 0 || cy >= Nc[1]) return -1;
  return p.dim == 3 ? cz * Nc[0] * Nc[1] + cy * Nc[0] + cx : cy * Nc[0] + cx;
}

__device__ __forceinline__ void colloid_pairs(const Dev& d, const BoxParams& p, int c,
                                              double (&F)[3]) {
  const int nc = d.ncoll, c0 = p.coll0, i = c - c0, lane = threadIdx.x & 31;
  const double* cs = d.cs;
  const int cell = coll_neigh_cell(p, cs[CS_X * nc + c], cs[CS_Y * nc + c], cs[CS_Z * nc + c], lane);
  int start = 0, num = 0;
  if (cell >= 0) {
    start = d.ccell_start[p.ccell0 + cell];
    num = max(d.ccell_end[p.ccell0 + cell] - start + 1, 0);
  }
  int upto = num;  // neighbours in this lane's cell and those before it
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(SPH_FULL, upto, o);
    if (lane >= o) upto += y;
  }
  const int total = __shfl_sync(SPH_FULL, upto, 31);
  auto pass = [&](auto pass_tag) {
    for (int t0 = 0; t0 < total; t0 += 32) {
      // neighbour t0 + lane: the first cell whose running count exceeds it
      const int t = t0 + lane;
      int q = 0;
      for (int l = 0; l < 31; ++l) q += __shfl_sync(SPH_FULL, upto, l) <= t ? 1 : 0;
      const int first = __shfl_sync(SPH_FULL, start, q), end = __shfl_sync(SPH_FULL, upto, q);
      const int cnt = __shfl_sync(SPH_FULL, num, q);
      double f[3] = {0.0, 0.0, 0.0};
      bool has = false;
      if (t < total) {
        const int j = d.cindex[c0 + first + (t - (end - cnt))];
        if (j != i) has = colloid_pair_force<decltype(pass_tag)::value>(d, p, i, j, f);
      }
      unsigned mask = __ballot_sync(SPH_FULL, has);
      while (mask) {
        const int l = __ffs(mask) - 1;
        mask &= mask - 1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double v = __shfl_sync(SPH_FULL, f[a], l);
          if (a < p.dim) F[a] = F[a] + v;
        }
      }
    }
  };
  pass(std::integral_constant<int, 0>{});
  pass(std::integral_constant<int, 1>{});
}

// One block per colloid.  PAIRS: then its repulsion and magnetic forces (first warp).  KICK: then
// its second half-kick (kernel_move_colloids_VV_part2.cu:14-46).  NT threads, no fewer than any
// colloid has particles or 256: the sums are then the same (the further threads of a larger block
// would add zeros).
template <bool PAIRS, bool KICK, int NT>
__global__ void __launch_bounds__(NT) k_collect_colloids(Dev d) {
  __shared__ double sh[6][NT];
  const int c = blockIdx.x;
  if (c >= d.ncoll) return;
  if (step_aborted(d)) return;
  const BoxParams& p = d.box[d.coll_box[c]];
  const int nc = d.ncoll, Np = d.Npad;
  const double cx = d.cs[CS_X * nc + c], cy = d.cs[CS_Y * nc + c], cz = d.cs[CS_Z * nc + c];
  const int j0 = d.coll_seg[c], j1 = d.coll_seg[c + 1];
  double v[6] = {0, 0, 0, 0, 0, 0};  // F x y z, T x y z
  for (int j = j0 + threadIdx.x; j < j1; j += NT) {
    const int s = d.inv[d.colloids_list[j]];
    const double4 x = d.pos[s];
    const double fx = d.f[s], fy = d.f[Np + s], fz = p.dim == 3 ? d.f[2 * Np + s] : 0.0;
    double rx = x.x - cx, ry = x.y - cy, rz = 0.0;
    if (rx > 0.5 * p.L[0]) rx -= p.L[0];
    if (rx < -0.5 * p.L[0]) rx += p.L[0];
    if (p.wall == 0) {
      if (ry > 0.5 * p.L[1]) ry -= p.L[1];
      if (ry < -0.5 * p.L[1]) ry += p.L[1];
    }
    if (p.dim == 3) {
      rz = x.z - cz;
      if (rz > 0.5 * p.L[2]) rz -= p.L[2];
      if (rz < -0.5 * p.L[2]) rz += p.L[2];
    }
    v[0] += fx;
    v[1] += fy;
    v[2] += fz;
    v[3] += ry * fz - rz * fy;
    v[4] += rz * fx - rx * fz;
    v[5] += rx * fy - ry * fx;
  }
  block_reduce<6>(v, sh);
  if (threadIdx.x >= 32) return;
  if (PAIRS && p.N_colloids >= 2) {
    if (p.dim == 2) v[2] = d.cs[CS_FZ * nc + c];
    double F[3] = {v[0], v[1], v[2]};
    colloid_pairs(d, p, c, F);
    v[0] = F[0];
    v[1] = F[1];
    v[2] = F[2];
  }
  if (threadIdx.x == 0) {
    double* cs = d.cs;
    cs[CS_FX * nc + c] = v[0];
    cs[CS_FY * nc + c] = v[1];
    cs[CS_TZ * nc + c] = v[5];
    if (p.dim == 3) {
      cs[CS_FZ * nc + c] = v[2];
      cs[CS_TX * nc + c] = v[3];
      cs[CS_TY * nc + c] = v[4];
    }
    if (KICK) vv2_colloid(d, p, c);
  }
}

// The moments alone (see set_moment): mode 0: of the next step (step + 1); mode 1: of the
// current one.
__global__ void k_advance_time(Dev d, int nboxes, int mode) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (step_aborted(d)) return;
  if (b < nboxes) set_moment(d, b, *d.step + (mode == 0 ? 1 : 0));
}

__global__ void k_count_step(Dev d) {
  if (step_aborted(d)) return;
  if (threadIdx.x == 0 && blockIdx.x == 0) *d.step += 1;
}

// Kinetic energy per box (kernel_calculate_macro_vars.cu:14-40).  Slots are cut into
// chunks that never straddle two boxes; each block sums one chunk in a fixed tree order
// and one thread per box adds its chunks in order, so the sum is reproducible.
__global__ void __launch_bounds__(kRedThreads) k_ke_partial(Dev d, double* partial) {
  __shared__ double sh[1][kRedThreads];
  const int c = blockIdx.x;
  const int lo = d.ke_chunk[c], hi = d.ke_chunk[c + 1];
  double v[1] = {0.0};
  for (int i = lo + threadIdx.x; i < hi; i += kRedThreads) {
    const double4 x = d.pos[i];
    const double4 u = d.vel[i];
    const BoxParams& p = d.box[box_of(d.tinfo[i])];
    const double v2 = p.dim == 3 ? u.x * u.x + u.y * u.y + u.z * u.z : u.x * u.x + u.y * u.y;
    v[0] += 0.5 * x.w * v2;
  }
  block_reduce<1>(v, sh);
  if (threadIdx.x == 0) partial[c] = v[0];
}

__global__ void k_ke_final(Dev d, const double* partial) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= d.nboxes) return;
  double ke = 0.0;
  for (int c = d.ke_box_chunk[b]; c < d.ke_box_chunk[b + 1]; ++c) ke += partial[c];
  d.ke[b] = ke;
}

// ---------------------------------------------------------------------------------
// Observables (no reference counterpart), one sample per box added to running sums:
//  [0] wall shear stress  -fx(top wall) / (Lx Lz), Lz = 1 in 2D (0 without walls);
//  [1] first normal-stress difference  N1 = <nkT (cxx - cyy)> over the fluid;
//  [2] chain order  <P2(e . m)> over colloid pairs closer than 2.5 R, e the unit bond and
//      m the current field direction; P2(c) = 2c^2 - 1 in 2D (cos 2 phi), (3c^2 - 1)/2 in
//      3D; 0 when no pair is that close;
//  [3] kinetic energy (k_ke_final must have run for this sample).
// Fixed-order reductions (slot chunks that never straddle boxes, then chunks in order),
// so the sums are bit-reproducible.
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(kRedThreads) k_obs_partial(Dev d, double* partial) {
  __shared__ double sh[2][kRedThreads];
  const int c = blockIdx.x;
  const int lo = d.ke_chunk[c], hi = d.ke_chunk[c + 1];
  const int Np = d.Npad;
  double v[2] = {0.0, 0.0};  // sum of nkT (cxx - cyy) over fluid, fluid count
  for (int i = lo + threadIdx.x; i < hi; i += kRedThreads) {
    const int ti = d.tinfo[i];
    if (type_of(ti) != 0) continue;
    v[0] += d.box[box_of(ti)].nkT * (d.conf[i] - d.conf[2 * Np + i]);
    v[1] += 1.0;
  }
  block_reduce<2>(v, sh);
  if (threadIdx.x == 0) {
    partial[2 * c] = v[0];
    partial[2 * c + 1] = v[1];
  }
}

__global__ void k_obs_final(Dev d, const double* partial, double* acc) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= d.nboxes) return;
  const BoxParams& p = d.box[b];
  double n1 = 0.0, nf = 0.0;
  for (int c = d.ke_box_chunk[b]; c < d.ke_box_chunk[b + 1]; ++c) {
    n1 += partial[2 * c];
    nf += partial[2 * c + 1];
  }
  n1 = nf > 0.0 ? n1 / nf : 0.0;
  double tw = 0.0;
  if (p.wall) tw = -d.wall_f[3 * (p.wall_seg0 + 1)] / (p.L[0] * (p.dim == 3 ? p.L[2] : 1.0));
  double so = 0.0;
  int npair = 0;
  const double mx = d.mag[3 * b], my = d.mag[3 * b + 1], mz = d.mag[3 * b + 2];
  const double mn = sqrt(mx * mx + my * my + mz * mz);
  const double rmax2 = (2.5 * p.coll_R) * (2.5 * p.coll_R);
  const int nc = d.ncoll, c0 = p.coll0;
  for (int a = 0; a < p.N_colloids && mn > 0.0; ++a)
    for (int e = a + 1; e < p.N_colloids; ++e) {
      double rx = d.cs[CS_X * nc + c0 + a] - d.cs[CS_X * nc + c0 + e];
      double ry = d.cs[CS_Y * nc + c0 + a] - d.cs[CS_Y * nc + c0 + e];
      double rz = p.dim == 3 ? d.cs[CS_Z * nc + c0 + a] - d.cs[CS_Z * nc + c0 + e] : 0.0;
      if (rx > p.halfL[0]) rx -= p.L[0];
      if (rx < -p.halfL[0]) rx += p.L[0];
      if (!p.wall) {
        if (ry > p.halfL[1]) ry -= p.L[1];
        if (ry < -p.halfL[1]) ry += p.L[1];
      }
      if (p.dim == 3) {
        if (rz > p.halfL[2]) rz -= p.L[2];
        if (rz < -p.halfL[2]) rz += p.L[2];
      }
      const double r2 = rx * rx + ry * ry + rz * rz;
      if (!(r2 < rmax2) || r2 <= 0.0) continue;
      const double cs = (rx * mx + ry * my + rz * mz) / (sqrt(r2) * mn);
      so += p.dim == 3 ? 1.5 * cs * cs - 0.5 : 2.0 * cs * cs - 1.0;
      ++npair;
    }
  acc[4 * b + 0] += tw;
  acc[4 * b + 1] += n1;
  acc[4 * b + 2] += npair > 0 ? so / npair : 0.0;
  acc[4 * b + 3] += d.ke[b];
}

// Field gather / scatter between slot order and original order.
__device__ __forceinline__ double* field_ptr(const Dev& d, int f, int& comp, bool& in_pos,
                                             bool& in_vel) {
  in_pos = in_vel = false;
  comp = 0;
  const int Np = d.Npad;
  switch (f) {
    case SPH_X: case SPH_Y: case SPH_Z: in_pos = true; comp = f - SPH_X; return nullptr;
    case SPH_MASS: in_pos = true; comp = 3; return nullptr;
    case SPH_VX: case SPH_VY: case SPH_VZ: in_vel = true; comp = f - SPH_VX; return nullptr;
    case SPH_FX: case SPH_FY: case SPH_FZ: return d.f + (f - SPH_FX) * Np;
    case SPH_DENS: return d.dens;
    case SPH_PRESS: return d.press;
    default: break;
  }
  if (f >= SPH_CXX && f <= SPH_CZZ) return d.conf + (f - SPH_CXX) * Np;
  if (f >= SPH_DCDT_XX && f <= SPH_DCDT_ZZ) return d.dcdt + (f - SPH_DCDT_XX) * Np;
  if (f >= SPH_GXX && f <= SPH_GZZ && d.gradv) return d.gradv + (f - SPH_GXX) * Np;
  return nullptr;
}

__global__ void k_gather_field(Dev d, int f, double* out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.Ntot) return;
  const int s = d.inv[g];
  int comp;
  bool ip, iv;
  const double* src = field_ptr(d, f, comp, ip, iv);
  double v = 0.0;
  if (ip) {
    const double4 x = d.pos[s];
    v = comp == 0 ? x.x : comp == 1 ? x.y : comp == 2 ? x.z : x.w;
  } else if (iv) {
    const double4 u = d.vel[s];
    v = comp == 0 ? u.x : comp == 1 ? u.y : u.z;
  } else if (src) {
    v = src[s];
  }
  out[g] = v;
}

__global__ void k_scatter_field(Dev d, int f, const double* in) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.Ntot) return;
  const int s = d.inv[g];
  int comp;
  bool ip, iv;
  double* dst = field_ptr(d, f, comp, ip, iv);
  const double v = in[g];
  if (ip) {
    double4 x = d.pos[s];
    if (comp == 0) x.x = v; else if (comp == 1) x.y = v; else if (comp == 2) x.z = v; else x.w = v;
    d.pos[s] = x;
    mark_outside(d);  // until the next search has looked at the new positions
  } else if (iv) {
    double4 u = d.vel[s];
    if (comp == 0) u.x = v; else if (comp == 1) u.y = v; else u.z = v;
    d.vel[s] = u;
  } else if (dst) {
    dst[s] = v;
  }
}

__global__ void k_gather_int(Dev d, const int* src, int* out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.Ntot) return;
  out[g] = src[d.inv[g]];
}

// ---------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------
namespace {
inline cudaStream_t S(const Launch& L) { return static_cast<cudaStream_t>(L.stream); }
inline int blocks(int n, int t) { return (n + t - 1) / t; }
inline int check(const Launch& L) {
  ++*L.launches;
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return 0;
  last_launch_error() = (int)e;
  return 1;
}
constexpr int kT = 128;
}  // namespace

int launch_vv1_particles(const Launch& L) {
  if (L.d.Ntot == 0) return 0;
  k_vv1_particles<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_vv1_colloids(const Launch& L) {
  if (L.d.ncoll == 0) return 0;
  k_vv1_colloids<<<L.d.ncoll, 128, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_vv1_hash(const Launch& L) {
  if (L.d.Ntot == 0) return 0;
  k_hash<true><<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_vv2(const Launch& L) {
  if (L.d.Ntot > 0) {
    k_vv2_particles<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
    if (check(L)) return 1;
  }
  if (L.d.ncoll > 0) {
    k_vv2_colloids<<<blocks(L.d.ncoll, kT), kT, 0, S(L)>>>(L.d);
    if (check(L)) return 1;
  }
  return 0;
}

int launch_hash(const Launch& L) {
  if (L.d.Ntot == 0) return 0;
  k_hash<false><<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
  return check(L);
}

// Up to kOneBlockSpans spans are scanned by one block (a second launch costs as much).
constexpr int kOneBlockSpans = 4;
int launch_cell_sort(const Launch& L, bool advance) {
  const int spans = blocks(L.d.Ctot > 0 ? L.d.Ctot : 1, kScanSpan);
  if (spans <= kOneBlockSpans) {
    k_cell_scan<<<1, kScanThreads, 0, S(L)>>>(L.d, spans, advance ? 1 : 0);
  } else {
    k_cell_sums<<<spans, kScanThreads, 0, S(L)>>>(L.d);
    if (check(L)) return 1;
    k_cell_scan<<<spans, kScanThreads, 0, S(L)>>>(L.d, 1, advance ? 1 : 0);
  }
  if (check(L)) return 1;
  if (L.d.Ntot == 0) return 0;
  k_bucket<<<blocks(L.d.Ntot, 256), 256, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_reorder(const Launch& L, bool permute_forces) {
  const int nb = blocks(L.d.Ntot, kT);
  const bool mixed = L.d.pos_f != nullptr;
  if (mixed && permute_forces) k_reorder<true, true><<<nb, kT, 0, S(L)>>>(L.d);
  else if (mixed) k_reorder<true, false><<<nb, kT, 0, S(L)>>>(L.d);
  else if (permute_forces) k_reorder<false, true><<<nb, kT, 0, S(L)>>>(L.d);
  else k_reorder<false, false><<<nb, kT, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_build_lists_dim(const Launch& L, int dim) {
  if (L.d.Ctot == 0) return 0;
  const bool half = L.list_tpc == 16;
  // Cells of more than 28 particles on average hold more than a warp's 32 here and there, and the
  // warps of those cells, with a second round, are what a small grid waits for: two warps per
  // cell, up to 64 cells per SM.  Measured in 3D (us, one / two): 4 cells per SM 41.5 / 27.9, 39
  // 82.0 / 74.6, 56 93.6 / 90.4, 60 105.0 / 99.4; 82 112.8 / 114.6, 106 134.0 / 138.8, 501 520 /
  // 566; and, with 27 per cell, 28 cells per SM, 40.9 / 50.3.
  const int split = L.d.Ntot / 28 > L.d.Ctot && L.d.Ctot <= 64 * L.nsm ? 2 : 1;
  const int nb = blocks(blocks(L.d.Ctot, half ? 2 : 1) * split, kListWarps);
  constexpr int nt = kListWarps * 32;
  if (dim == 3) {
    if (half) k_build_lists_half<3><<<nb, nt, 0, S(L)>>>(L.d, split);
    else k_build_lists<3><<<nb, nt, 0, S(L)>>>(L.d, split);
  } else {
    if (half) k_build_lists_half<2><<<nb, nt, 0, S(L)>>>(L.d, split);
    else k_build_lists<2><<<nb, nt, 0, S(L)>>>(L.d, split);
  }
  return check(L);
}

int launch_colloid_cells_n(const Launch& L, int nboxes, int max_coll) {
  if (L.d.ncoll == 0) return 0;
  k_colloid_cells<<<nboxes, 128, sizeof(int) * (max_coll > 0 ? max_coll : 1), S(L)>>>(L.d, nboxes);
  return check(L);
}

// A context of so few particles that its warps (one per 32) hardly fill the SMs: a pass then
// takes as long as one warp's walk over its lists, and what shortens the walk is work side by
// side in the warp (its registers are free), in one-warp blocks spread over all SMs.
inline bool few_warps(const Launch& L, int per_sm) { return L.d.Ntot <= 32 * per_sm * L.nsm; }

// Up to few_density warps per SM: the terms of eight list entries side by side.  Measured (us,
// two at a time / eight), FP64: 3D at 13.5 warps per SM 53.5 / 49.5, at 15.6 53.5 / 51.5, at 16.8
// 57.4 / 78.7; 2D (overlap 4) at 13.8 23.7 / 22.8, at 15.4 22.8 / 22.8, at 16.6 24.9 / 31.6 (an SM
// holds 16 of its warps).  Float: 3D at 13.5 45.2 / 39.2, at 18.0 47.4 / 45.4, at 20.6 49.5 / 50.3
// (the whole step 282 / 280), at 23.4 the step 277 / 275; 2D at 15.4 20.8 / 18.9, at 17.8 20.8 /
// 21.2, at 20.3 21.6 / 22.8 (the step 123.1 / 124.1).
// density_block 64, 128 and 256 are then one form (density_one_form).
constexpr int few_density(bool fp64, int dim) { return fp64 ? 14 : dim == 3 ? 24 : 18; }
bool density_one_form(const Launch& L, int dim) {
  return few_warps(L, few_density(L.prec == SPH_PREC_FP64, dim));
}
template <typename T, int DIM>
static void density_launch(const Launch& L) {
  if (density_one_form(L, DIM)) {
    k_density<T, DIM, 8><<<blocks(L.d.Ntot, 32), 32, 0, S(L)>>>(L.d);
  } else {
    const int nt = L.density_block;
    k_density<T, DIM, 2><<<blocks(L.d.Ntot, nt), nt, 0, S(L)>>>(L.d);
  }
}

int launch_density_dim(const Launch& L, int dim) {
  if (L.d.Ntot == 0) return 0;
  if (L.density_block == 0) {
    // neighbour-cell tiles, one warp per cell
    const int nb = blocks(L.d.Ctot, kDensWarps);
    constexpr int nt = kDensWarps * 32;
    if (L.prec == SPH_PREC_FP64) {
      if (dim == 3) k_density_cells<double, 3><<<nb, nt, 0, S(L)>>>(L.d);
      else k_density_cells<double, 2><<<nb, nt, 0, S(L)>>>(L.d);
    } else {
      if (dim == 3) k_density_cells<float, 3><<<nb, nt, 0, S(L)>>>(L.d);
      else k_density_cells<float, 2><<<nb, nt, 0, S(L)>>>(L.d);
    }
    return check(L);
  }
  if (L.prec == SPH_PREC_FP64) {
    if (dim == 3) density_launch<double, 3>(L);
    else density_launch<double, 2>(L);
  } else {
    if (dim == 3) density_launch<float, 3>(L);
    else density_launch<float, 2>(L);
  }
  return check(L);
}

int launch_pressure(const Launch& L) {
  const int nb = blocks(L.d.Ntot, kT);
  if (L.prec == SPH_PREC_FP64)
    k_pressure<double><<<nb, kT, 0, S(L)>>>(L.d);
  else
    k_pressure<float><<<nb, kT, 0, S(L)>>>(L.d);
  return check(L);
}

template <typename T, int DIM, bool ONE>
static void pairs_launch(const Launch& L, int mode, int with_ext) {
  constexpr int nt = PairShape<T, DIM>::kWarps * 32;
  const int nb = blocks(L.d.Ntot, nt);
  if (mode == kPairGradvAll)
    k_pairs<T, DIM, kPairGradvAll, false, ONE><<<nb, nt, 0, S(L)>>>(L.d);
  else if (mode == kPairForcesOnly)
    k_pairs<T, DIM, kPairForcesOnly, false, ONE><<<nb, nt, 0, S(L)>>>(L.d);
  else if (with_ext)
    k_pairs<T, DIM, kPairFused, true, ONE><<<nb, nt, 0, S(L)>>>(L.d);
  else
    k_pairs<T, DIM, kPairFused, false, ONE><<<nb, nt, 0, S(L)>>>(L.d);
}

// One-box 3D contexts take the constant-bank form; 2D ones are mostly ensembles.
template <typename T, int DIM>
static void pairs_dispatch(const Launch& L, int mode, int with_ext) {
  if (DIM == 3 && L.d.one_box)
    pairs_launch<T, DIM, DIM == 3>(L, mode, with_ext);
  else
    pairs_launch<T, DIM, false>(L, mode, with_ext);
}

int launch_pairs_dim(const Launch& L, int dim, int mode, int with_ext) {
  if (L.d.Ntot == 0) return 0;
  if (L.prec == SPH_PREC_FP64) {
    if (dim == 3) pairs_dispatch<double, 3>(L, mode, with_ext);
    else pairs_dispatch<double, 2>(L, mode, with_ext);
  } else {
    if (dim == 3) pairs_dispatch<float, 3>(L, mode, with_ext);
    else pairs_dispatch<float, 2>(L, mode, with_ext);
  }
  return check(L);
}

int launch_ext_force(const Launch& L) {
  k_ext_force<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_dcdt_from_gradv(const Launch& L) {
  k_dcdt<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_wall_forces(const Launch& L) {
  if (L.d.nwallchunks == 0) return 0;  // wall_f stays zero
  k_wall_forces<<<L.d.nwallchunks, kRedThreads, 0, S(L)>>>(L.d);
  return check(L);
}

template <int NT>
static void collect_colloids_launch(const Launch& L, int with_pairs, int kick) {
  const int nb = L.d.ncoll;
  if (with_pairs && kick) k_collect_colloids<true, true, NT><<<nb, NT, 0, S(L)>>>(L.d);
  else if (with_pairs) k_collect_colloids<true, false, NT><<<nb, NT, 0, S(L)>>>(L.d);
  else if (kick) k_collect_colloids<false, true, NT><<<nb, NT, 0, S(L)>>>(L.d);
  else k_collect_colloids<false, false, NT><<<nb, NT, 0, S(L)>>>(L.d);
}

int launch_colloid_forces(const Launch& L, int with_pairs, int kick) {
  if (L.d.ncoll == 0) return 0;
  // The smallest block that gives every particle of the largest colloid its own thread: ensembles
  // of small colloids are many blocks that each wait on a chain of loads and on the first warp's
  // pair forces, and more of them fit an SM (12,288 colloids of up to 64 particles: 0.086 ms with
  // 256 threads, 0.038 with 64).
  if (L.coll_particles <= 64) collect_colloids_launch<64>(L, with_pairs, kick);
  else if (L.coll_particles <= 128) collect_colloids_launch<128>(L, with_pairs, kick);
  else collect_colloids_launch<kRedThreads>(L, with_pairs, kick);
  return check(L);
}

int launch_advance_time(const Launch& L, int mode) {
  k_advance_time<<<blocks(L.d.nboxes, 64), 64, 0, S(L)>>>(L.d, L.d.nboxes, mode);
  return check(L);
}

int launch_count_step(const Launch& L) {
  k_count_step<<<1, 32, 0, S(L)>>>(L.d);
  return check(L);
}

int launch_kinetic_energy(const Launch& L, double* partial) {
  k_ke_partial<<<L.d.nkechunks, kRedThreads, 0, S(L)>>>(L.d, partial);
  if (check(L)) return 1;
  k_ke_final<<<blocks(L.d.nboxes, 64), 64, 0, S(L)>>>(L.d, partial);
  return check(L);
}

int launch_observe(const Launch& L, double* ke_partial, double* obs_partial, double* acc) {
  if (launch_kinetic_energy(L, ke_partial)) return 1;
  k_obs_partial<<<L.d.nkechunks, kRedThreads, 0, S(L)>>>(L.d, obs_partial);
  if (check(L)) return 1;
  k_obs_final<<<blocks(L.d.nboxes, 64), 64, 0, S(L)>>>(L.d, obs_partial, acc);
  return check(L);
}

int launch_gather_field(const Launch& L, int field, double* out) {
  k_gather_field<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d, field, out);
  return check(L);
}

int launch_scatter_field(const Launch& L, int field, const double* in) {
  k_scatter_field<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d, field, in);
  return check(L);
}

int launch_gather_int(const Launch& L, const int* src, int* out) {
  k_gather_int<<<blocks(L.d.Ntot, kT), kT, 0, S(L)>>>(L.d, src, out);
  return check(L);
}

}  // namespace sph
