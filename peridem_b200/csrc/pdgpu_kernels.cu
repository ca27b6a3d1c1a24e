// FP64 kernels of the explicit step.  This file is compiled with
// --fmad=false: every product and sum rounds separately, as in the
// reference's x86-64 build (no -march, so no FMA contraction), which keeps
// the bond-break, contact and neighbour-search decisions bit-identical to
// the reference for the same inputs.
//
// Layout in HBM: node vectors are stored with a stride of 2 doubles in 2-D
// (double2) and 4 doubles in 3-D (double4, last lane unused), so one node is
// one aligned 16- or 32-byte access; peridynamic bonds are CSR (int64 row
// offsets, int32 columns) with one broken-bit per bond in a uint32 bitmap.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "pdgpu_internal.h"
#include "pdgpu_pdl.cuh"

namespace pdgpu {

namespace {

constexpr double kPi = 3.14159265358979323846;  // M_PI
constexpr int kBlock = 256;

// util::isGreater / util::isLess with COMPARE_EPS = 1e-5
// (src/util/function.cpp:15-23, function.h:18)
__device__ __forceinline__ bool is_greater(double a, double b) {
  const double fa = fabs(a), fb = fabs(b);
  return (a - b) > ((fa < fb ? fb : fa) * 1.0e-5);
}
__device__ __forceinline__ bool is_less(double a, double b) {
  const double fa = fabs(a), fb = fabs(b);
  return (b - a) > ((fa < fb ? fb : fa) * 1.0e-5);
}

template <int DIM>
__device__ __forceinline__ void ldv(const double *__restrict__ a, int64_t i, double (&o)[3]) {
  if constexpr (DIM == 2) {
    const double2 t = reinterpret_cast<const double2 *>(a)[i];
    o[0] = t.x;
    o[1] = t.y;
    o[2] = 0.0;
  } else {
    const double2 *p = reinterpret_cast<const double2 *>(a) + 2 * i;
    const double2 t0 = p[0], t1 = p[1];
    o[0] = t0.x;
    o[1] = t0.y;
    o[2] = t1.x;
  }
}

template <int DIM>
__device__ __forceinline__ void ldg_v(const double *__restrict__ a, int64_t i, double (&o)[3]) {
  if constexpr (DIM == 2) {
    const double2 t = __ldg(reinterpret_cast<const double2 *>(a) + i);
    o[0] = t.x;
    o[1] = t.y;
    o[2] = 0.0;
  } else {
    const double2 *p = reinterpret_cast<const double2 *>(a) + 2 * i;
    const double2 t0 = __ldg(p), t1 = __ldg(p + 1);
    o[0] = t0.x;
    o[1] = t0.y;
    o[2] = t1.x;
  }
}

template <int DIM>
__device__ __forceinline__ void stv(double *__restrict__ a, int64_t i, const double (&o)[3]) {
  if constexpr (DIM == 2) {
    reinterpret_cast<double2 *>(a)[i] = make_double2(o[0], o[1]);
  } else {
    double2 *p = reinterpret_cast<double2 *>(a) + 2 * i;
    p[0] = make_double2(o[0], o[1]);
    p[1] = make_double2(o[2], 0.0);
  }
}

// util::Point::length / dot: ((x*x + y*y) + z*z); the z term is an exact
// no-op in 2-D (z = 0), so it is skipped there.
template <int DIM>
__device__ __forceinline__ double dot3(const double (&a)[3], const double (&b)[3]) {
  double s = a[0] * b[0] + a[1] * b[1];
  if constexpr (DIM == 3) s = s + a[2] * b[2];
  return s;
}
template <int DIM>
__device__ __forceinline__ double len3(const double (&a)[3]) {
  return sqrt(dot3<DIM>(a, a));
}

// J(r / horizon) of the process-wide influence function
// (influenceFn.cpp:21-23, 55-57, 86-88; material.h:431-433)
__device__ __forceinline__ double influence(const Influence &f, double r, double horizon) {
  const double q = r / horizon;
  if (f.type == PDGPU_INF_LINEAR) return f.p0 + f.p1 * q;
  if (f.type == PDGPU_INF_CONST) return f.p0;
  return f.p0 * exp(-q * q / f.p1);
}

template <int LPN>
__device__ __forceinline__ unsigned group_mask() {
  if constexpr (LPN == 32) {
    return 0xffffffffu;
  } else {
    const unsigned lane = threadIdx.x & 31u;
    return ((1u << LPN) - 1u) << (lane / LPN * LPN);
  }
}

template <int LPN>
__device__ __forceinline__ double group_sum(double v, unsigned m) {
#pragma unroll
  for (int o = LPN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(m, v, o);
  return v;
}
template <int LPN>
__device__ __forceinline__ double group_max(double v, unsigned m) {
#pragma unroll
  for (int o = LPN / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(m, v, o));
  return v;
}
template <int LPN>
__device__ __forceinline__ int64_t group_sum_i(int64_t v, unsigned m) {
#pragma unroll
  for (int o = LPN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(m, v, o);
  return v;
}

__device__ __forceinline__ void set_error(CtrlState *c, int code, int64_t info) {
  if (atomicCAS(&c->error, 0, code) == 0) c->error_info = info;
}

// non-negative doubles order like their bit patterns
__device__ __forceinline__ void atomic_max_nonneg(unsigned long long *a, double v) {
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

template <int DIM>
__device__ __forceinline__ int cell_coord(double x, const Grid &g, int d) {
  double c = floor((x - g.lo[d]) * g.inv_cell);
  if (c < 0.0) c = 0.0;
  const double hi = (double)(g.dims[d] - 1);
  if (c > hi) c = hi;
  return (int)c;
}

template <int DIM>
__device__ __forceinline__ int cell_index(const double (&p)[3], const Grid &g) {
  int c = cell_coord<DIM>(p[0], g, 0) + g.dims[0] * cell_coord<DIM>(p[1], g, 1);
  if constexpr (DIM == 3) c += g.dims[0] * g.dims[1] * cell_coord<DIM>(p[2], g, 2);
  return c;
}

// ---------------------------------------------------------------------------
// layout conversion
// ---------------------------------------------------------------------------

template <int DIM>
__global__ void k_pack(const double *__restrict__ aos3, double *__restrict__ dst, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double o[3] = {aos3[3 * i], aos3[3 * i + 1], aos3[3 * i + 2]};
  stv<DIM>(dst, i, o);
}

template <int DIM>
__global__ void k_unpack(const double *__restrict__ src, double *__restrict__ aos3, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double o[3];
  ldv<DIM>(src, i, o);
  aos3[3 * i] = o[0];
  aos3[3 * i + 1] = o[1];
  aos3[3 * i + 2] = (DIM == 3) ? o[2] : 0.0;
}

// ---------------------------------------------------------------------------
// DEMModel::applyInitialCondition (demModel.cpp:1068-1095): every node of a
// listed particle gets the IC velocity (all three components).
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void k_apply_ic(DevData d) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (!d.ic_particle[d.ptid[i]]) return;
  double o[3] = {d.ic_v[0], d.ic_v[1], d.ic_v[2]};
  stv<DIM>(d.v, i, o);
}

// ---------------------------------------------------------------------------
// DEMModel::integrateCD (demModel.cpp:349-390) and the first half of
// DEMModel::integrateVerlet (:392-424), over d_fPdCompNodes, free dofs only.
// Also folds |v| into the running maximum that the contact-search control
// reads (updateContactNeighborSearchParameters, :1862-1883).
// ---------------------------------------------------------------------------
template <int DIM, bool VERLET>
__global__ void __launch_bounds__(kBlock) k_integrate(DevData d) {
  __shared__ double smax[kBlock / 32];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double vm = 0.0;
  if (i < d.n_nodes && (d.flags[i] & NODE_ACTIVE) && !d.ctrl->error) {
    const double rho = d.particles[d.ptid[i]].density;
    const uint8_t fix = d.fix[i];
    double v[3], u[3], x[3], f[3];
    ldv<DIM>(d.v, i, v);
    ldv<DIM>(d.u, i, u);
    ldv<DIM>(d.x, i, x);
    ldv<DIM>(d.f, i, f);
    const double dt = d.dt;
    const double k = VERLET ? 0.5 * (dt / rho) : dt / rho;
#pragma unroll
    for (int dof = 0; dof < DIM; dof++) {
      if (!((fix >> dof) & 1u)) {
        v[dof] += k * f[dof];
        u[dof] += dt * v[dof];
        x[dof] += dt * v[dof];
      }
    }
    stv<DIM>(d.v, i, v);
    stv<DIM>(d.u, i, u);
    stv<DIM>(d.x, i, x);
    vm = len3<DIM>(v);
    d.vmag[i] = vm;
  }
  // block max of |v| -> one atomic per block
  for (int o = 16; o > 0; o >>= 1) vm = fmax(vm, __shfl_xor_sync(0xffffffffu, vm, o));
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = vm;
  __syncthreads();
  if (threadIdx.x < 32) {
    double m = threadIdx.x < kBlock / 32 ? smax[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0 && m > 0.0) atomic_max_nonneg(&d.ctrl->vmax_bits, m);
  }
}

// second half kick of DEMModel::integrateVerlet (:436-459)
template <int DIM>
__global__ void k_verlet_second(DevData d) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes || !(d.flags[i] & NODE_ACTIVE) || d.ctrl->error) return;
  const double rho = d.particles[d.ptid[i]].density;
  const uint8_t fix = d.fix[i];
  double v[3], f[3];
  ldv<DIM>(d.v, i, v);
  ldv<DIM>(d.f, i, f);
  const double k = 0.5 * (d.dt / rho);
#pragma unroll
  for (int dof = 0; dof < DIM; dof++)
    if (!((fix >> dof) & 1u)) v[dof] += k * f[dof];
  stv<DIM>(d.v, i, v);
  d.vmag[i] = len3<DIM>(v);
}

// ---------------------------------------------------------------------------
// Step control (one thread): time advance (integrateCD :381-383) and the
// contact-list update decision of
// DEMModel::updateContactNeighborSearchParameters (demModel.cpp:1808-1955).
// mode 0: a time step; 1: the computeForces call of the integrate() prelude;
// 2: the contact list build of DEMModel::init.
// ---------------------------------------------------------------------------
// the fields the step control changes, written back in one go
__device__ __forceinline__ void ctrl_commit(CtrlState *dst, const CtrlState &c) {
  dst->n = c.n;
  dst->time = c.time;
  dst->first_bc = c.first_bc;
  dst->init_calls = c.init_calls;
  dst->counter = c.counter;
  dst->interval = c.interval;
  dst->radius = c.radius;
  dst->max_velocity = c.max_velocity;
  dst->update = c.update;
  dst->sur_check = c.sur_check;
}

// pre: a copy of the state taken earlier in the same kernel (its fields are
// written only here), or null to read it now
__device__ __noinline__ void ctrl_step(const DevData &d, int mode, const CtrlState *pre = nullptr) {
  CtrlState *cp = d.ctrl;
  CtrlState c = pre ? *pre : *cp;  // one pass over the state instead of a chain of loads
  if (c.error) return;
  if (mode == 0) {
    c.n += 1;
    c.time += d.dt;
    c.first_bc = 0;
  }
  // learned surrogate: every sur_interval-th step (and the first) re-judges
  // it with the full bond loop
  c.sur_check = d.sur_interval > 0 && (c.n % d.sur_interval == 0 || c.n <= 1);
  // read and reset atomically: other CTAs raised it with atomicMax
  const double vmax_now =
      fmax(__longlong_as_double((long long)atomicExch(&cp->vmax_bits, 0ull)), c.static_vmax);
  if (!d.n_zones) {  // single particle: no contact
    c.update = 0;
    ctrl_commit(cp, c);
    return;
  }
  const int64_t n = c.n;
  if (n == 0) {
    c.init_calls += 1;
    if (c.init_calls == 1) {
      c.update = 1;
      ctrl_commit(cp, c);
      return;
    }
    if (c.init_calls == 2) {
      c.counter += 1;
      c.update = ((c.counter - 1) % c.interval) == 0;
      ctrl_commit(cp, c);
      return;
    }
  }
  // restart: the counter of the restart step (demModel.cpp:1833-1837)
  if (d.restart_step >= 0 && n == d.restart_step) c.counter = n % c.interval;
  if (c.interval == 1) {
    c.radius = d.max_contact_r;
    c.counter += 1;
    c.update = ((c.counter - 1) % c.interval) == 0;
    ctrl_commit(cp, c);
    return;
  }
  const int64_t upi = c.interval > 5 ? (int64_t)(0.2 * (double)c.interval) : 1;
  if (c.counter > 0 && c.counter % upi != 0) {
    c.counter += 1;
    c.update = ((c.counter - 1) % c.interval) == 0;
    ctrl_commit(cp, c);
    return;
  }
  c.max_velocity = vmax_now;
  const double safety = d.search_factor > 5 ? d.search_factor : 10.0;
  const double r_contact = d.search_factor * d.max_contact_r;
  const double r_vel = c.max_velocity * d.dt * (double)d.search_interval * safety;
  if (is_greater(r_vel, r_contact)) {
    c.interval = (int64_t)(d.max_contact_r / (c.max_velocity * d.dt));
    c.radius = r_contact;
    c.counter = 0;
    if (c.interval < 1) {
      c.interval = 1;
      c.radius = d.max_contact_r;
    }
  } else {
    c.radius = c.interval < 2 ? d.max_contact_r : r_contact;
  }
  c.counter += 1;
  c.update = ((c.counter - 1) % c.interval) == 0;
  ctrl_commit(cp, c);
}

__global__ void k_ctrl(const __grid_constant__ DevData d, int mode) { ctrl_step(d, mode); }


// ---------------------------------------------------------------------------
// DEMModel::computeExternalDisplacementBC -> ParticleULoading::apply
// (particleULoading.cpp:115-230).  One thread per BC node applies that node's
// sets in deck order; the spatial factor of each (node, set) is precomputed
// on the host from the reference configuration.
// ---------------------------------------------------------------------------
template <int DIM>
__device__ __noinline__ void apply_ubc(const DevData &d, int t, int64_t i, double time, int first,
                                          double (&u)[3], double (&v)[3], double (&x)[3]) {
  double xr[3];
  ldg_v<DIM>(d.xref, i, xr);
  for (int e = d.ubc_row[t]; e < d.ubc_row[t + 1]; e++) {
    if (d.ubc_once[e] && !first) continue;
    const BcSetDev bc = d.ubc_sets[d.ubc_set[e]];
    const double umax = d.ubc_val[e];
    double du = 0.0, dv = 0.0;
    switch (bc.time_fn) {
      case PDGPU_TIME_CONSTANT: du = umax; break;
      case PDGPU_TIME_LINEAR: du = umax * time; dv = umax; break;
      case PDGPU_TIME_QUADRATIC:
        du = umax * time + bc.tp[1] * time * time;
        dv = umax + bc.tp[1] * time;
        break;
      case PDGPU_TIME_SIN: {
        const double a = kPi * bc.tp[1];
        du = umax * sin(a * time);
        dv = umax * a * cos(a * time);
        break;
      }
      default: break;
    }
    double ui[3] = {0.0, 0.0, 0.0}, vi[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < 3; q++)
      if ((bc.dir_mask >> q) & 1) {
        ui[q] = du;
        vi[q] = dv;
      }
    if (bc.time_fn == PDGPU_TIME_ROTATION) {
      const double dx0 = xr[0] - bc.tp[1], dx1 = xr[1] - bc.tp[2];
      const double th = bc.tp[0] * time;
      const double ct = cos(th), st = sin(th);
      // util::rotate2D / derRotate2D (transformation.cpp:53-65)
      const double r0 = dx0 * ct - dx1 * st, r1 = dx0 * st + dx1 * ct;
      const double d0 = -dx0 * st - dx1 * ct, d1 = dx0 * ct - dx1 * st;
      ui[0] += r0 - dx0;
      ui[1] += r1 - dx1;
      ui[2] += 0.0 - (xr[2] - bc.tp[3]);
      vi[0] += bc.tp[0] * d0;
      vi[1] += bc.tp[0] * d1;
      vi[2] += bc.tp[0] * 0.0;
    }
    for (int q = 0; q < DIM; q++)
      if ((bc.dir_mask >> q) & 1) {
        u[q] = ui[q];
        v[q] = vi[q];
        x[q] = ui[q] + xr[q];
      }
  }
}

template <int DIM>
__global__ void k_bc(const __grid_constant__ DevData d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.n_ubc_nodes || d.ctrl->error) return;
  const int64_t i = d.ubc_node[t];
  double u[3], v[3], x[3];
  ldv<DIM>(d.u, i, u);
  ldv<DIM>(d.v, i, v);
  ldv<DIM>(d.x, i, x);
  apply_ubc<DIM>(d, t, i, d.ctrl->time, d.ctrl->first_bc, u, v, x);
  stv<DIM>(d.u, i, u);
  stv<DIM>(d.v, i, v);
  stv<DIM>(d.x, i, x);
}

// ---------------------------------------------------------------------------
// First kernel of a step: integrateCD / the first Verlet half (as k_integrate),
// then the displacement BC of each BC node at the step's new time (as k_bc
// after k_ctrl: zero-displacement sets are not re-applied), then — in the
// last CTA to finish — the step control (as k_ctrl, mode 0).
// ---------------------------------------------------------------------------
constexpr int kBeginNodes = 2;  // nodes per thread of the step-begin kernel

template <int DIM, bool VERLET>
__global__ void __launch_bounds__(kBlock) k_step_begin(const __grid_constant__ DevData d) {
  __shared__ double smax[kBlock / 32];
  __shared__ int last;
  __shared__ __align__(8) CtrlState s_ctrl;
  static_assert(sizeof(CtrlState) % 8 == 0 && sizeof(CtrlState) / 8 <= kBlock, "CtrlState copy");
  pdl_start();
  // CTAs run in reverse node order: the boundary-condition nodes (walls, at
  // the end of the node array) then start in the first wave.  Each thread
  // takes kBeginNodes nodes, kBlock apart, and issues every load of all of
  // them before the first update; what no kernel writes, ahead of the wait.
  const int64_t base = (int64_t)(gridDim.x - 1 - blockIdx.x) * (kBlock * kBeginNodes) + threadIdx.x;
  uint8_t fl[kBeginNodes], fix[kBeginNodes];
  int32_t pid[kBeginNodes];
#pragma unroll
  for (int k = 0; k < kBeginNodes; k++) {
    const int64_t i = base + (int64_t)k * kBlock;
    fl[k] = 0;
    if (i < d.n_nodes) {
      fl[k] = d.flags[i];
      fix[k] = d.fix[i];
      pid[k] = d.ptid[i];
    }
  }
  pdl_wait();
  // every block copies the step-control state now, while its nodes load: the
  // last block's step control then starts without a chain of cold loads
  if (threadIdx.x < sizeof(CtrlState) / 8)
    reinterpret_cast<uint64_t *>(&s_ctrl)[threadIdx.x] = reinterpret_cast<const uint64_t *>(d.ctrl)[threadIdx.x];
  double vm = 0.0;
  if (!d.ctrl->error) {
    double v[kBeginNodes][3], u[kBeginNodes][3], x[kBeginNodes][3], f[kBeginNodes][3];
#pragma unroll
    for (int k = 0; k < kBeginNodes; k++) {
      const int64_t i = base + (int64_t)k * kBlock;
      if (i < d.n_nodes) {
        ldv<DIM>(d.v, i, v[k]);
        ldv<DIM>(d.u, i, u[k]);
        ldv<DIM>(d.x, i, x[k]);
        ldv<DIM>(d.f, i, f[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < kBeginNodes; k++) {
      const int64_t i = base + (int64_t)k * kBlock;
      if (!(fl[k] & (NODE_ACTIVE | NODE_UBC))) continue;
      if (fl[k] & NODE_ACTIVE) {
        const double rho = d.particles[pid[k]].density;
        const double dt = d.dt;
        const double kk = VERLET ? 0.5 * (dt / rho) : dt / rho;
#pragma unroll
        for (int dof = 0; dof < DIM; dof++) {
          if (!((fix[k] >> dof) & 1u)) {
            v[k][dof] += kk * f[k][dof];
            u[k][dof] += dt * v[k][dof];
            x[k][dof] += dt * v[k][dof];
          }
        }
        const double m = len3<DIM>(v[k]);
        vm = fmax(vm, m);
        d.vmag[i] = m;
      }
      // the step control advances time by dt before the BC pass (through
      // copies: only they have their address taken, so the per-node arrays
      // stay in registers)
      if (fl[k] & NODE_UBC) {
        double ub[3], vb[3], xb[3];
#pragma unroll
        for (int q = 0; q < 3; q++) ub[q] = u[k][q], vb[q] = v[k][q], xb[q] = x[k][q];
        apply_ubc<DIM>(d, d.ubc_of[i], i, d.ctrl->time + d.dt, 0, ub, vb, xb);
#pragma unroll
        for (int q = 0; q < 3; q++) u[k][q] = ub[q], v[k][q] = vb[q], x[k][q] = xb[q];
      }
      stv<DIM>(d.v, i, v[k]);
      stv<DIM>(d.u, i, u[k]);
      stv<DIM>(d.x, i, x[k]);
    }
  }
  // block max of |v| -> one atomic per block
  for (int o = 16; o > 0; o >>= 1) vm = fmax(vm, __shfl_xor_sync(0xffffffffu, vm, o));
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = vm;
  __syncthreads();
  if (threadIdx.x < 32) {
    double m = threadIdx.x < kBlock / 32 ? smax[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) {
      if (m > 0.0) atomic_max_nonneg(&d.ctrl->vmax_bits, m);
      __threadfence();
      last = atomicAdd(&d.ctrl->begin_done, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    d.ctrl->begin_done = 0u;
    ctrl_step(d, 0, &s_ctrl);
  }
}

// ---------------------------------------------------------------------------
// Contact candidate lists: DEMModel::updateContactNeighborlist
// (demModel.cpp:1696-1756) with the kd-tree exclude-tag radius search
// (nsearch.h:278-301; strict  sum_d (q_d - p_d)^2 < r*r  of
// nanoflann.hpp:611-621 / nflannSetup.h:272) replaced by a cell list.
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void k_cell_count(DevData d, const double *__restrict__ pos, Grid g) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (d.ctrl->error || !d.ctrl->update) return;
  double p[3];
  ldv<DIM>(pos, i, p);
  const int c = cell_index<DIM>(p, g);
  d.cell_of[i] = c;
  atomicAdd(d.cell_cnt + c, 1);
}

__global__ void k_cell_scatter(DevData d) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (d.ctrl->error || !d.ctrl->update) return;
  const int c = d.cell_of[i];
  const int pos = d.cell_start[c] + atomicAdd(d.cell_fill + c, 1);
  d.cell_tmp[pos] = (int32_t)i;
}

// one warp per cell: order the cell's nodes by index (rank counting), so
// candidate lists do not depend on atomic arrival order
__global__ void k_cell_sort(DevData d) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= d.grid.ncells) return;
  if (d.ctrl->error || !d.ctrl->update) return;
  const int s = d.cell_start[c], e = d.cell_start[c + 1];
  for (int a = s + lane; a < e; a += 32) {
    const int32_t va = d.cell_tmp[a];
    int rank = 0;
    for (int b = s; b < e; b++) rank += d.cell_tmp[b] < va;
    d.cell_nodes[s + rank] = va;
  }
  if (lane == 0) d.cell_fill[c] = 0;
}

__global__ void k_zero_cells(DevData d) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > d.grid.ncells) return;
  if (!d.ctrl->update) return;
  d.cell_cnt[c] = 0;
}





// ---------------------------------------------------------------------------
// The whole contact-list rebuild as one cooperative launch: every phase is
// separated by a grid-wide barrier of the cooperative launch (all blocks are
// co-resident by construction).  On steps without a rebuild every block
// returns after reading the control word, so the rebuild costs one launch.
// ---------------------------------------------------------------------------
namespace cg = cooperative_groups;
constexpr int kCoopBlock = 256;

// Grid-wide barrier with a bounded wait: thread 0 of each block arrives on
// a counter in the step-control state; the last to arrive resets it and
// advances the generation the others poll.  All blocks of the cooperative
// launch are resident, so the wait ends unless a block faulted; after
// d.bar_wait_ns of the GPU's global timer (30 s by default, far beyond any phase)
// the block records DEV_ERR_BARRIER_TIMEOUT and every block leaves the
// rebuild at its next barrier (the step's later kernels see the error word
// and do nothing).  Returns false when the rebuild must stop.
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ bool grid_bar(const DevData &d) {
  __shared__ int s_ok;
  CtrlState *c = d.ctrl;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *gen = &c->bar_gen;
    const unsigned g0 = *gen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(&c->bar_count, 1u) == gridDim.x - 1) {
      atomicExch(&c->bar_count, 0u);
      __threadfence();
      atomicAdd(&c->bar_gen, 1u);
    } else {
      const unsigned long long t0 = global_ns(), limit = d.bar_wait_ns;
      const unsigned every = limit ? 255u : 0u;
      unsigned polls = 0;
      while (*gen == g0) {
        // the clock is read every 256 polls (a limit of 0: at the first); the
        // poll count is a second, clock-independent bound (2^31 polls of at
        // least a few ns each)
        if ((++polls & every) == 0 && (global_ns() - t0 >= limit || polls > (1u << 31))) {
          ok = 0;
          atomicCAS(&c->error, 0, DEV_ERR_BARRIER_TIMEOUT);
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
    s_ok = ok && !((volatile int *)&c->error)[0];
  }
  __syncthreads();
  return s_ok != 0;
}

// exclusive scan over the whole grid: out[i] = sum_{k<i} in(k) for
// i = 0..n, each block scanning one contiguous chunk; false when a barrier
// gave up
template <class Tout, class F>
__device__ bool grid_scan(const DevData &d, F in, Tout *out, int64_t n, int64_t *bsum) {
  __shared__ int64_t wsum[kCoopBlock / 32];
  __shared__ int64_t carry;
  const int64_t nb = gridDim.x;
  const int64_t chunk = (n + nb - 1) / nb;
  const int64_t b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // block totals
  int64_t t = 0;
  for (int64_t k = b0 + threadIdx.x; k < b1; k += blockDim.x) t += (int64_t)in(k);
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) wsum[warp] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t s = 0;
    for (int w = 0; w < kCoopBlock / 32; w++) s += wsum[w];
    bsum[blockIdx.x] = s;
  }
  if (!grid_bar(d)) return false;
  {
    // carry = sum of the earlier blocks' totals, summed by the whole block
    // (integers: any order gives the same sum); read past L1, which may
    // hold this array from an earlier scan of the same launch
    int64_t s = 0;
    for (int64_t b = threadIdx.x; b < blockIdx.x; b += blockDim.x) s += __ldcg(bsum + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) wsum[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      int64_t c = 0;
      for (int w = 0; w < kCoopBlock / 32; w++) c += wsum[w];
      carry = c;
    }
    __syncthreads();
  }
  for (int64_t base = b0; base < b1; base += blockDim.x) {
    const int64_t k = base + threadIdx.x;
    const int64_t v = k < b1 ? (int64_t)in(k) : 0;
    int64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int64_t woff = 0;
    for (int w = 0; w < warp; w++) woff += wsum[w];
    if (k < b1) out[k] = (Tout)(carry + woff + incl - v);
    __syncthreads();
    if (threadIdx.x == 0) {
      int64_t s = 0;
      for (int w = 0; w < kCoopBlock / 32; w++) s += wsum[w];
      carry += s;
    }
    __syncthreads();
  }
  if (blockIdx.x == nb - 1 && threadIdx.x == 0) out[n] = (Tout)carry;
  return grid_bar(d);
}


// Exclusive scans of the candidate counts and of the nodes that have any, in
// one pass over the nodes: emit(i, count, row start, compacted position); the
// last block's totals go to tot[0], tot[1].  bsum: 2 values per block.
template <class Emit>
__device__ bool scan_rows(const DevData &d, const int64_t *cnt, int64_t n, int64_t *bsum, int64_t (&tot)[2], Emit emit) {
  __shared__ int64_t wsum[2][kCoopBlock / 32];
  __shared__ int64_t carry[2];
  const int64_t nb = gridDim.x;
  const int64_t chunk = (n + nb - 1) / nb;
  const int64_t b0 = min(n, blockIdx.x * chunk), b1 = min(n, b0 + chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // sum of two values over the block, in t[0], t[1] of thread 0
  auto block_sum = [&](int64_t (&t)[2]) {
#pragma unroll
    for (int q = 0; q < 2; q++) {
      for (int o = 16; o > 0; o >>= 1) t[q] += __shfl_xor_sync(0xffffffffu, t[q], o);
      if (lane == 0) wsum[q][warp] = t[q];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 0; q < 2; q++) {
        t[q] = 0;
        for (int w = 0; w < kCoopBlock / 32; w++) t[q] += wsum[q][w];
      }
  };
  int64_t t[2] = {0, 0};
  for (int64_t k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
    const int64_t c = cnt[k];
    t[0] += c;
    t[1] += c > 0;
  }
  block_sum(t);
  if (threadIdx.x == 0) {
    bsum[2 * blockIdx.x] = t[0];
    bsum[2 * blockIdx.x + 1] = t[1];
  }
  if (!grid_bar(d)) return false;
  // carry = sum of the earlier blocks' totals (integers: any order gives the
  // same sum), read past L1, which may hold this array from an earlier scan
  t[0] = t[1] = 0;
  for (int64_t k = threadIdx.x; k < blockIdx.x; k += blockDim.x) {
    t[0] += __ldcg(bsum + 2 * k);
    t[1] += __ldcg(bsum + 2 * k + 1);
  }
  block_sum(t);
  if (threadIdx.x == 0) carry[0] = t[0], carry[1] = t[1];
  __syncthreads();
  for (int64_t base = b0; base < b1; base += blockDim.x) {
    const int64_t k = base + threadIdx.x;
    const int64_t v[2] = {k < b1 ? cnt[k] : 0, k < b1 && cnt[k] > 0 ? 1 : 0};
    int64_t incl[2] = {v[0], v[1]};
#pragma unroll
    for (int q = 0; q < 2; q++) {
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl[q], o);
        if (lane >= o) incl[q] += y;
      }
      if (lane == 31) wsum[q][warp] = incl[q];
    }
    __syncthreads();
    int64_t off[2] = {carry[0], carry[1]};
    for (int w = 0; w < warp; w++) off[0] += wsum[0][w], off[1] += wsum[1][w];
    if (k < b1) emit(k, v[0], off[0] + incl[0] - v[0], off[1] + incl[1] - v[1]);
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < kCoopBlock / 32; w++) carry[0] += wsum[0][w], carry[1] += wsum[1][w];
    __syncthreads();
  }
  tot[0] = carry[0];
  tot[1] = carry[1];
  return true;
}

// Candidate search: the nodes of the 3^DIM cells around a node's own (z, y, x
// ascending; each cell's nodes ascending), those of its own particle skipped,
// with the strict test sum_d (q_d - p_d)^2 < r^2 (nanoflann's L2 order).  A cell
// whose nodes all belong to the searching node's particle is skipped whole
// (cell_pid).  Particle and position of the nodes are read in cell order
// (cell_p, cell_x), so an entry costs one round of loads.
//
// Count pass: LPN lanes per node, nodes in cell order, so that the groups of a
// warp walk the same few cells and read the same entries.  Bound by the latency
// of its loads at 1 024 threads per SM.  Against a warp per cell with the
// neighbourhood staged in shared memory (B200, us): 2-D, 332 000 nodes 82 -> 30
// (1 / 4 / 8 lanes per node: 40 / 37 / 58), 1.3 M nodes 176 -> 92; 3-D, 244 000
// nodes 82 -> 50 (8 lanes 85, 16 lanes 142), 95 000 nodes 78 -> 30.
constexpr int kCandLanes2 = 2, kCandLanes3 = 4;

template <int DIM, int LPN>
__device__ void cand_count(const DevData &d, uint8_t search_bit) {
  constexpr int kUnroll = 4;
  const Grid G = d.grid;
  const double r = d.ctrl->radius;
  const double r2 = r * r;
  const int sub = threadIdx.x % LPN;
  const int64_t groups = (int64_t)gridDim.x * blockDim.x / LPN;
  // all lanes of a warp stay in the loop together
  for (int64_t a0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x - (threadIdx.x & 31)) / LPN; a0 < d.n_nodes;
       a0 += groups) {
    const int64_t a = a0 + (threadIdx.x & 31) / LPN;
    int64_t n = 0;
    int32_t i = -1;
    if (a < d.n_nodes) {
      i = d.cell_nodes[a];
      const int cell0 = d.cell_of[i];
      if (d.flags[i] & search_bit) {
        double q[3];
        ldv<DIM>(d.cell_x, a, q);
        const int32_t pi = d.cell_p[a];
        const int cx0 = cell0 % G.dims[0], cy0 = cell0 / G.dims[0] % G.dims[1];
        const int cz0 = DIM == 3 ? cell0 / G.dims[0] / G.dims[1] : 0;
        const int zlo = DIM == 3 ? max(cz0 - 1, 0) : 0, zhi = DIM == 3 ? min(cz0 + 1, G.dims[2] - 1) : 0;
        for (int cz = zlo; cz <= zhi; cz++)
          for (int cy = max(cy0 - 1, 0); cy <= min(cy0 + 1, G.dims[1] - 1); cy++)
            for (int cx = max(cx0 - 1, 0); cx <= min(cx0 + 1, G.dims[0] - 1); cx++) {
              const int cell = cx + G.dims[0] * (cy + G.dims[1] * cz);
              if (d.cell_pid[cell] == pi) continue;
              const int e = d.cell_start[cell + 1];
              for (int b = d.cell_start[cell] + sub; b < e; b += LPN * kUnroll) {
                int32_t pb[kUnroll];
                double pos[kUnroll][3];
#pragma unroll
                for (int k = 0; k < kUnroll; k++) {
                  const int c = min(b + k * LPN, e - 1);
                  pb[k] = b + k * LPN < e ? d.cell_p[c] : pi;
                  ldv<DIM>(d.cell_x, c, pos[k]);
                }
#pragma unroll
                for (int k = 0; k < kUnroll; k++) {
                  double dd = 0.0;
#pragma unroll
                  for (int t = 0; t < DIM; t++) {
                    const double df = q[t] - pos[k][t];
                    dd += df * df;
                  }
                  n += pb[k] != pi && dd < r2;
                }
              }
            }
      }
    }
    __syncwarp();
    for (int o = LPN / 2; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (i >= 0 && sub == 0) d.c_cnt[i] = n;
  }
}

// Fill pass over the nodes that have candidates (c_nodes[0, nn)): a warp per
// node walks the same neighbourhood in the same order as the count pass and
// writes the columns.  Lane t first takes neighbour cell t (empty when it
// lies outside the grid or holds only nodes of this node's particle); the
// cells' node ranges, concatenated in traversal order, are then walked 32
// entries at a time, two groups in flight.
template <int DIM>
__device__ void cand_fill_nodes(const DevData &d, int64_t nn) {
  constexpr int kNb = DIM == 3 ? 27 : 9;
  const Grid G = d.grid;
  const double r = d.ctrl->radius;
  const double r2 = r * r;
  const int l32 = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (kCoopBlock / 32);
  for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nn; t += nwarps) {
    const int32_t i = d.c_nodes[t];
    const int2 sp = d.c_span[t];
    double q[3];
    ldv<DIM>(d.x, i, q);
    const int32_t pi = d.ptid[i];
    const int cell0 = d.cell_of[i];
    int64_t out = sp.x;
    const int64_t out_end = min((int64_t)sp.y, d.contact_cap);
    for (int64_t e = out + l32; e < out_end; e += 32) d.c_own[e] = i;
    const int cx0 = cell0 % G.dims[0], cy0 = cell0 / G.dims[0] % G.dims[1];
    const int cz0 = DIM == 3 ? cell0 / G.dims[0] / G.dims[1] : 0;
    int a = 0, cnt = 0;
    if (l32 < kNb) {
      const int cx = cx0 + l32 % 3 - 1, cy = cy0 + (l32 / 3) % 3 - 1, cz = DIM == 3 ? cz0 + l32 / 9 - 1 : 0;
      if (cx >= 0 && cx < G.dims[0] && cy >= 0 && cy < G.dims[1] && cz >= 0 && cz < (DIM == 3 ? G.dims[2] : 1)) {
        const int cell = cx + G.dims[0] * (cy + G.dims[1] * cz);
        if (d.cell_pid[cell] != pi) {  // a cell of this node's particle only holds no candidate
          a = d.cell_start[cell];
          cnt = d.cell_start[cell + 1] - a;
        }
      }
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (l32 >= o) incl += y;
    }
    int inc[kNb];
#pragma unroll
    for (int c = 0; c < kNb; c++) inc[c] = __shfl_sync(0xffffffffu, incl, c);
    const int total = inc[kNb - 1];
    for (int base = 0; base < total && out < out_end; base += 64) {
      int at[2];
      bool hit[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int g = base + 32 * h + l32;
        int k = 0;
#pragma unroll
        for (int c = 0; c < kNb; c++) k += inc[c] <= g;
        const int ak = __shfl_sync(0xffffffffu, a, k & 31);
        const int ek = __shfl_sync(0xffffffffu, incl - cnt, k & 31);
        at[h] = ak + (g - ek);
        hit[h] = g < total;
      }
      int32_t pb[2] = {pi, pi};
      double pos[2][3];
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (hit[h]) {
          pb[h] = d.cell_p[at[h]];
          ldv<DIM>(d.cell_x, at[h], pos[h]);
        }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if (hit[h]) {
          double dd = 0.0;
#pragma unroll
          for (int u = 0; u < DIM; u++) {
            const double df = q[u] - pos[h][u];
            dd += df * df;
          }
          hit[h] = pb[h] != pi && dd < r2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, hit[h]);
        const int64_t to = out + __popc(bal & ((1u << l32) - 1u));
        if (hit[h] && to < out_end) d.c_col[to] = d.cell_nodes[at[h]];
        out += __popc(bal);
      }
    }
  }
}

// The learned surrogate's list of the tiles the bond loop runs this step:
// those of the particles not on the surrogate (sur_on && !sur_near is the
// test the surrogate's scatter applies).  The order follows the atomic
// claims; each tile's forces do not depend on it.
__device__ void list_live_tiles(const DevData &d) {
  if (!d.tile_live) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < d.n_tile_live_src; t += gridDim.x * blockDim.x) {
    const int p = d.tile_particle[t];
    if (d.sur_on[p] && !d.sur_near[p]) continue;
    const unsigned k = atomicAdd(d.tile_live_n, 1u);
    if (k < (unsigned)d.n_tile_live_src) d.tile_live[k] = t;
  }
}

template <int DIM>
__global__ void __launch_bounds__(kCoopBlock, 4) k_contact_rebuild(const __grid_constant__ DevData d, uint8_t search_bit,
                                                                  int64_t *bsum) {
  pdl_wait();
  if (d.ctrl->error) return;
  if (!d.ctrl->update) {
    list_live_tiles(d);
    return;
  }
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // phase clock (profiling): the first CTA's time past each barrier
  int mark = 0;
  auto stamp = [&]() {
    if (d.phase_ns && tid == 0 && mark < kRebuildPhases) d.phase_ns[mark] = global_ns();
    mark++;
  };
  stamp();
  stamp();  // nothing to clear
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  const int64_t N = d.n_nodes;
  const Grid G = d.grid;
  // nodes per cell (the counters are zero between rebuilds; where a rebuild that
  // stopped at a barrier is followed by others, the host clears them)
  if (d.sur_near_gate)
    for (int64_t p = tid; p < d.n_particles; p += nth) d.sur_near[p] = 0;
  for (int64_t i = tid; i < N; i += nth) {
    double p[3];
    ldv<DIM>(d.x, i, p);
    const int c = cell_index<DIM>(p, G);
    d.cell_of[i] = c;
    atomicAdd(d.cell_cnt + c, 1);
  }
  if (!grid_bar(d)) return;
  stamp();
  const int32_t *cc = d.cell_cnt;
  if (!grid_scan<int32_t>(d, [cc](int64_t k) { return cc[k]; }, d.cell_start, G.ncells, bsum)) return;
  stamp();
  for (int64_t i = tid; i < N; i += nth) {
    const int c = d.cell_of[i];
    d.cell_tmp[d.cell_start[c] + atomicAdd(d.cell_fill + c, 1)] = (int32_t)i;
  }
  if (!grid_bar(d)) return;
  stamp();
  {
    // per cell: its nodes in index order (rank counting), their particles and
    // positions in that order and, when they all belong to one particle, that
    // particle; the counters back to zero
    const int lane = threadIdx.x & 31;
    for (int64_t c = tid >> 5; c < G.ncells; c += nth >> 5) {
      const int s = d.cell_start[c], e = d.cell_start[c + 1];
      int32_t pmin = INT32_MAX, pmax = -1;
      for (int a = s + lane; a < e; a += 32) {
        const int32_t va = d.cell_tmp[a];
        const int32_t p = d.ptid[va];
        double xa[3];
        ldv<DIM>(d.x, va, xa);
        int rank = 0;
        for (int b = s; b < e; b++) rank += d.cell_tmp[b] < va;
        d.cell_nodes[s + rank] = va;
        d.cell_p[s + rank] = p;
        stv<DIM>(d.cell_x, s + rank, xa);
        pmin = min(pmin, p);
        pmax = max(pmax, p);
      }
      for (int o = 16; o > 0; o >>= 1) {
        pmin = min(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
        pmax = max(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
      }
      if (lane == 0) {
        d.cell_pid[c] = (e > s && pmin == pmax) ? pmin : -1;
        d.cell_cnt[c] = 0;
        d.cell_fill[c] = 0;
      }
    }
  }
  if (!grid_bar(d)) return;
  stamp();
  cand_count<DIM, DIM == 2 ? kCandLanes2 : kCandLanes3>(d, search_bit);
  if (!grid_bar(d)) return;
  stamp();
  // row offsets and the compacted list of nodes with candidates
  int64_t tot[2];
  const bool ok = scan_rows(d, d.c_cnt, N, bsum, tot, [&](int64_t i, int64_t cnt, int64_t row, int64_t at) {
    d.c_row[i] = row;
    if (cnt > 0) {
      d.c_nodes[at] = (int32_t)i;
      d.c_span[at] = make_int2((int)row, (int)(row + cnt));
      if (d.sur_near_gate) d.sur_near[d.ptid[i]] = 1;  // every writer stores the same value
    }
  });
  if (!ok) return;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    d.c_row[N] = tot[0];
    d.ctrl->c_nnodes = tot[1];
  }
  if (!grid_bar(d)) return;
  list_live_tiles(d);  // the proximity flags are final
  for (int k = 0; k < 3; k++) stamp();  // row offsets, compaction offsets, lists: one pass
  cand_fill_nodes<DIM>(d, d.ctrl->c_nnodes);
  stamp();  // the first CTA's share of the fill done
  if (tid == 0) {
    const int64_t total = d.c_row[N];
    d.ctrl->entries = total;
    d.ctrl->updates += 1;
    if (total > d.contact_cap) set_error(d.ctrl, DEV_ERR_CONTACT_OVERFLOW, total);
  }
}

// ---------------------------------------------------------------------------
// Distance pass ahead of the contact node pass: one thread per candidate
// entry marks the entries inside the largest contact radius of the zone-pair
// table (R < rc_max; every pair the node pass can accept, is_less(R, rc),
// has R < rc <= rc_max, and R is computed by the same operations there).
// Flat over the entries, so each thread carries one gather chain instead of
// a node's whole candidate row.
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_contact_near(DevData d) {
  if (d.ctrl->error) return;
  const int64_t E = d.ctrl->entries < d.contact_cap ? d.ctrl->entries : d.contact_cap;
  const double rmax = d.rc_max;
  for (int64_t e = (int64_t)blockIdx.x * kBlock + threadIdx.x; e < E; e += (int64_t)gridDim.x * kBlock) {
    const int32_t i = d.c_own[e], j = d.c_col[e];
    double yi[3], yj[3], yji[3];
    ldv<DIM>(d.x, i, yi);
    ldv<DIM>(d.x, j, yj);
#pragma unroll
    for (int q = 0; q < 3; q++) yji[q] = yj[q] - yi[q];
    d.c_hit[e] = len3<DIM>(yji) < rmax ? 1 : 0;
  }
}

// the node of every candidate entry, from the compacted lists (after a
// state snapshot restores them)
__global__ void k_contact_owner(DevData d) {
  const int64_t nn = d.ctrl->c_nnodes;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nn; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = d.c_nodes[t];
    const int2 sp = d.c_span[t];
    for (int64_t e = sp.x; e < sp.y && e < d.contact_cap; e++) d.c_own[e] = i;
  }
}

// ---------------------------------------------------------------------------
// Node pass of DEMModel::computeContactForces (demModel.cpp:832-934):
// penalty normal force + Coulomb-type friction for candidates inside the
// zone-pair contact radius; f_i += sum.  Particle-wall pairs inside the
// contact radius are recorded for the particle-wall damping (:994-1017),
// and the test wall's contact reaction is summed per block.
// ---------------------------------------------------------------------------
constexpr int kZonePairsSmem = 256;

// Every load a candidate needs is issued together: the compacted node and
// its candidate span (speculatively, before the node count arrives), then the
// node's own data with its candidate columns, then all of each candidate's
// data at once; the zone-pair table sits in shared memory.
template <int DIM, int LPN>
__global__ void __launch_bounds__(kBlock) k_contact(DevData d) {
  __shared__ ContactPair cps[kZonePairsSmem];
  __shared__ double scr[kBlock / LPN];
  const int lane = threadIdx.x % LPN;
  const int nz = d.n_zones;
  const bool tab = nz * nz <= kZonePairsSmem;
  const int64_t gstride = (int64_t)gridDim.x * (kBlock / LPN);
  int64_t t = (int64_t)blockIdx.x * (kBlock / LPN) + threadIdx.x / LPN;
  int32_t i_next = t < d.n_nodes ? d.c_nodes[t] : 0;
  int2 sp_next = t < d.n_nodes ? d.c_span[t] : make_int2(0, 0);
  const int64_t nn_raw = d.ctrl->c_nnodes;
  const int err = d.ctrl->error;
  if (tab)
    for (int a = threadIdx.x; a < nz * nz; a += kBlock) cps[a] = d.contact[a];
  __syncthreads();
  const int64_t nn = err ? 0 : nn_raw;
  double crd_acc = 0.0;
  for (; t < nn; t += gstride) {
    const int64_t i = i_next;
    const int2 sp = sp_next;
    if (t + gstride < nn) {
      i_next = d.c_nodes[t + gstride];
      sp_next = d.c_span[t + gstride];
    }
    const unsigned gm = group_mask<LPN>();
    const int32_t pi = d.ptid[i];
    const int zi = d.nzone[i];
    double yi[3], vi[3];
    ldv<DIM>(d.x, i, yi);
    ldv<DIM>(d.v, i, vi);
    double fx = 0.0, fy = 0.0, fz = 0.0, crd = 0.0;
    for (int k = sp.x + lane; k < sp.y; k += LPN) {
      // most candidates lie in the search skin, beyond every zone pair's
      // contact radius: k_contact_near marked the others
      if (!d.c_hit[k]) continue;
      const int32_t j = d.c_col[k];
      double yj[3];
      ldv<DIM>(d.x, j, yj);
      double yji[3];
#pragma unroll
      for (int q = 0; q < 3; q++) yji[q] = yj[q] - yi[q];
      const double R = len3<DIM>(yji);
      double vj[3];
      ldv<DIM>(d.v, j, vj);
      const double volj = d.vol[j];
      const int32_t pj = d.ptid[j];
      const int zj = d.nzone[j];
      const bool wall = (d.flags[j] & NODE_WALL) != 0;
      const ContactPair cp = tab ? cps[zi * nz + zj] : d.contact[zi * nz + zj];
      if (is_less(R, cp.rc)) {
        double vji[3], en[3], et[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
          vji[q] = vj[q] - vi[q];
          en[q] = yji[q] / R;
        }
        const double vn = dot3<DIM>(vji, en);
#pragma unroll
        for (int q = 0; q < 3; q++) et[q] = vji[q] - vn * en[q];
        const double etl = len3<DIM>(et);
        if (is_greater(etl, 0.)) {
#pragma unroll
          for (int q = 0; q < 3; q++) et[q] = et[q] / etl;
        } else {
          et[0] = et[1] = et[2] = 0.0;
        }
        double sf = cp.kn * (R - cp.rc) * volj;
        if (sf > 0.) sf = 0.;
        const double mf = cp.mu * sf;
        const double cx = sf * en[0], cy = sf * en[1], cz = sf * en[2];
        fx += cx;
        fy += cy;
        if constexpr (DIM == 3) fz += cz;
        fx += mf * et[0];
        fy += mf * et[1];
        if constexpr (DIM == 3) fz += mf * et[2];
        if (wall) {
          const int slot = atomicAdd(d.wp_cnt + pi, 1);
          if (slot < d.wp_cap) d.wp[(int64_t)pi * d.wp_cap + slot] = j;
          else set_error(d.ctrl, DEV_ERR_WALLPAIR_OVERFLOW, pi);
        }
        if (d.pwall_test ? d.pwall_test[pj] != 0 : pj == d.test_wall) {
          const int td = d.test_dir;
          crd += td == 0 ? cx + mf * et[0] : (td == 1 ? cy + mf * et[1] : cz + mf * et[2]);
        }
      }
    }
    fx = group_sum<LPN>(fx, gm);
    fy = group_sum<LPN>(fy, gm);
    if constexpr (DIM == 3) fz = group_sum<LPN>(fz, gm);
    crd = group_sum<LPN>(crd, gm);
    if (lane == 0) {
      const double f[3] = {fx, fy, fz};
      stv<DIM>(d.fc, i, f);
      crd_acc += crd * d.vol[i];
      if (d.cr_t) d.cr_t[t] = crd * d.vol[i];
    }
  }
  // deterministic per-block partial of the test wall's contact reaction
  if (lane == 0) scr[threadIdx.x / LPN] = crd_acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int g = 0; g < kBlock / LPN; g++) sum += scr[g];
    d.cr_partial[blockIdx.x] = sum;
  }
}

// ---------------------------------------------------------------------------
// Particle damping of DEMModel::computeContactForces (demModel.cpp:937-1050):
// particle-particle through particle centres and particle-wall through the
// condensed wall nodes; the force density is applied to all nodes of the
// particle by the external-force pass.
//
// Particle-particle: one warp per particle, kBlock / 32 of them per CTA.  The
// CTA stages the centres of kBlock particles at a time in FP32 and every warp
// tests its particle against them with an 8 % margin over the largest reach
// any zone pair allows (coordinates rounded to FP32 move a distance by far
// less), so that only pairs the FP64 test can pass read FP64 data.
//
// It reads positions only, so its CTAs ride in the contact pass's launch: a
// launch of its own behind the contact pass finds the SMs full of bond-loop
// CTAs (one CTA of 128 threads and 39 KB per particle or group of four, 504 /
// 2 002 particles: 20 / 84 us beside the bond loop; a warp per particle there,
// 14 to 21 / 73 to 85).  In the contact launch the pass ends 3.6 / 12 us later
// than without them, and the wall part behind it takes 2 to 3 us.
// ---------------------------------------------------------------------------
template <int DIM>
__device__ __forceinline__ void damp_pairs(const DevData &d, int block, ContactPair *cps) {
  __shared__ float4 s_c[kBlock];  // {x, y, z, bounding radius}
  __shared__ int s_range[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = block * (kBlock / 32) + warp;
  const int nz = d.n_zones;
  const bool tab = nz * nz <= kZonePairsSmem;
  if (tab)
    for (int a = threadIdx.x; a < nz * nz; a += kBlock) cps[a] = d.contact[a];
  if (threadIdx.x < 2) {
    // the scenes of the CTA's particles, which are consecutive
    const int last = min((block + 1) * (kBlock / 32), d.n_particles) - 1;
    s_range[threadIdx.x] = threadIdx.x == 0 ? d.dpart[block * (kBlock / 32)].q0 : d.dpart[last].q1;
  }
  DampParticle P{};
  P.type = 1;
  double xi[3] = {0, 0, 0}, vi[3] = {0, 0, 0};
  if (p < d.n_particles) {
    P = d.dpart[p];
    ldv<DIM>(d.x, P.center, xi);
    ldv<DIM>(d.v, P.center, vi);
  }
  const float fxi = (float)xi[0], fyi = (float)xi[1], fzi = (float)xi[2];
  const double Ri = P.bound_r, vol_pi = kPi * Ri * Ri;
  const float fr = (float)Ri, rc_f = (float)(1.01 * d.rc_max);
  double acc[3] = {0.0, 0.0, 0.0};
  if (__syncthreads_or(d.ctrl->error != 0)) return;
  const int q_lo = s_range[0], q_hi = s_range[1];
  for (int tb = q_lo; tb < q_hi; tb += kBlock) {
    __syncthreads();  // the previous centres are no longer read
    if (tb + (int)threadIdx.x < q_hi) {
      const int q = tb + threadIdx.x;
      double xq[3];
      ldv<DIM>(d.x, d.dpart[q].center, xq);
      s_c[threadIdx.x] = make_float4((float)xq[0], (float)xq[1], (float)xq[2], (float)d.dpart[q].bound_r);
    }
    __syncthreads();
    if (P.type != 0) continue;
#pragma unroll 4
    for (int k = 0; k < kBlock / 32; k++) {
      const int q = tb + lane + 32 * k;
      if (q >= P.q1 || q < P.q0 || q == p) continue;
      const float4 cf = s_c[lane + 32 * k];
      const float ex = cf.x - fxi, ey = cf.y - fyi, ez = cf.z - fzi;
      const float rm = cf.w + fr + rc_f;
      if (ex * ex + ey * ey + ez * ez > 1.17f * rm * rm) continue;
      const DampParticle Q = d.dpart[q];
      if (Q.type != 0) continue;
      double xcj[3], vcj[3];
      ldv<DIM>(d.x, Q.center, xcj);
      ldv<DIM>(d.v, Q.center, vcj);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        xcj[c] -= xi[c];
        vcj[c] -= vi[c];
      }
      const double Rj = Q.bound_r;
      const double d2 = dot3<DIM>(xcj, xcj);
      const ContactPair cp = tab ? cps[P.zone * nz + Q.zone] : d.contact[P.zone * nz + Q.zone];
      const double reach = Rj + Ri + 1.01 * cp.rc;
      // pairs well beyond the reach cannot pass the relative-tolerance test
      if (d2 > 1.0625 * reach * reach) continue;
      const double dist = sqrt(d2);
      if (is_less(dist, reach)) {
        const double vol_pj = kPi * Rj * Rj;
        const double m1 = P.density * vol_pi, m2 = Q.density * vol_pj;
        const double meq = 2. * m1 * m2 / (m1 + m2);  // util::equivalentMass
        const double bn = cp.betan * sqrt(cp.kappa * cp.rc * meq);
        double hat[3] = {0.0, 0.0, 0.0};
        if (is_greater(dist, 0.))
          for (int c = 0; c < 3; c++) hat[c] = xcj[c] / dist;
        double vm = vcj[0] * hat[0] + vcj[1] * hat[1] + vcj[2] * hat[2];
        if (vm > 0.) vm = 0.;
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c] += bn * vm * hat[c] / vol_pi;
      }
    }
  }
  if (P.type != 0) return;  // uniform over the warp
#pragma unroll
  for (int t = 0; t < 3; t++) {
    for (int o = 16; o > 0; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
    if (lane == 0) d.fdamp[4 * p + t] = acc[t];
  }
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_damp_pairs(const __grid_constant__ DevData d) {
  __shared__ ContactPair cps[kZonePairsSmem];
  damp_pairs<DIM>(d, (int)blockIdx.x, cps);
}

// ---------------------------------------------------------------------------
// The contact node pass in one kernel, warp-cooperative (the default, one
// lane per node): a warp takes up to 32 consecutive compacted nodes, whose
// candidate rows are consecutive in the entry array, and walks their entries
// coalesced, kContactBatch x 32 at a time: first the distance of every entry
// (its node's and its candidate's positions, all loads of a batch in flight),
// then, only for groups of 32 with a pair inside the largest contact radius,
// the forces.  There each lane finds its entry's node among the warp's (binary
// search over the row starts, held one per lane) and takes that node's data by
// shuffle.  The contributions are then handed, in entry order, to the lane
// that owns the node, which adds them in the reference's order (normal part,
// then friction part, candidate by candidate).  Results equal the node pass
// with one lane per node.
//
// Bound by the latency of its dependent loads (entry, position), so it wants
// many entries in flight: a warp takes 8 or 16 nodes instead of 32 while the
// launch has warps left over.  Against 32 nodes per warp and one group of
// entries at a time, beside the bond loop: 332 000 nodes 12.3 -> 5.5 us, 1.3 M
// nodes 27 -> 14, a 24 000-node packing 9.9 -> 3.8.  Limits of 80 or 64
// registers, for more CTAs beside the bond loop, gain nothing (spills).
// The CTAs past the contact grid run the particle-particle damping beside it.
// ---------------------------------------------------------------------------
constexpr int kContactBatch = 4;

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_contact_warp(const __grid_constant__ DevData d) {
  __shared__ ContactPair cps[kZonePairsSmem];
  __shared__ double scr[kBlock];
  pdl_start();
  const int l32 = threadIdx.x & 31;
  const int nz = d.n_zones;
  const bool tab = nz * nz <= kZonePairsSmem;
  if ((int)blockIdx.x >= d.contact_grid) {
    damp_pairs<DIM>(d, (int)blockIdx.x - d.contact_grid, cps);
    return;
  }
  const int64_t nn_raw = d.ctrl->c_nnodes;
  const int err = d.ctrl->error;
  if (tab)
    for (int a = threadIdx.x; a < nz * nz; a += kBlock) cps[a] = d.contact[a];
  __syncthreads();
  const int64_t nn = err ? 0 : nn_raw;
  const double rmax = d.rc_max;
  const int64_t nwarps = (int64_t)d.contact_grid * (kBlock / 32);
  const int npw = nn <= 8 * nwarps ? 8 : (nn <= 16 * nwarps ? 16 : 32);  // nodes per warp
  double crd_acc = 0.0;
  // warp w of block b takes group w * grid + b: few groups spread over the SMs
  for (int64_t w = (int64_t)(threadIdx.x >> 5) * d.contact_grid + blockIdx.x; w * npw < nn; w += nwarps) {
    const int64_t t = w * npw + l32;
    const int nval = (int)min((int64_t)npw, nn - w * npw);  // lanes with a node
    const bool own = l32 < nval;
    int32_t i = 0;
    int2 sp = make_int2(0, 0);
    double yi[3] = {0, 0, 0}, vi[3] = {0, 0, 0};
    int32_t pi = -1;
    int zi = 0;
    if (own) {
      i = d.c_nodes[t];
      sp = d.c_span[t];
    }
    const int e0 = __shfl_sync(0xffffffffu, sp.x, 0);
    const int e1 = __shfl_sync(0xffffffffu, sp.y, nval - 1);
    if (own) {
      pi = d.ptid[i];
      zi = d.nzone[i];
      ldv<DIM>(d.x, i, yi);
      ldv<DIM>(d.v, i, vi);
    }
    double fx = 0.0, fy = 0.0, fz = 0.0, crd = 0.0;
    for (int base0 = e0; base0 < e1; base0 += 32 * kContactBatch) {
      int32_t jb[kContactBatch], ib[kContactBatch];
#pragma unroll
      for (int b = 0; b < kContactBatch; b++) {
        const int e = base0 + 32 * b + l32;
        jb[b] = ib[b] = 0;
        if (e < e1) {
          jb[b] = d.c_col[e];
          ib[b] = d.c_own[e];
        }
      }
      double yb[kContactBatch][3];
      unsigned near = 0;  // bit b: this lane's entry of group b is inside rmax
#pragma unroll
      for (int b = 0; b < kContactBatch; b++) {
        double yo[3];
        ldv<DIM>(d.x, ib[b], yo);
        ldv<DIM>(d.x, jb[b], yb[b]);
#pragma unroll
        for (int q = 0; q < 3; q++) yb[b][q] = yb[b][q] - yo[q];
      }
#pragma unroll
      for (int b = 0; b < kContactBatch; b++)
        if (base0 + 32 * b + l32 < e1 && len3<DIM>(yb[b]) < rmax) near |= 1u << b;
#pragma unroll
      for (int b = 0; b < kContactBatch; b++) {
        const bool hit = (near >> b) & 1u;
        if (!__any_sync(0xffffffffu, hit)) continue;
        const int e = base0 + 32 * b + l32;
        // the entry's node: the last lane whose row starts at or before e
        int o = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const int cnd = o + step;
          const int st = __shfl_sync(0xffffffffu, sp.x, cnd & 31);
          if (cnd < nval && st <= e) o = cnd;
        }
        double vo[3];
#pragma unroll
        for (int q = 0; q < 3; q++) vo[q] = __shfl_sync(0xffffffffu, vi[q], o);
        const int32_t po = __shfl_sync(0xffffffffu, pi, o);
        const int zo = __shfl_sync(0xffffffffu, zi, o);
        double cxn = 0.0, cyn = 0.0, czn = 0.0, cxt = 0.0, cyt = 0.0, czt = 0.0, cr = 0.0;
        bool contrib = false;
        if (hit) {
          const int32_t j = jb[b];
          const double(&yji)[3] = yb[b];
          const double R = len3<DIM>(yji);
          double vj[3];
          ldv<DIM>(d.v, j, vj);
          const double volj = d.vol[j];
          const int32_t pj = d.ptid[j];
          const int zj = d.nzone[j];
          const bool wall = (d.flags[j] & NODE_WALL) != 0;
          const ContactPair cp = tab ? cps[zo * nz + zj] : d.contact[zo * nz + zj];
          if (is_less(R, cp.rc)) {
            double vji[3], en[3], et[3];
#pragma unroll
            for (int q = 0; q < 3; q++) {
              vji[q] = vj[q] - vo[q];
              en[q] = yji[q] / R;
            }
            const double vn = dot3<DIM>(vji, en);
#pragma unroll
            for (int q = 0; q < 3; q++) et[q] = vji[q] - vn * en[q];
            const double etl = len3<DIM>(et);
            if (is_greater(etl, 0.)) {
#pragma unroll
              for (int q = 0; q < 3; q++) et[q] = et[q] / etl;
            } else {
              et[0] = et[1] = et[2] = 0.0;
            }
            double sf = cp.kn * (R - cp.rc) * volj;
            if (sf > 0.) sf = 0.;
            const double mf = cp.mu * sf;
            cxn = sf * en[0];
            cyn = sf * en[1];
            czn = sf * en[2];
            cxt = mf * et[0];
            cyt = mf * et[1];
            czt = mf * et[2];
            contrib = true;
            if (wall) {
              const int slot = atomicAdd(d.wp_cnt + po, 1);
              if (slot < d.wp_cap) d.wp[(int64_t)po * d.wp_cap + slot] = j;
              else set_error(d.ctrl, DEV_ERR_WALLPAIR_OVERFLOW, po);
            }
            if (d.pwall_test ? d.pwall_test[pj] != 0 : pj == d.test_wall) {
              const int td = d.test_dir;
              cr = td == 0 ? cxn + cxt : (td == 1 ? cyn + cyt : czn + czt);
            } else {
              cr = -0.0;  // marks "no test-wall term" (never added)
            }
          }
        }
        // hand the contributions to their nodes' lanes in entry order
        unsigned m = __ballot_sync(0xffffffffu, contrib);
        while (m) {
          const int src = __ffs(m) - 1;
          m &= m - 1;
          const int dst = __shfl_sync(0xffffffffu, o, src);
          const double ax = __shfl_sync(0xffffffffu, cxn, src), ay = __shfl_sync(0xffffffffu, cyn, src);
          const double bx = __shfl_sync(0xffffffffu, cxt, src), by = __shfl_sync(0xffffffffu, cyt, src);
          const double c = __shfl_sync(0xffffffffu, cr, src);
          double az = 0.0, bz = 0.0;
          if constexpr (DIM == 3) {
            az = __shfl_sync(0xffffffffu, czn, src);
            bz = __shfl_sync(0xffffffffu, czt, src);
          }
          if (l32 == dst) {
            fx += ax;
            fy += ay;
            if constexpr (DIM == 3) fz += az;
            fx += bx;
            fy += by;
            if constexpr (DIM == 3) fz += bz;
            if (!(c == 0.0 && signbit(c))) crd += c;
          }
        }
      }
    }
    if (own) {
      if (fx != 0.0 || fy != 0.0 || (DIM == 3 && fz != 0.0)) {
        const double f[3] = {fx, fy, fz};
        stv<DIM>(d.fc, i, f);
      }
      if (crd != 0.0) crd_acc += crd * d.vol[i];
      if (d.cr_t) d.cr_t[t] = crd * d.vol[i];
    }
  }
  // deterministic per-block partial of the test wall's contact reaction
  if (!__syncthreads_or(crd_acc != 0.0)) {
    if (threadIdx.x == 0) d.cr_partial[blockIdx.x] = 0.0;
    return;
  }
  scr[threadIdx.x] = crd_acc;
  __syncthreads();
  for (int h = kBlock / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) scr[threadIdx.x] += scr[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) d.cr_partial[blockIdx.x] = scr[0];
}

// ---------------------------------------------------------------------------
// Particle-wall damping, after the contact pass has recorded the wall nodes:
// one warp per particle, a particle that touches no wall leaves at once.
// Added to the particle-particle part in fdamp.
// ---------------------------------------------------------------------------
constexpr int kDampBlock = 128;
constexpr int kWallSort = 4096;  // wall pairs of one particle, at most
constexpr int kWallWarp = 128;   // up to here the particle's own warp orders them

// particle p's sorted wall nodes wn[0 .. nw), each distinct node once
template <int DIM>
__device__ __forceinline__ void damp_wall_sum(const DevData &d, int p, const int32_t *wn, int nw) {
  const int lane = threadIdx.x & 31, nz = d.n_zones;
  const DampParticle P = d.dpart[p];
  const double vol_pi = kPi * P.bound_r * P.bound_r;
  double xc[3], vc[3], acc[3] = {0.0, 0.0, 0.0};
  ldv<DIM>(d.x, P.center, xc);
  ldv<DIM>(d.v, P.center, vc);
  for (int a = lane; a < nw; a += 32) {
    const int32_t w = wn[a];
    if (a > 0 && wn[a - 1] == w) continue;
    const ContactPair cp = d.contact[P.zone * nz + d.nzone[w]];
    const double meq = P.density * vol_pi;
    const double bn = cp.betan * sqrt(cp.kappa * cp.rc * meq);
    double xk[3], vk[3];
    ldv<DIM>(d.x, w, xk);
    ldv<DIM>(d.v, w, vk);
#pragma unroll
    for (int t = 0; t < 3; t++) {
      xk[t] -= xc[t];
      vk[t] -= vc[t];
    }
    const double l = len3<DIM>(xk);
    double hat[3] = {0.0, 0.0, 0.0};
    if (is_greater(l, 0.))
      for (int t = 0; t < 3; t++) hat[t] = xk[t] / l;
    double vm = vk[0] * hat[0] + vk[1] * hat[1] + vk[2] * hat[2];
    if (vm > 0.) vm = 0.;
#pragma unroll
    for (int t = 0; t < 3; t++) acc[t] += bn * vm * hat[t] / vol_pi;
  }
#pragma unroll
  for (int t = 0; t < 3; t++) {
    for (int o = 16; o > 0; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
    if (lane == 0) d.fdamp[4 * p + t] += acc[t];
  }
  if (lane == 0) d.wp_cnt[p] = 0;
}

template <int DIM>
__global__ void __launch_bounds__(kDampBlock) k_damp_walls(const __grid_constant__ DevData d) {
  __shared__ int32_t wn[kWallSort];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * (kDampBlock / 32) + warp;
  const int cap = min(d.wp_cap, kWallSort);  // the capacity is validated on the host
  pdl_wait();
  const int nw = p < d.n_particles && !d.ctrl->error ? min(d.wp_cnt[p], cap) : 0;
  if (nw > 0 && nw <= kWallWarp) {  // ordered by counting
    int32_t *mine = wn + warp * (2 * kWallWarp);
    for (int a = lane; a < nw; a += 32) mine[a] = d.wp[(int64_t)p * d.wp_cap + a];
    __syncwarp();
    for (int a = lane; a < nw; a += 32) {
      const int32_t va = mine[a];
      int rank = 0;
      for (int b = 0; b < nw; b++) rank += mine[b] < va || (mine[b] == va && b < a);
      mine[kWallWarp + rank] = va;
    }
    __syncwarp();
    damp_wall_sum<DIM>(d, p, mine + kWallWarp, nw);
  }
  if (!__syncthreads_or(nw > kWallWarp)) return;
  // more: the whole CTA sorts them, one particle after another
  __shared__ int s_nw[kDampBlock / 32];
  if (lane == 0) s_nw[warp] = nw;
  __syncthreads();
  for (int k = 0; k < kDampBlock / 32; k++) {
    const int n = s_nw[k];
    if (n <= kWallWarp) continue;  // uniform over the CTA
    const int pk = blockIdx.x * (kDampBlock / 32) + k;
    int sz = 1;
    while (sz < n) sz <<= 1;
    for (int a = threadIdx.x; a < sz; a += kDampBlock)
      wn[a] = a < n ? d.wp[(int64_t)pk * d.wp_cap + a] : INT32_MAX;
    __syncthreads();
    for (int kk = 2; kk <= sz; kk <<= 1)
      for (int jj = kk >> 1; jj > 0; jj >>= 1) {
        for (int a = threadIdx.x; a < sz; a += kDampBlock) {
          const int b = a ^ jj;
          if (b > a) {
            const bool up = (a & kk) == 0;
            const int32_t va = wn[a], vb = wn[b];
            if ((va > vb) == up) {
              wn[a] = vb;
              wn[b] = va;
            }
          }
        }
        __syncthreads();
      }
    if (warp == k) damp_wall_sum<DIM>(d, pk, wn, n);
    __syncthreads();  // the array is free
  }
}

// ---------------------------------------------------------------------------
// Damping force to all nodes of each particle (demModel.cpp:1053-1064), then
// DEMModel::computeExternalForces (:791-812): gravity, then force BCs
// (ParticleFLoading::apply, particleFLoading.cpp:85-173).
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void k_external(DevData d) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes || d.ctrl->error) return;
  // nodes outside d_fPdCompNodes carry no peridynamic or contact force: the
  // reference zeroes f for all nodes at the start of computeForces (:473-478)
  double f[3] = {0.0, 0.0, 0.0};
  const uint8_t fl = d.flags[i];
  if (fl & NODE_ACTIVE) {
    ldv<DIM>(d.f, i, f);
    // contact forces (computeContactForces adds them after the bond loop);
    // only searching nodes can carry one
    if (d.fc && (fl & (NODE_SEARCH | NODE_SEARCH0))) {
      double c[3];
      ldv<DIM>(d.fc, i, c);
      if (c[0] != 0.0 || c[1] != 0.0 || (DIM == 3 && c[2] != 0.0)) {
#pragma unroll
        for (int q = 0; q < DIM; q++) f[q] += c[q];
        const double z[3] = {0.0, 0.0, 0.0};
        stv<DIM>(d.fc, i, z);
      }
    }
  }
  const int32_t p = d.ptid[i];
  if (d.flags[i] & NODE_PARTICLE) {
#pragma unroll
    for (int q = 0; q < DIM; q++) f[q] += d.fdamp[4 * p + q];
  }
  if (d.gravity_on) {
    const double rho = d.particles[p].density;
#pragma unroll
    for (int q = 0; q < DIM; q++) f[q] += rho * d.gravity[q];
  }
  stv<DIM>(d.f, i, f);
}

template <int DIM>
__device__ __noinline__ void apply_fbc(const DevData &d, int t, double time, double (&f)[3]) {
  for (int e = d.fbc_row[t]; e < d.fbc_row[t + 1]; e++) {
    const BcSetDev bc = d.fbc_sets[d.fbc_set[e]];
    double fmax = d.fbc_val[e];
    switch (bc.time_fn) {
      case PDGPU_TIME_LINEAR: fmax *= time; break;
      case PDGPU_TIME_LINEAR_STEP: {
        // util::linearStepFunc (function.cpp:62-85)
        const double x1 = bc.tp[1], x2 = bc.tp[2];
        const double period = floor(time / (x1 + x2));
        const double val =
            is_less(time, period * (x1 + x2) + x1) ? time - period * x2 : (period + 1.) * x1;
        fmax *= val;
        break;
      }
      case PDGPU_TIME_LINEAR_SLOW_FAST:
        if (is_greater(time, bc.tp[1])) fmax *= bc.tp[3] * time;
        else fmax *= bc.tp[2] * time;
        break;
      case PDGPU_TIME_SIN: fmax *= sin(kPi * bc.tp[1] * time); break;
      default: break;
    }
    fmax *= bc.tp[0];
    for (int q = 0; q < DIM; q++)
      if ((bc.dir_mask >> q) & 1) f[q] += fmax;
  }
}

template <int DIM>
__global__ void k_force_bc(const __grid_constant__ DevData d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.n_fbc_nodes || d.ctrl->error) return;
  const int64_t i = d.fbc_node[t];
  double f[3];
  ldv<DIM>(d.f, i, f);
  apply_fbc<DIM>(d, t, d.ctrl->time, f);
  stv<DIM>(d.f, i, f);
}

// ---------------------------------------------------------------------------
// Post-processing every test_interval steps: DEMModel::ppCompressiveTest
// (demModel.cpp:2202-2250) or ppTwoParticleTest (:2096-2149).
// ---------------------------------------------------------------------------
// doubles as unsigned keys of the same order (0 below every key)
__device__ __forceinline__ unsigned long long to_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b >> 63 ? ~b : b | (1ull << 63);
}
__device__ __forceinline__ double from_key(unsigned long long k) {
  if (k == 0) return -DBL_MAX;  // no value
  return __longlong_as_double((long long)(k >> 63 ? k & ~(1ull << 63) : ~k));
}

// The test's post-processing (demModel.cpp ppCompressiveTest / ppTwoParticleTest)
// run by one 1024-thread block; forces of the current step are read past L1,
// since other CTAs of the same kernel may have written them.
// pre: the positions it needs, where the caller has moved the nodes on already
// (TurnState; null: they are in d.x)
template <int DIM>
__device__ __noinline__ void postprocess_block(const DevData &d, const TurnState *pre = nullptr) {
  // sums are formed as by a 1024-thread block (per-thread strided partials,
  // warp butterflies, then the 32 warp sums in order), whatever blockDim is
  constexpr int kV = 1024;
  __shared__ double red[2][kV / 32];
  CtrlState *c = d.ctrl;
  if (c->error) return;
  const int64_t n = c->n;
  if (!(n % d.test_interval == 0 && n >= d.test_interval)) return;
  const int st = DIM == 2 ? 2 : 4;
  if (d.test == PDGPU_TEST_COMPRESSIVE) {
    const DevParticle W = d.particles[d.test_wall];
    const int dir = d.test_dir;
    for (int vt = threadIdx.x; vt < kV; vt += blockDim.x) {
      double s = 0.0;
      for (int64_t i = W.start + vt; i < W.end; i += kV) s += __ldcg(d.f + st * i + dir) * d.vol[i];
      double cr = 0.0;
      for (int b = vt; b < d.cr_blocks; b += kV) cr += d.cr_partial[b];
      for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        cr += __shfl_xor_sync(0xffffffffu, cr, o);
      }
      if ((vt & 31) == 0) {
        red[0][vt >> 5] = s;
        red[1][vt >> 5] = cr;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double rs = 0.0, rc = 0.0;
      for (int w = 0; w < kV / 32; w++) {
        rs += red[0][w];
        rc += red[1][w];
      }
      const double delta = (pre ? pre->wall[dir] : d.x[st * W.start + dir]) - d.xref[st * W.start + dir];
      c->reaction = rs;
      c->contact_reaction = -rc;
      c->penetration = delta;
      const int64_t h = c->history_count;
      if (h < d.history_cap) {
        d.history[4 * h] = c->time;
        d.history[4 * h + 1] = delta;
        d.history[4 * h + 2] = rs;
        d.history[4 * h + 3] = -rc;
      }
      c->history_count = h + 1;
    }
  } else if (d.test == PDGPU_TEST_TWO_PARTICLE && d.n_particles >= 2) {
    const DevParticle P0 = d.particles[0], P1 = d.particles[1];
    for (int vt = threadIdx.x; vt < kV && !pre; vt += blockDim.x) {
      double m = -DBL_MAX;
      for (int64_t i = P1.start + vt; i < P1.end; i += kV) m = fmax(m, d.x[st * i + 1]);
      for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((vt & 31) == 0) red[0][vt >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double my = pre ? from_key(pre->max_y) : -DBL_MAX;
      for (int w = 0; w < kV / 32 && !pre; w++) my = fmax(my, red[0][w]);
      double dx[3] = {0, 0, 0};
      for (int q = 0; q < DIM; q++)
        dx[q] = pre ? pre->centre[1][q] - pre->centre[0][q] : d.x[st * P1.center + q] - d.x[st * P0.center + q];
      const double r = P0.bound_r;
      const ContactPair cp = d.contact[P0.zone * d.n_zones + P1.zone];
      const double re = r + cp.rc;
      double pen = sqrt(dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2]) - re - r;
      double car = 0.0;
      if (is_less(pen, 0.)) car = sqrt(re * re - (re + pen) * (re + pen));
      else if (is_greater(pen, 0.)) {
        pen = 0.;
        car = 0.;
      }
      c->pen_dist = pen;
      c->contact_area_radius = car;
      c->max_y = is_less(0.0, my) ? my : 0.0;
    }
  }
}

// Compressive-test output of every scene of a batched ensemble, one CTA per
// scene (the single-scene form is postprocess_block): the test wall's
// reaction sum f vol over its nodes, the contact reaction summed over the
// scene's run of the compacted contact nodes (ascending node ids, so each
// scene's nodes form one run), and the wall's displacement.
template <int DIM>
__global__ void __launch_bounds__(256) k_scene_post(const __grid_constant__ DevData d) {
  __shared__ double red[2][8];
  __shared__ int64_t range[2];
  pdl_start();
  pdl_wait();
  const CtrlState *c = d.ctrl;
  if (c->error) return;
  const int64_t n = c->n;
  if (!(n % d.test_interval == 0 && n >= d.test_interval)) return;
  const int64_t h = n / d.test_interval - 1;
  const int s = blockIdx.x;
  if (h >= d.scene_hist_cap || s >= d.n_scenes || d.scene_wall[s] < 0) return;
  const int st = DIM == 2 ? 2 : 4;
  const DevParticle W = d.particles[d.scene_wall[s]];
  const int dir = d.test_dir;
  const int64_t nn = c->c_nnodes;
  if (threadIdx.x < 2) {
    const int64_t key = d.scene_node[s + threadIdx.x];
    int64_t lo = 0, hi = nn;  // first compacted index whose node is >= key
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (d.c_nodes[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    range[threadIdx.x] = lo;
  }
  __syncthreads();
  double rs = 0.0, rc = 0.0;
  for (int64_t i = W.start + threadIdx.x; i < W.end; i += blockDim.x) rs += d.f[st * i + dir] * d.vol[i];
  for (int64_t t = range[0] + threadIdx.x; t < range[1]; t += blockDim.x) rc += d.cr_t[t];
  for (int o = 16; o > 0; o >>= 1) {
    rs += __shfl_xor_sync(0xffffffffu, rs, o);
    rc += __shfl_xor_sync(0xffffffffu, rc, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = rs;
    red[1][threadIdx.x >> 5] = rc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < 8; w++) {
      a += red[0][w];
      b += red[1][w];
    }
    double *o = d.scene_hist + 4 * ((int64_t)s * d.scene_hist_cap + h);
    o[0] = c->time;
    o[1] = d.x[st * W.start + dir] - d.xref[st * W.start + dir];
    o[2] = a;
    o[3] = -b;
  }
}

template <int DIM>
__global__ void __launch_bounds__(1024) k_postprocess(const __grid_constant__ DevData d) {
  postprocess_block<DIM>(d);
}

// ---------------------------------------------------------------------------
// Last kernel of a step: per node, the external-force pass
// (as k_external: bond forces, then contact forces, damping, gravity), the
// force BC (as k_force_bc) and, for velocity Verlet, the second half kick (as
// k_verlet_second); then the last CTA to finish runs the post-processing (as
// k_postprocess) when `post` is set.
// ---------------------------------------------------------------------------
constexpr int kEndNodes = 2;  // nodes per thread of the step-end kernel

template <int DIM, bool VERLET>
__global__ void __launch_bounds__(kBlock) k_step_end(const __grid_constant__ DevData d, int post) {
  __shared__ int last;
  pdl_start();
  const int64_t n_step = d.ctrl->n;
  // each thread takes kEndNodes nodes, kBlock apart, and issues the node
  // loads of all of them (independent of their flags) before the sums
  const int64_t base = (int64_t)blockIdx.x * (kBlock * kEndNodes) + threadIdx.x;
  if (!d.ctrl->error) {
    uint8_t fl[kEndNodes];
    int32_t pid[kEndNodes];
    double fa[kEndNodes][3];
#pragma unroll
    for (int k = 0; k < kEndNodes; k++) {
      const int64_t i = base + (int64_t)k * kBlock;
      fl[k] = 0;
      pid[k] = 0;
      if (i < d.n_nodes) {
        fl[k] = d.flags[i];
        pid[k] = d.ptid[i];
        ldv<DIM>(d.f, i, fa[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < kEndNodes; k++) {
      const int64_t i = base + (int64_t)k * kBlock;
      if (i >= d.n_nodes) continue;
      const int32_t p = pid[k];
      double f[3] = {0.0, 0.0, 0.0};
      // the contact force only where the node searches (elsewhere it is never
      // written and its lines are cold)
      if (fl[k] & NODE_ACTIVE) {
#pragma unroll
        for (int q = 0; q < DIM; q++) f[q] = fa[k][q];
        if (d.fc && (fl[k] & (NODE_SEARCH | NODE_SEARCH0))) {
          double c[3];
          ldv<DIM>(d.fc, i, c);
          if (c[0] != 0.0 || c[1] != 0.0 || (DIM == 3 && c[2] != 0.0)) {
#pragma unroll
            for (int q = 0; q < DIM; q++) f[q] += c[q];
            const double z[3] = {0.0, 0.0, 0.0};
            stv<DIM>(d.fc, i, z);
          }
        }
      }
      if (fl[k] & NODE_PARTICLE) {
#pragma unroll
        for (int q = 0; q < DIM; q++) f[q] += d.fdamp[4 * p + q];
      }
      double rho = 0.0;
      if (d.gravity_on || (VERLET && (fl[k] & NODE_ACTIVE))) rho = d.particles[p].density;
      if (d.gravity_on) {
#pragma unroll
        for (int q = 0; q < DIM; q++) f[q] += rho * d.gravity[q];
      }
      if (fl[k] & NODE_FBC) {  // through a copy, so that f stays in registers
        double fb[3] = {f[0], f[1], f[2]};
        apply_fbc<DIM>(d, d.fbc_of[i], d.ctrl->time, fb);
#pragma unroll
        for (int q = 0; q < 3; q++) f[q] = fb[q];
      }
      stv<DIM>(d.f, i, f);
      if (VERLET && (fl[k] & NODE_ACTIVE)) {
        const uint8_t fix = d.fix[i];
        double v[3];
        ldv<DIM>(d.v, i, v);
        const double kk = 0.5 * (d.dt / rho);
#pragma unroll
        for (int dof = 0; dof < DIM; dof++)
          if (!((fix >> dof) & 1u)) v[dof] += kk * f[dof];
        stv<DIM>(d.v, i, v);
        d.vmag[i] = len3<DIM>(v);
      }
    }
  }
  // the post-processing tail only on the steps that record test output
  if (!post || d.test == PDGPU_TEST_NONE) return;
  if (!(n_step % d.test_interval == 0 && n_step >= d.test_interval)) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&d.ctrl->end_done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    __threadfence();
    if (threadIdx.x == 0) d.ctrl->end_done = 0u;
    postprocess_block<DIM>(d);
  }
}

// ---------------------------------------------------------------------------
// Between two steps of a graph: the last kernel of one step (k_step_end) and
// the first of the next (k_step_begin) in one pass over the nodes, with their
// operations in their order: f is written but not read again, node constants
// and control state are read once, and a launch goes.  On test-output steps
// the positions the post-processing needs go to d.turn before they move on;
// the last CTA runs it, then the step control.
//
// For scenes up to about a wave of CTAs (kTurnMaxNodes), where the two kernels are
// a chain of latencies: us per step without / with it, two discs FP64 14.8 / 13.1,
// PMB with Verlet 18.5 / 15.7, 24 000 nodes 26.4 / 24.9, 151 000 nodes 32.5 / 28.8
// (FP64 52.3 / 48.6); 3-D, 113 000 nodes 84.4 / 81.3, 147 000 nodes 56.4 / 54.7
// (Verlet 96.5 / 93.3, FP64 114.8 / 112.6).  Larger ones gain nothing (332 000
// nodes 49.2 / 49.2 to 50.0, 1.3 M 154.1 / 152.8 to 158.7 over one or two nodes
// per thread, bulk prefetch of later CTAs' nodes 156.5; 3-D, 244 000 nodes
// 142.8 / 144.4): the traffic saved is a tenth, and the longer kernel holds fewer
// warps.
// ---------------------------------------------------------------------------
template <int DIM, bool VERLET>
__global__ void __launch_bounds__(kBlock) k_step_turn(const __grid_constant__ DevData d) {
  __shared__ double smax[kBlock / 32];
  __shared__ int last;
  __shared__ __align__(8) CtrlState s_ctrl;
  pdl_start();
  if (threadIdx.x < sizeof(CtrlState) / 8)
    reinterpret_cast<uint64_t *>(&s_ctrl)[threadIdx.x] = reinterpret_cast<const uint64_t *>(d.ctrl)[threadIdx.x];
  const int64_t n_step = d.ctrl->n;
  const double time = d.ctrl->time;
  const bool post = d.test != PDGPU_TEST_NONE && n_step % d.test_interval == 0 && n_step >= d.test_interval;
  // reverse node order, as step begin
  const int64_t i = (int64_t)(gridDim.x - 1 - blockIdx.x) * kBlock + threadIdx.x;
  double vm = 0.0;
  unsigned long long ymax = 0;
  if (!d.ctrl->error && i < d.n_nodes) {
    double v[3], u[3], x[3], f[3];
    const uint8_t fl = d.flags[i], fix = d.fix[i];
    const int32_t pid = d.ptid[i];
    ldv<DIM>(d.f, i, f);
    ldv<DIM>(d.v, i, v);
    ldv<DIM>(d.u, i, u);
    ldv<DIM>(d.x, i, x);
    const bool active = fl & NODE_ACTIVE;
    const double rho = d.particles[pid].density;
    // ---- end of the step (k_step_end)
    if (!active) f[0] = f[1] = f[2] = 0.0;
    if (active && d.fc && (fl & (NODE_SEARCH | NODE_SEARCH0))) {
      double c[3];
      ldv<DIM>(d.fc, i, c);
      if (c[0] != 0.0 || c[1] != 0.0 || (DIM == 3 && c[2] != 0.0)) {
#pragma unroll
        for (int q = 0; q < DIM; q++) f[q] += c[q];
        const double z[3] = {0.0, 0.0, 0.0};
        stv<DIM>(d.fc, i, z);
      }
    }
    if (fl & NODE_PARTICLE) {
#pragma unroll
      for (int q = 0; q < DIM; q++) f[q] += d.fdamp[4 * pid + q];
    }
    if (d.gravity_on) {
#pragma unroll
      for (int q = 0; q < DIM; q++) f[q] += rho * d.gravity[q];
    }
    if (fl & NODE_FBC) {  // through a copy, so that f stays in registers
      double fb[3] = {f[0], f[1], f[2]};
      apply_fbc<DIM>(d, d.fbc_of[i], time, fb);
#pragma unroll
      for (int q = 0; q < 3; q++) f[q] = fb[q];
    }
    stv<DIM>(d.f, i, f);
    if (post) {
      TurnState *t = d.turn;
      if (d.test == PDGPU_TEST_COMPRESSIVE) {
        if (i == d.particles[d.test_wall].start)
          for (int q = 0; q < DIM; q++) t->wall[q] = x[q];
      } else if (d.n_particles >= 2 && pid <= 1) {
        if (i == d.particles[pid].center)
          for (int q = 0; q < DIM; q++) t->centre[pid][q] = x[q];
        if (pid == 1 && x[1] == x[1]) ymax = to_key(x[1]);
      }
    }
    // ---- begin of the next (k_step_begin)
    if (fl & (NODE_ACTIVE | NODE_UBC)) {
      if (active) {
        const double dt = d.dt;
        const double kk = VERLET ? 0.5 * (dt / rho) : dt / rho;
#pragma unroll
        for (int dof = 0; dof < DIM; dof++) {
          if (!((fix >> dof) & 1u)) {
            if (VERLET) v[dof] += kk * f[dof];  // the ended step's second half
            v[dof] += kk * f[dof];
            u[dof] += dt * v[dof];
            x[dof] += dt * v[dof];
          }
        }
        vm = len3<DIM>(v);
        d.vmag[i] = vm;
      }
      if (fl & NODE_UBC) {
        double ub[3], vb[3], xb[3];
#pragma unroll
        for (int q = 0; q < 3; q++) ub[q] = u[q], vb[q] = v[q], xb[q] = x[q];
        apply_ubc<DIM>(d, d.ubc_of[i], i, time + d.dt, 0, ub, vb, xb);
#pragma unroll
        for (int q = 0; q < 3; q++) u[q] = ub[q], v[q] = vb[q], x[q] = xb[q];
      }
      stv<DIM>(d.v, i, v);
      stv<DIM>(d.u, i, u);
      stv<DIM>(d.x, i, x);
    }
  }
  if (post && d.test == PDGPU_TEST_TWO_PARTICLE && ymax) atomicMax(&d.turn->max_y, ymax);
  // block max of |v| -> one atomic per block
  for (int o = 16; o > 0; o >>= 1) vm = fmax(vm, __shfl_xor_sync(0xffffffffu, vm, o));
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = vm;
  if (post) __threadfence();  // this thread's f and d.turn, for the last CTA
  __syncthreads();
  if (threadIdx.x < 32) {
    double m = threadIdx.x < kBlock / 32 ? smax[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) {
      if (m > 0.0) atomic_max_nonneg(&d.ctrl->vmax_bits, m);
      __threadfence();
      last = atomicAdd(&d.ctrl->begin_done, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (post) {
    __shared__ TurnState s_turn;
    if (threadIdx.x == 0) {
      for (int q = 0; q < 3; q++) {
        s_turn.wall[q] = __ldcg(d.turn->wall + q);
        s_turn.centre[0][q] = __ldcg(d.turn->centre[0] + q);
        s_turn.centre[1][q] = __ldcg(d.turn->centre[1] + q);
      }
      s_turn.max_y = atomicExch(&d.turn->max_y, 0ull);
    }
    __syncthreads();
    postprocess_block<DIM>(d, &s_turn);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    d.ctrl->begin_done = 0u;
    ctrl_step(d, 0, &s_ctrl);
  }
}

// ---------------------------------------------------------------------------
// Set-up kernels
// ---------------------------------------------------------------------------

// DEMModel::updatePeridynamicNeighborlist (demModel.cpp:1659-1694): same
// particle, j != i, strict squared distance against horizon^2, computed in
// nanoflann's order (query minus point, dims 0..2).
template <int DIM, int LPN, bool FILL>
__global__ void __launch_bounds__(kBlock) k_pd_cand(DevData d, Grid g, int64_t *row) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LPN;
  const int lane = threadIdx.x % LPN;
  if (i >= d.n_nodes) return;
  const unsigned gm = group_mask<LPN>();
  const unsigned lane_base = (threadIdx.x & 31u) / LPN * LPN;
  double q[3];
  ldv<DIM>(d.x, i, q);
  const int32_t pi = d.ptid[i];
  const double r = d.particles[pi].horizon;
  const double r2 = r * r;
  int c[3] = {cell_coord<DIM>(q[0], g, 0), cell_coord<DIM>(q[1], g, 1),
              DIM == 3 ? cell_coord<DIM>(q[2], g, 2) : 0};
  int64_t out = FILL ? row[i] : 0;
  int64_t count = 0;
  const int zlo = DIM == 3 ? max(c[2] - 1, 0) : 0;
  const int zhi = DIM == 3 ? min(c[2] + 1, g.dims[2] - 1) : 0;
  for (int cz = zlo; cz <= zhi; cz++)
    for (int cy = max(c[1] - 1, 0); cy <= min(c[1] + 1, g.dims[1] - 1); cy++)
      for (int cx = max(c[0] - 1, 0); cx <= min(c[0] + 1, g.dims[0] - 1); cx++) {
        const int cell = cx + g.dims[0] * (cy + g.dims[1] * cz);
        const int s = d.cell_start[cell], e = d.cell_start[cell + 1];
        for (int base = s; base < e; base += LPN) {
          const int a = base + lane;
          bool hit = false;
          int32_t j = -1;
          if (a < e) {
            j = d.cell_nodes[a];
            if (j != i && d.ptid[j] == pi) {
              double p[3];
              ldv<DIM>(d.x, j, p);
              double dd = 0.0;
#pragma unroll
              for (int t = 0; t < DIM; t++) {
                const double df = q[t] - p[t];
                dd += df * df;
              }
              hit = dd < r2;
            }
          }
          const unsigned bal = (__ballot_sync(gm, hit) & gm) >> lane_base;
          if (FILL) {
            if (hit) d.pd_col[out + __popc(bal & ((1u << lane) - 1u))] = j;
            out += __popc(bal);
          } else {
            count += __popc(bal);
          }
        }
      }
  if (!FILL && lane == 0) row[i + 1] = count;
}

// order each node's neighbour list by node index (one warp per node)
__global__ void k_pd_sort_rows(DevData d, int32_t *tmp) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= d.n_nodes) return;
  const int64_t s = d.pd_row[i], e = d.pd_row[i + 1];
  for (int64_t a = s + lane; a < e; a += 32) tmp[a] = d.pd_col[a];
  __syncwarp();
  for (int64_t a = s + lane; a < e; a += 32) {
    const int32_t va = tmp[a];
    int64_t rank = 0;
    for (int64_t b = s; b < e; b++) rank += tmp[b] < va;
    d.pd_col[s + rank] = va;
  }
}

// material::computeStateMxI (materialUtil.cpp:21-73).  One thread per node
// sums its row in list order, as the reference does, so that with the
// reference's own neighbour order the result is the reference's to the bit
// (FP64, no FMA contraction in this unit).
template <int DIM, int LPN>
__global__ void k_mx(DevData d) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LPN;
  const int lane = threadIdx.x % LPN;
  if (i >= d.n_nodes) return;
  const unsigned gm = group_mask<LPN>();
  const DevParticle &P = d.particles[d.ptid[i]];
  double xi[3];
  ldv<DIM>(d.xref, i, xi);
  double m = 0.0;
  for (int64_t k = d.pd_row[i] + lane; k < d.pd_row[i + 1]; k += LPN) {
    const int32_t j = d.pd_col[k];
    double xj[3], dx[3];
    ldv<DIM>(d.xref, j, xj);
    for (int q = 0; q < 3; q++) dx[q] = xj[q] - xi[q];
    const double rji = len3<DIM>(dx);
    if (is_greater(rji, P.horizon)) continue;
    double volj = d.vol[j];
    if (is_greater(rji, P.check_low)) volj *= (P.check_up - rji) / P.h;
    m += rji * rji * influence(d.inf, rji, P.horizon) * volj;
  }
  m = group_sum<LPN>(m, gm);
  if (lane == 0) {
    d.mx[i] = m;
    if (is_less(m, 1.0e-18)) set_error(d.ctrl, DEV_ERR_NONFINITE, i);
  }
}

inline unsigned blocks_for(int64_t n, int per_block) {
  return (unsigned)((n + per_block - 1) / per_block);
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

#define PDGPU_DIM_DISPATCH(d, KERNEL, ...)            \
  do {                                               \
    if ((d).dim == 2) KERNEL<2> __VA_ARGS__;         \
    else KERNEL<3> __VA_ARGS__;                      \
  } while (0)

void launch_pack_vec(const DevData &d, const double *aos3, double *dst, cudaStream_t s) {
  PDGPU_DIM_DISPATCH(d, k_pack, <<<blocks_for(d.n_nodes, kBlock), kBlock, 0, s>>>(aos3, dst, d.n_nodes));
}
void launch_unpack_vec(const DevData &d, const double *src, double *aos3, cudaStream_t s) {
  PDGPU_DIM_DISPATCH(d, k_unpack, <<<blocks_for(d.n_nodes, kBlock), kBlock, 0, s>>>(src, aos3, d.n_nodes));
}
void launch_apply_ic(const DevData &d, cudaStream_t s) {
  PDGPU_DIM_DISPATCH(d, k_apply_ic, <<<blocks_for(d.n_nodes, kBlock), kBlock, 0, s>>>(d));
}
void launch_integrate(const DevData &d, int verlet, cudaStream_t s) {
  const unsigned g = blocks_for(d.n_nodes, kBlock);
  if (d.dim == 2) {
    if (verlet) k_integrate<2, true><<<g, kBlock, 0, s>>>(d);
    else k_integrate<2, false><<<g, kBlock, 0, s>>>(d);
  } else {
    if (verlet) k_integrate<3, true><<<g, kBlock, 0, s>>>(d);
    else k_integrate<3, false><<<g, kBlock, 0, s>>>(d);
  }
}
void launch_verlet_second(const DevData &d, cudaStream_t s) {
  PDGPU_DIM_DISPATCH(d, k_verlet_second, <<<blocks_for(d.n_nodes, kBlock), kBlock, 0, s>>>(d));
}
void launch_ctrl(const DevData &d, int mode, cudaStream_t s) { k_ctrl<<<1, 1, 0, s>>>(d, mode); }
void launch_bc(const DevData &d, cudaStream_t s) {
  if (!d.n_ubc_nodes) return;
  PDGPU_DIM_DISPATCH(d, k_bc, <<<blocks_for(d.n_ubc_nodes, 128), 128, 0, s>>>(d));
}

size_t scan_temp_bytes(int64_t n) {
  size_t a = 0, b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, a, (int32_t *)nullptr, (int32_t *)nullptr, (int)n);
  cub::DeviceScan::InclusiveSum(nullptr, b, (int64_t *)nullptr, (int64_t *)nullptr, n);
  return a > b ? a : b;
}


template <int DIM>
static cudaError_t rebuild_dim(const DevData &d, uint8_t bit, int64_t *bsum, int grid, cudaStream_t s) {
  DevData dd = d;
  void *args[] = {(void *)&dd, (void *)&bit, (void *)&bsum};
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(kCoopBlock);
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 2;
  return cudaLaunchKernelExC(&c, (const void *)k_contact_rebuild<DIM>, args);
}

// Blocks of the cooperative rebuild: at most what is resident at once, and no
// more than the nodes and cells keep busy (the whole
// rebuild of a 634-node scene: 69 us with every resident block, 27 us with five)
int rebuild_grid_blocks(const DevData &d) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const void *f = d.dim == 2 ? (const void *)k_contact_rebuild<2> : (const void *)k_contact_rebuild<3>;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, kCoopBlock, 0);
  const int64_t most = (int64_t)sms * (per > 0 ? per : 1);
  const int64_t want = std::max<int64_t>((d.n_nodes + 127) / 128, ((int64_t)d.grid.ncells + 31) / 32);
  return (int)std::min(most, want);
}

cudaError_t launch_contact_rebuild(const DevData &d, int64_t *bsum, int grid, int init, cudaStream_t s) {
  const uint8_t bit = init ? NODE_SEARCH0 : NODE_SEARCH;
  return d.dim == 2 ? rebuild_dim<2>(d, bit, bsum, grid, s) : rebuild_dim<3>(d, bit, bsum, grid, s);
}

int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

void launch_contact_owner(const DevData &d, cudaStream_t s) {
  k_contact_owner<<<sm_count() * 4, kBlock, 0, s>>>(d);
}

void launch_contact_force(const DevData &d, int lanes, cudaStream_t s) {
  const unsigned g = (unsigned)d.contact_grid;
  if (lanes == 1) {  // one kernel, a warp per 32 nodes
    const unsigned gc = g + blocks_for(d.n_particles, kBlock / 32);
    // In front of the FP32 2-D bond loop (150 KB of shared memory per SM over its
    // ten CTAs) the pass asks for the same carve-out, since an SM changes its
    // carve-out only when empty: the bond loop's CTAs then start beside the
    // contact pass's.  us per step without / with: two discs 14.7 / 14.5, 24 000
    // nodes 22.9 / 21.5, 332 000 47.9 / 47.7, an ensemble of 416 000 55.3 / 55.3.
    // Not for 1.3 M nodes, where the pass wants its L1 (154.0 / 154.9), nor before
    // the FP64 loop (88.8 / 90.0).
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(gc);
    c.blockDim = dim3(kBlock);
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = d.precision == PDGPU_PREC_MIXED && d.dim == 2 && d.n_nodes <= 4 * kTurnMaxNodes ? 1 : 0;
    cudaLaunchKernelEx(&c, d.dim == 2 ? k_contact_warp<2> : k_contact_warp<3>, d);
    return;
  }
  PDGPU_DIM_DISPATCH(d, k_damp_pairs, <<<blocks_for(d.n_particles, kBlock / 32), kBlock, 0, s>>>(d));
  // the distance pass: eight CTAs per SM, grid-stride over the entries
  if (d.dim == 2) k_contact_near<2><<<sm_count() * 8, kBlock, 0, s>>>(d);
  else k_contact_near<3><<<sm_count() * 8, kBlock, 0, s>>>(d);
  if (d.dim == 2) {
    if (lanes == 1) k_contact<2, 1><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 2) k_contact<2, 2><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 4) k_contact<2, 4><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 8) k_contact<2, 8><<<g, kBlock, 0, s>>>(d);
    else k_contact<2, 32><<<g, kBlock, 0, s>>>(d);
  } else {
    if (lanes == 1) k_contact<3, 1><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 2) k_contact<3, 2><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 4) k_contact<3, 4><<<g, kBlock, 0, s>>>(d);
    else if (lanes == 8) k_contact<3, 8><<<g, kBlock, 0, s>>>(d);
    else k_contact<3, 32><<<g, kBlock, 0, s>>>(d);
  }
}

void launch_scene_post(const DevData &d, cudaStream_t s) {
  if (d.n_scenes <= 1) return;
  launch_dependent(d.dim == 2 ? k_scene_post<2> : k_scene_post<3>, d.n_scenes, 256, 0, s, d);
}

void launch_damping(const DevData &d, cudaStream_t s) {
  if (!d.has_walls) return;
  launch_dependent(d.dim == 2 ? k_damp_walls<2> : k_damp_walls<3>, blocks_for(d.n_particles, kDampBlock / 32),
                   kDampBlock, 0, s, d);
}

void launch_external(const DevData &d, cudaStream_t s) {
  PDGPU_DIM_DISPATCH(d, k_external, <<<blocks_for(d.n_nodes, kBlock), kBlock, 0, s>>>(d));
  if (d.n_fbc_nodes)
    PDGPU_DIM_DISPATCH(d, k_force_bc, <<<blocks_for(d.n_fbc_nodes, 128), 128, 0, s>>>(d));
}

void launch_step_begin(const DevData &d, int verlet, cudaStream_t s) {
  const unsigned g = blocks_for(d.n_nodes, kBlock * kBeginNodes);
  if (d.dim == 2) launch_dependent(verlet ? k_step_begin<2, true> : k_step_begin<2, false>, g, kBlock, 0, s, d);
  else launch_dependent(verlet ? k_step_begin<3, true> : k_step_begin<3, false>, g, kBlock, 0, s, d);
}

void launch_step_end(const DevData &d, int verlet, int post, cudaStream_t s) {
  const unsigned g = blocks_for(d.n_nodes, kBlock * kEndNodes);
  if (d.dim == 2) {
    if (verlet) k_step_end<2, true><<<g, kBlock, 0, s>>>(d, post);
    else k_step_end<2, false><<<g, kBlock, 0, s>>>(d, post);
  } else {
    if (verlet) k_step_end<3, true><<<g, kBlock, 0, s>>>(d, post);
    else k_step_end<3, false><<<g, kBlock, 0, s>>>(d, post);
  }
}

void launch_step_turn(const DevData &d, int verlet, cudaStream_t s) {
  const unsigned g = blocks_for(d.n_nodes, kBlock);
  if (d.dim == 2) {
    if (verlet) k_step_turn<2, true><<<g, kBlock, 0, s>>>(d);
    else k_step_turn<2, false><<<g, kBlock, 0, s>>>(d);
  } else {
    if (verlet) k_step_turn<3, true><<<g, kBlock, 0, s>>>(d);
    else k_step_turn<3, false><<<g, kBlock, 0, s>>>(d);
  }
}

void launch_postprocess(const DevData &d, cudaStream_t s) {
  if (d.test == PDGPU_TEST_NONE) return;
  PDGPU_DIM_DISPATCH(d, k_postprocess, <<<1, 1024, 0, s>>>(d));
}

void launch_build_pd(const DevData &d, double cell, int64_t *row, int32_t *tmp, void *scan_tmp,
                     size_t scan_bytes, int pass, cudaStream_t s) {
  // pass 0: grid + counts; pass 1: fill + sort rows.  d.grid holds the
  // horizon-sized grid built by the caller; d.ctrl->update must be 1.
  const int lanes = d.dim == 2 ? 8 : 32;
  const unsigned g = blocks_for(d.n_nodes * lanes, kBlock);
  (void)cell;
  if (pass == 0) {
    const unsigned gn = blocks_for(d.n_nodes, kBlock);
    k_zero_cells<<<blocks_for(d.grid.ncells + 1, kBlock), kBlock, 0, s>>>(d);
    PDGPU_DIM_DISPATCH(d, k_cell_count, <<<gn, kBlock, 0, s>>>(d, d.x, d.grid));
    cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, d.cell_cnt, d.cell_start, d.grid.ncells + 1, s);
    k_cell_scatter<<<gn, kBlock, 0, s>>>(d);
    k_cell_sort<<<blocks_for((int64_t)d.grid.ncells * 32, kBlock), kBlock, 0, s>>>(d);
    if (d.dim == 2) k_pd_cand<2, 8, false><<<g, kBlock, 0, s>>>(d, d.grid, row);
    else k_pd_cand<3, 32, false><<<g, kBlock, 0, s>>>(d, d.grid, row);
    cub::DeviceScan::InclusiveSum(scan_tmp, scan_bytes, row + 1, row + 1, d.n_nodes, s);
  } else {
    if (d.dim == 2) k_pd_cand<2, 8, true><<<g, kBlock, 0, s>>>(d, d.grid, row);
    else k_pd_cand<3, 32, true><<<g, kBlock, 0, s>>>(d, d.grid, row);
    k_pd_sort_rows<<<blocks_for(d.n_nodes * 32, kBlock), kBlock, 0, s>>>(d, tmp);
  }
}

void launch_compute_mx(const DevData &d, cudaStream_t s) {
  const unsigned g = blocks_for(d.n_nodes, kBlock);
  if (d.dim == 2) k_mx<2, 1><<<g, kBlock, 0, s>>>(d);
  else k_mx<3, 1><<<g, kBlock, 0, s>>>(d);
}

}  // namespace pdgpu
