// Tiled bond loop of DEMModel::computePeridynamicForces
// (demModel.cpp:602-789), FP64 form: the reference's arithmetic (compiled with
// --fmad=false; its order of operations, quotients and square roots rounded to
// nearest but for the cases pdgpu_quot.cuh names).
//
// One CTA per tile of one particle's nodes.  The tile's neighbour columns,
// row offsets and words of the broken-bond bitmap and the window of nodes its
// bonds reach arrive in shared memory by bulk copies, so the bond loop reads
// only shared memory; each law is its own instantiation.
//
// What bounds it: the FP64 pipe (64 lanes per SM) and the latency of its
// chains.  A bond needs up to 13 quotients and roots, many instructions each as
// plain divisions and sqrt; here
//   * sqrt(a), 1/sqrt(a) and quotients by one correction each (pdgpu_quot.cuh),
//     a quotient at three operations;
//   * quantities of one node (15 G / m_x, 3 K / m_x - 5 G / m_x) are computed
//     once per node at set-up instead of once per bond.
// A node is summed without tests of broken or breaking bonds first; the tests
// run in a second sum of that node where they can matter.
//
// Measured per launch (B200, us), against one CTA per tile with the compiler's
// divides, the law chosen per bond and every operand in its own array:
//   2-D, RNP, 333 000 nodes, 7.6 M bonds: 226 -> 74 (FP64 pipe 59 % and issue
//   71 % busy; 78 FP64 and 105 other thread instructions per bond, the nodes'
//   own included);
//   3-D, PD state, 75 000 sphere nodes, 6.4 M bonds: pre-pass 126 -> 54, main
//   loop 337 -> 69 (FP64 pipe 48 and 53 %, issue 45 and 46 % at one CTA per SM);
//   3-D, PD elastic, 63 000 sphere nodes, 5.3 M bonds: 304 -> 55 (54 %, 48 %).
// The outputs are the same to the bit at equal lanes per node.  Four CTAs of
// 256 threads per SM in 2-D (64 registers; 32 to 84 bytes of spill stores and 36
// to 116 of spill loads in the main loops): a step of the 333 000-node RNP
// compression takes 91.8 us, with three (80 registers) 94.5; with two (114
// registers) the launch alone took a third longer.  The other laws run that way
// too; 151 000 nodes, us per step before and now: PMB 106.9 -> 45.8, PD elastic
// 124.6 -> 47.7, PD state 173.8 -> 80.1.
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "pdgpu_bulk.cuh"
#include "pdgpu_internal.h"
#include "pdgpu_pdl.cuh"
#include "pdgpu_quot.cuh"

namespace pdgpu {
namespace {

// threads per CTA: in 3-D a tile's window takes 100-200 KB of shared memory,
// one CTA fits an SM, and 512 threads fill its register file
template <int DIM>
constexpr int kThreads64 = DIM == 3 ? 512 : 256;

enum { LAW_RNP = 0, LAW_PMB = 1, LAW_ELASTIC = 2, LAW_STATE = 3 };

// util::isGreater (function.cpp:15-18)
__device__ __forceinline__ bool gt(double a, double b) {
  const double fa = fabs(a), fb = fabs(b);
  return (a - b) > ((fa < fb ? fb : fa) * 1.0e-5);
}

// Shared-memory plan of one tile (byte offsets), identical on host and
// device.  The window's node data always sit in shared memory; where it is
// too wide for the rest, first the state law's {3K/m - 5G/m, 15G/m} pairs, then
// its dilatations, then the bond data stay in global memory (ST_* bits).
enum { ST_FA = 1, ST_TH = 2, ST_BONDS = 4, ST_ALL = 7 };

struct Plan64 {
  int64_t col0, word0, row0, vol0;
  uint32_t col_bytes, bit_bytes, row_bytes, vol_bytes;
  uint32_t off_bits, off_row, off_x, off_u, off_z, off_vol, off_th, off_fa, total;
};

__host__ __device__ inline Plan64 plan64(int dim, bool state, int stage, int col_size, const BondTile &T) {
  Plan64 p{};
  const int64_t w = T.win_end - T.win_begin;
  const int64_t per16 = 16 / col_size;
  uint32_t at = 0;
  if (stage & ST_BONDS) {
    p.col0 = T.bond_begin / per16 * per16;
    p.col_bytes = (uint32_t)(((T.bond_end + per16 - 1) / per16 * per16 - p.col0) * col_size);
    p.word0 = (T.bond_begin >> 5) / 4 * 4;
    p.bit_bytes = (uint32_t)((((((T.bond_end + 31) >> 5) + 3) / 4 * 4) - p.word0) * 4);
    p.row0 = T.node_begin / 2 * 2;
    p.row_bytes = (uint32_t)(((T.node_end + 2) / 2 * 2 - p.row0) * 8);
    p.off_bits = p.col_bytes;
    p.off_row = p.off_bits + p.bit_bytes;
    at = p.off_row + p.row_bytes;
  }
  p.off_x = at;  // 2-D double2 {x, y}; 3-D double4 {x, y, z, vol}
  at += (uint32_t)((dim == 2 ? 16 : 32) * w);
  p.off_u = at;  // double2 {ux, uy}
  at += (uint32_t)(16 * w);
  if (dim == 3) {
    p.off_z = at;  // double uz
    at += (uint32_t)((8 * w + 15) / 16 * 16);
  } else {
    p.vol0 = T.win_begin / 2 * 2;
    p.vol_bytes = (uint32_t)(((T.win_end + 1) / 2 * 2 - p.vol0) * 8);
    p.off_vol = at;  // double vol
    at += p.vol_bytes;
  }
  if (state && (stage & ST_TH)) {
    p.off_th = at;
    at += (uint32_t)((8 * w + 15) / 16 * 16);
  }
  if (state && (stage & ST_FA)) {
    p.off_fa = at;
    at += (uint32_t)(16 * w);
  }
  p.total = at;
  return p;
}

template <int DIM>
__device__ __forceinline__ double dotd(const double (&a)[3], const double (&b)[3]) {
  double s = a[0] * b[0] + a[1] * b[1];
  if constexpr (DIM == 3) s = s + a[2] * b[2];
  return s;
}

// the staged window
template <int DIM>
struct Win {
  const double2 *x, *u;
  const double *z, *vol;
  __device__ __forceinline__ void node(int l, double (&xq)[3], double (&uq)[3], double &v) const {
    if constexpr (DIM == 2) {
      const double2 a = x[l];
      xq[0] = a.x, xq[1] = a.y, xq[2] = 0.0;
      v = vol[l];
    } else {
      const double2 a = x[2 * l], b = x[2 * l + 1];
      xq[0] = a.x, xq[1] = a.y, xq[2] = b.x;
      v = b.y;
    }
    const double2 c = u[l];
    uq[0] = c.x, uq[1] = c.y;
    uq[2] = DIM == 3 ? z[l] : 0.0;
  }
};

// a particle's constants and its tile's view, held in registers
template <int DIM>
struct Bond64 {
  Win<DIM> V;
  double p0, p1, inv_p1, horizon, inv_hor, h, inv_h, up, low;
  double m0, m1, m2, m3, m4, inv_m3, kn, rc;
  bool irrev, gauss;
  const double *th;    // state: dilatation of a window node
  const double2 *fa;   // state: {3K/m - 5G/m, 15G/m} of a window node

  // J(r / horizon) (influenceFn.cpp:21-23, 55-57, 86-88); a constant function
  // is a linear one of slope 0
  __device__ __forceinline__ double infl(double r) const {
    const double q = quot(r, horizon, inv_hor);
    if (!gauss) return p0 + p1 * q;
    return p0 * exp(quot(-q * q, p1, inv_p1));
  }
  // volume of a neighbour inside the horizon, by its distance (isGreater for
  // r > 0, low >= 0: below low the difference is negative)
  __device__ __forceinline__ double corrected(double r, double vol) const {
    const double t = vol * quot(up - r, h, inv_h);
    return (r - low) > r * 1.0e-5 ? t : vol;
  }
};

__device__ __forceinline__ bool not_finite(double a) { return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000; }

template <int LPN>
__device__ __forceinline__ double gmax64(double v, int lanes) {
#pragma unroll
  for (int o = (LPN ? LPN : lanes) / 2; o > 0; o >>= 1) {
    const double b = __shfl_xor_sync(kFullWarp, v, o);
    v = b > v ? b : v;
  }
  return v;
}

struct Node64 {
  double x[3], u[3];
  double th, f, a;
};

struct Sum64 {
  double f[3], zmax, theta;
};

// One bond (i, j).  TEST: the bond may be broken or break now (returned true);
// a bond that breaks carries no force and repels from the next evaluation on.
// Without TEST neither is looked at: a node none of whose bonds starts broken
// is summed that way first, and again with TEST only when its largest stretch
// measure could break a bond or a stretch may have overflowed (the caller's
// decision): only TEST yields an infinite stretch, where the other yields NaN,
// which the largest measure passes over.  RANGE: every reference
// distance of the lists is inside root_in_range's.
template <int DIM, int LAW, bool PRE, bool TEST, bool RANGE>
__device__ __forceinline__ bool bond64(const Bond64<DIM> &B, const Node64 &I, int lj, bool broken, Sum64 &s) {
  double xj[3], uj[3], volj, dx[3], du[3], y[3];
  B.V.node(lj, xj, uj, volj);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    dx[q] = xj[q] - I.x[q];
    if constexpr (PRE) {
      y[q] = (dx[q] + uj[q]) - I.u[q];
    } else {
      du[q] = uj[q] - I.u[q];
      y[q] = dx[q] + du[q];
    }
  }
  const double r2 = dotd<DIM>(dx, dx);
  const Root R = RANGE ? root_in_range(r2) : root(r2);
  const double rji = R.r;
  auto stretch = [](double a, double b, double y) { return TEST ? quot_or_inf(a, b, y) : quot(a, b, y); };
  bool breaks = false;
  double S, ly = 0.0, inv_ly = 0.0, cl = 0.0;
  if constexpr (LAW == LAW_RNP) {
    S = stretch(dotd<DIM>(dx, du), r2, R.inv * R.inv);
    const double zq = S * S * rji;  // Z = |S| sqrt(r) / rbar
    s.zmax = zq > s.zmax ? zq : s.zmax;
  } else {
    const Root L = root(dotd<DIM>(y, y));
    ly = L.r;
    inv_ly = L.inv;
    cl = ly - rji;
    S = stretch(cl, rji, R.inv);
    const double za = fabs(S);
    s.zmax = za > s.zmax ? za : s.zmax;
  }
  if constexpr (PRE) {
    if constexpr (TEST) {
      if (broken) return false;
      breaks = gt(fabs(S), B.m2 + 1.0e-10);
    }
    if (!breaks) s.theta += rji * cl * B.infl(rji) * B.corrected(rji, volj);
    return breaks;
  } else {
    if constexpr (TEST) {
      if (broken) {
        // y = (xj + uj) - (xi + ui) (demModel.cpp:762)
        double yb[3];
#pragma unroll
        for (int q = 0; q < 3; q++) yb[q] = (xj[q] + uj[q]) - (I.x[q] + I.u[q]);
        const double Rb = sqrt(dotd<DIM>(yb, yb));
        double sf = B.kn * volj * (Rb - B.rc) / Rb;
        if (sf > 0.) sf = 0.;
#pragma unroll
        for (int q = 0; q < DIM; q++) s.f[q] += sf * yb[q];
        return false;
      }
      if constexpr (LAW == LAW_RNP) breaks = B.irrev && gt(fabs(S), B.m4 * (B.m2 / sqrt(rji)));
      if constexpr (LAW == LAW_PMB) breaks = gt(fabs(S), B.m1 + 1.0e-10);
    }
    double ef = 0.0;
    const double J = B.infl(rji);
    if constexpr (LAW == LAW_RNP) {
      if (!breaks) ef = quot(J * 4. * S * B.m0 * B.m1 * exp(-B.m1 * rji * S * S), B.m3, B.inv_m3);
    } else if constexpr (LAW == LAW_STATE) {
      const double2 fj = B.fa[lj];
      cl = S * rji;
      const double efi = J * (rji * I.th * I.f + cl * I.a);
      const double efj = J * (rji * B.th[lj] * fj.x + cl * fj.y);
      ef = efi + efj;
    } else {
      if (!breaks) ef = J * B.m0 * S;
    }
    const double sf = ef * B.corrected(rji, volj);
    // bond-based RNP acts along the reference bond, the others along y
    const double len = LAW == LAW_RNP ? rji : ly, inv = LAW == LAW_RNP ? R.inv : inv_ly;
#pragma unroll
    for (int q = 0; q < DIM; q++) s.f[q] += sf * quot(LAW == LAW_RNP ? dx[q] : y[q], len, inv);
    return breaks;
  }
}

// PRE: the PD state pre-pass (demModel.cpp:610-679); else the main loop
// (:685-788).  COL: type of the staged neighbour columns (uint16_t
// particle-local or int32_t global); COL = void reads whatever form the
// columns have, with the row offsets and bitmap, from global memory (tiles
// whose window leaves no room, and reference distances outside the range of
// the unchecked root).  LPN lanes per node; LPN = 0, of the last two, whose
// scenes are rare: as many as `lanes` says.
template <int DIM, int LPN, int LAW, bool PRE, typename COL>
__global__ void __launch_bounds__(kThreads64<DIM>, DIM == 2 ? 4 : 1)
    k_bonds_fp64(const __grid_constant__ DevData d, const BondTile *__restrict__ tiles, int stage, int lanes) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  constexpr int kT = kThreads64<DIM>;
  constexpr bool kState = LAW == LAW_STATE && !PRE;
  constexpr bool kStaged = !std::is_void<COL>::value;
  pdl_start();
  pdl_wait();
  if (d.ctrl->error) return;
  const BondTile T = tiles[blockIdx.x];
  const DevParticle &P = d.particles[T.particle];
  const int w = (int)(T.win_end - T.win_begin);
  const Plan64 p = plan64(DIM, kState, stage, d.use16 ? 2 : 4, T);
  constexpr int st = DIM == 2 ? 2 : 4;
  double2 *s_u = reinterpret_cast<double2 *>(smem + p.off_u);
  double *s_z = reinterpret_cast<double *>(smem + p.off_z);
  if (threadIdx.x == 0) bar_init(&bar);
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t xb = (DIM == 2 ? 16u : 32u) * (uint32_t)w;
    const uint32_t ub = DIM == 2 ? 16u * (uint32_t)w : 0u;
    const bool fa = kState && (stage & ST_FA);
    bar_arrive_tx(&bar, p.col_bytes + p.bit_bytes + p.row_bytes + xb + ub + p.vol_bytes + (fa ? 16u * (uint32_t)w : 0u));
    bulk_load(smem + p.off_x, d.xref + st * T.win_begin, xb, &bar);
    if constexpr (DIM == 2) {
      bulk_load(smem + p.off_u, d.u + st * T.win_begin, ub, &bar);
      bulk_load(smem + p.off_vol, d.vol + p.vol0, p.vol_bytes, &bar);
    }
    if constexpr (kStaged) {
      const COL *col = std::is_same<COL, uint16_t>::value ? (const COL *)d.pd_col16 : (const COL *)d.pd_col;
      if (p.col_bytes) bulk_load(smem, col + p.col0, p.col_bytes, &bar);
      if (p.bit_bytes) bulk_load(smem + p.off_bits, d.bond_bits + p.word0, p.bit_bytes, &bar);
      bulk_load(smem + p.off_row, d.pd_row + p.row0, p.row_bytes, &bar);
    }
    if (fa) bulk_load(smem + p.off_fa, d.fa + T.win_begin, 16u * (uint32_t)w, &bar);
  }
  if constexpr (DIM == 3) {
    for (int a = threadIdx.x; a < w; a += kT) {
      const double2 *q = reinterpret_cast<const double2 *>(d.u) + 2 * (T.win_begin + a);
      s_u[a] = q[0];
      s_z[a] = q[1].x;
    }
  }
  Bond64<DIM> B;
  B.th = d.theta + T.win_begin;
  B.fa = d.fa + T.win_begin;
  if constexpr (kState) {
    if (stage & ST_TH) {
      double *s_th = reinterpret_cast<double *>(smem + p.off_th);
      for (int a = threadIdx.x; a < w; a += kT) s_th[a] = B.th[a];
      B.th = s_th;
    }
    if (stage & ST_FA) B.fa = reinterpret_cast<const double2 *>(smem + p.off_fa);
  }
  // the particle's constants, while the copies land
  B.gauss = d.inf.type == PDGPU_INF_GAUSSIAN;
  B.p0 = d.inf.p0, B.p1 = d.inf.type == PDGPU_INF_CONST ? 0.0 : d.inf.p1;
  B.inv_p1 = d.inf_inv_p1;
  B.horizon = P.horizon, B.inv_hor = P.inv_horizon, B.h = P.h, B.inv_h = P.inv_h;
  B.up = P.check_up, B.low = P.check_low;
  B.m0 = P.mat[0], B.m1 = P.mat[1], B.m2 = P.mat[2], B.m3 = P.mat[3], B.m4 = P.mat[4];
  B.irrev = P.mat[5] != 0.0;
  B.inv_m3 = P.inv_mat3;
  B.kn = P.kn, B.rc = P.rc;
  __syncthreads();
  const bool landed = bar_wait(&bar, 0);
  if (__syncthreads_or(!landed)) {
    // the copies did not land: record it, give them one more bounded wait so
    // that none is left writing into this CTA's shared memory, and stop
    if (threadIdx.x == 0 && atomicCAS(&d.ctrl->error, 0, DEV_ERR_STAGE_TIMEOUT) == 0)
      d.ctrl->error_info = blockIdx.x;
    if (!landed) bar_wait(&bar, 0);
    return;
  }

  B.V = Win<DIM>{reinterpret_cast<const double2 *>(smem + p.off_x), s_u, s_z,
                 reinterpret_cast<const double *>(smem + p.off_vol) + (T.win_begin - p.vol0)};
  const int lpn = LPN ? LPN : lanes, lane = threadIdx.x & (lpn - 1);
  const int64_t kb = T.bond_begin;
  // bond indices are relative to the tile's first bond; the bitmap's to the
  // word that holds it
  const int64_t word0 = kStaged ? p.word0 : kb >> 5;
  const uint32_t *bits = kStaged ? reinterpret_cast<const uint32_t *>(smem + p.off_bits) : d.bond_bits + word0;
  const int64_t *rows = kStaged ? reinterpret_cast<const int64_t *>(smem + p.off_row) - p.row0 : d.pd_row;
  const int bit_off = (int)(kb - 32 * word0);
  const int shift = (kStaged ? std::is_same<COL, uint16_t>::value : d.use16 != 0) ? (int)(P.start - T.win_begin) : (int)(-T.win_begin);
  auto neighbour = [&](int k) -> int {
    if constexpr (kStaged) return (int)reinterpret_cast<const COL *>(smem)[k + (int)(kb - p.col0)] + shift;
    else return (d.use16 ? (int)d.pd_col16[kb + k] : d.pd_col[kb + k]) + shift;
  };
  auto break_bond = [&](int k) {
    const int64_t kg = kb + k;
    atomicOr(d.bond_bits + (kg >> 5), 1u << (kg & 31));
  };

  // where bonds can break at all, none of a node does while its largest S^2 r
  // (RNP) or |S| is at most break_z
  const bool may_break = LAW == LAW_RNP ? B.irrev : (LAW == LAW_PMB || PRE);
  const double break_z = LAW == LAW_RNP ? P.break_q : (LAW == LAW_PMB ? B.m1 : B.m2);
  // a warp's 32 / lpn nodes go through the loop together; past the tile's end
  // a group has an empty row
  for (int64_t wb = T.node_begin + threadIdx.x / 32 * (32 / lpn); wb < T.node_end; wb += kT / lpn) {
    const int64_t i_raw = wb + (threadIdx.x & 31) / lpn;
    const bool in_tile = i_raw < T.node_end;
    const int64_t i = in_tile ? i_raw : T.node_end - 1;
    const int li = (int)(i - T.win_begin);
    Node64 I{};
    double vi;
    B.V.node(li, I.x, I.u, vi);
    const int k0 = (int)(rows[i] - kb), k1 = in_tile ? (int)(rows[i + 1] - kb) : k0;
    if constexpr (kState) {
      I.th = B.th[li];
      const double2 q = B.fa[li];
      I.f = q.x;
      I.a = q.y;
    }
    Sum64 s{};
    bool test = any_broken<LPN>(bits, k0 + bit_off, k1 + bit_off, lpn);
    if (!test) {
#pragma unroll 1
      for (int k = k0 + lane; k < k1; k += lpn) bond64<DIM, LAW, PRE, false, kStaged>(B, I, neighbour(k), false, s);
    }
    s.zmax = gmax64<LPN>(s.zmax, lpn);
    test |= may_break && !(s.zmax <= break_z);
    // a stretch that overflowed leaves its lane's force not a number
    if constexpr (!PRE) {
#pragma unroll
      for (int q = 0; q < DIM; q++) test |= not_finite(s.f[q]);
    }
    if (__any_sync(kFullWarp, test)) {
      if (test) {
        s = Sum64{};
#pragma unroll 1
        for (int k = k0 + lane; k < k1; k += lpn) {
          const int b = k + bit_off;
          const bool broken = (bits[b >> 5] >> (b & 31)) & 1u;
          if (bond64<DIM, LAW, PRE, true, kStaged>(B, I, neighbour(k), broken, s)) break_bond(k);
        }
      }
      __syncwarp();
      s.zmax = gmax64<LPN>(s.zmax, lpn);
    }
    if constexpr (PRE) {
      s.theta = gsum<LPN>(s.theta, lpn);
      if (lane == 0 && in_tile) d.theta[i] = 3.0 * s.theta / d.mx[i];
    } else {
#pragma unroll
      for (int q = 0; q < DIM; q++) s.f[q] = gsum<LPN>(s.f[q], lpn);
      if (lane == 0 && in_tile) {
        reinterpret_cast<double2 *>(d.f)[DIM == 2 ? i : 2 * i] = make_double2(s.f[0], s.f[1]);
        if constexpr (DIM == 3) d.f[4 * i + 2] = s.f[2];
        // |S| over the critical stretch (PD elastic: none, DBL_MAX)
        const double z = LAW == LAW_RNP ? sqrt(s.zmax) / B.m2
                                        : s.zmax / (LAW == LAW_ELASTIC ? DBL_MAX : (LAW == LAW_PMB ? B.m1 : B.m2));
        d.Z[i] = (float)z;
      }
    }
  }
}

// per node of a state-based particle: {3K/m_x - a/3, a} with a = 15G/m_x (the
// factors of its own and its neighbours' terms, material.h:1440-1475); in 3-D
// the volume goes into the unused fourth lane of the reference position, so
// that the window arrives by one bulk copy
__global__ void k_fp64_setup(const __grid_constant__ DevData d) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (d.dim == 3) d.xref[4 * i + 3] = d.vol[i];
  const DevParticle &P = d.particles[d.ptid[i]];
  if (!d.fa || P.material != PDGPU_MAT_PDSTATE) return;
  const double m = d.mx[i];
  const double a = 15. * P.mat[1] / m;
  d.fa[i] = make_double2((3. * P.mat[0] / m) - a / 3., a);
}

// any reference distance of the lists outside root_in_range's range? (a warp
// per node: its list is contiguous)
__global__ void k_fp64_range(const __grid_constant__ DevData d, int32_t *outside) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= d.n_nodes) return;
  const int st = d.dim == 2 ? 2 : 4;
  const int64_t e = d.pd_row[i + 1];
  bool out = false;
  for (int64_t k = d.pd_row[i] + (threadIdx.x & 31); k < e; k += 32) {
    double r2 = 0.0;
    for (int q = 0; q < d.dim; q++) {
      const double dx = d.xref[st * (int64_t)d.pd_col[k] + q] - d.xref[st * i + q];
      r2 += dx * dx;
    }
    out |= !(r2 > 0x1p-900 && r2 < 0x1p+890);
  }
  if (out) *outside = 1;
}

template <int DIM, int LPN, int LAW, bool PRE, typename COL>
void launch_one(const DevData &d, const BondTile *t, int n, int lanes, int stage, size_t smem, cudaStream_t s) {
  // behind the pre-pass (see launch_one of the FP32 form for the others)
  if constexpr (LAW == LAW_STATE && !PRE) launch_dependent(k_bonds_fp64<DIM, LPN, LAW, PRE, COL>, n, kThreads64<DIM>, smem, s, d, t, stage, lanes);
  else k_bonds_fp64<DIM, LPN, LAW, PRE, COL><<<n, kThreads64<DIM>, smem, s>>>(d, t, stage, lanes);
}

template <int DIM, int LAW, bool PRE>
void launch_lanes(const DevData &d, const BondTile *t, int n, int lanes, int stage, size_t smem, cudaStream_t s) {
  if (!(stage & ST_BONDS)) launch_one<DIM, 0, LAW, PRE, void>(d, t, n, lanes, stage, smem, s);
  else if (!d.use16) launch_one<DIM, 0, LAW, PRE, int32_t>(d, t, n, lanes, stage, smem, s);
  else if (lanes == 4) launch_one<DIM, 4, LAW, PRE, uint16_t>(d, t, n, lanes, stage, smem, s);
  else if (lanes == 8) launch_one<DIM, 8, LAW, PRE, uint16_t>(d, t, n, lanes, stage, smem, s);
  else if (lanes == 16) launch_one<DIM, 16, LAW, PRE, uint16_t>(d, t, n, lanes, stage, smem, s);
  else launch_one<DIM, 32, LAW, PRE, uint16_t>(d, t, n, lanes, stage, smem, s);
}

template <int DIM>
void launch_laws(const DevData &d, const BondTile *t, const int *law_begin, int lanes, int stage, size_t smem,
                 cudaStream_t s) {
  for (int law = 0; law < 4; law++) {
    const BondTile *b = t + law_begin[law];
    const int n = law_begin[law + 1] - law_begin[law];
    if (n <= 0) continue;
    switch (law) {
      case PDGPU_MAT_RNP: launch_lanes<DIM, LAW_RNP, false>(d, b, n, lanes, stage, smem, s); break;
      case PDGPU_MAT_PMB: launch_lanes<DIM, LAW_PMB, false>(d, b, n, lanes, stage, smem, s); break;
      case PDGPU_MAT_PDELASTIC: launch_lanes<DIM, LAW_ELASTIC, false>(d, b, n, lanes, stage, smem, s); break;
      default: launch_lanes<DIM, LAW_STATE, false>(d, b, n, lanes, stage, smem, s); break;
    }
  }
}

template <int DIM, int LAW, bool PRE>
bool limit_law(size_t bytes) {
  const void *fs[] = {
      (const void *)k_bonds_fp64<DIM, 4, LAW, PRE, uint16_t>,  (const void *)k_bonds_fp64<DIM, 8, LAW, PRE, uint16_t>,
      (const void *)k_bonds_fp64<DIM, 16, LAW, PRE, uint16_t>, (const void *)k_bonds_fp64<DIM, 32, LAW, PRE, uint16_t>,
      (const void *)k_bonds_fp64<DIM, 0, LAW, PRE, int32_t>,   (const void *)k_bonds_fp64<DIM, 0, LAW, PRE, void>};
  for (auto f : fs)
    if (!allow_smem(f, bytes)) return false;
  return true;
}

template <int DIM>
int set_limit(size_t bytes) {
  return limit_law<DIM, LAW_RNP, false>(bytes) && limit_law<DIM, LAW_PMB, false>(bytes) &&
                 limit_law<DIM, LAW_ELASTIC, false>(bytes) && limit_law<DIM, LAW_STATE, false>(bytes) &&
                 limit_law<DIM, LAW_STATE, true>(bytes)
             ? 0
             : -1;
}
}  // namespace

void launch_fp64_setup(const DevData &d, cudaStream_t s) {
  k_fp64_setup<<<(unsigned)((d.n_nodes + 255) / 256), 256, 0, s>>>(d);
}

void launch_fp64_range(const DevData &d, int32_t *outside, cudaStream_t s) {
  k_fp64_range<<<(unsigned)((d.n_nodes + 7) / 8), 256, 0, s>>>(d, outside);
}

void launch_pd_tiled_fp64(const DevData &d, const BondTile *t, const int *law_begin, int lanes, int stage,
                          size_t smem, cudaStream_t s) {
  if (d.dim == 2) launch_laws<2>(d, t, law_begin, lanes, stage, smem, s);
  else launch_laws<3>(d, t, law_begin, lanes, stage, smem, s);
}

void launch_prepass_tiled_fp64(const DevData &d, const BondTile *t, const int *law_begin, int lanes, int stage,
                               size_t smem, cudaStream_t s) {
  const BondTile *b = t + law_begin[PDGPU_MAT_PDSTATE];
  const int n = law_begin[PDGPU_MAT_PDSTATE + 1] - law_begin[PDGPU_MAT_PDSTATE];
  if (n <= 0) return;
  if (d.dim == 2) launch_lanes<2, LAW_STATE, true>(d, b, n, lanes, stage, smem, s);
  else launch_lanes<3, LAW_STATE, true>(d, b, n, lanes, stage, smem, s);
}

size_t tile_smem_fp64(int dim, bool state, int stage, bool col16, const BondTile &t) {
  return plan64(dim, state, stage, col16 ? 2 : 4, t).total;
}

int set_tile_smem_limit_fp64(int dim, size_t bytes) { return dim == 2 ? set_limit<2>(bytes) : set_limit<3>(bytes); }

}  // namespace pdgpu
