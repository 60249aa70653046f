// gb_integrate.cu - NVE velocity Verlet, SHAKE/RATTLE, kinetic stress and the
// Verlet-list displacement check on the device.
//
// Follows:
//   nve_0_vv            source/nve.F90:38-235 (stage 1 :131-174, stage 2 :198-217)
//   constraints_tags    source/constraints.F90:438-586
//   constraints_shake_vv source/constraints.F90:777-1030, apply_shake :1071-1200
//   constraints_rattle  source/constraints.F90:587-775, apply_rattle :1032-1069
//   kinstress           source/kinetics.F90:218-262
//   vnl_check           source/neighbours.F90:123-296
// SHAKE and RATTLE are Jacobi iterations with one global convergence test per
// sweep, exactly as the reference: a cooperative-grid kernel runs the sweeps
// with grid-wide barriers, at most shake_maxit of them, and returns the
// iteration count and a status bit instead of spinning.  k_shake and k_rattle sum
// an atom's corrections in constraint order from a per-atom constraint table and apply
// them listot(i) times, so positions round as the reference's do; k_constrain_cl adds a cluster's
// in registers, and k_constrain_small (clusters of at most 3 constraints, but not in the FP64
// form by instructions) sweeps one double-float scalar per constraint and moves the atoms once.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include <map>
#include <string>

#include "gb_common.cuh"
#include "gb_dfr.cuh"

namespace cg = cooperative_groups;

namespace {

inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

__device__ __forceinline__ double image1(double d, double c, double a) {
  // images, cubic branch (numerics.F90:1527-1532): d - c*Anint(a*d)
  return sub_rn(d, mul_rn(c, round(mul_rn(a, d))));
}

__device__ __forceinline__ long long absbits(double v) { return __double_as_longlong(v) & 0x7fffffffffffffffll; }

// d - c*Anint(a*d), skipping the FP64 work when |d| < quarter (bits) makes the shift zero
__device__ __forceinline__ double image_short(double d, long long quarter_bits, double c, double a) {
  if (absbits(d) < quarter_bits) return d;
  return image1(d, c, a);
}

// Velocity Verlet stages (nve.F90:127-217).  hdw[i] = (tstep/2) / weight(i), formed once
// with the same correctly rounded division the reference performs each step, and 0 for
// an atom with weight <= 1e-6 (which the stages skip): the stages then read one array
// instead of dividing on the FP64 unit.
__global__ void k_vv1(int n, const double* __restrict__ hdw, double tstep, const double* __restrict__ fx,
                      const double* __restrict__ fy, const double* __restrict__ fz, double* vx, double* vy, double* vz,
                      double* x, double* y, double* z, StopIf stop) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || stop.set()) return;
  const double tmp = hdw[i];
  if (tmp > 0.0) {
    vx[i] = vx[i] + tmp * fx[i];
    vy[i] = vy[i] + tmp * fy[i];
    vz[i] = vz[i] + tmp * fz[i];
    x[i] = x[i] + tstep * vx[i];
    y[i] = y[i] + tstep * vy[i];
    z[i] = z[i] + tstep * vz[i];
  }
}

__global__ void k_vv2(int n, const double* __restrict__ hdw, const double* __restrict__ fx,
                      const double* __restrict__ fy, const double* __restrict__ fz, double* vx, double* vy,
                      double* vz, StopIf stop, unsigned long long* t_ns) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  stamp_time(t_ns);
  if (i >= n || stop.set()) return;
  const double tmp = hdw[i];
  if (tmp > 0.0) {
    vx[i] = vx[i] + tmp * fx[i];
    vy[i] = vy[i] + tmp * fy[i];
    vz[i] = vz[i] + tmp * fz[i];
  }
}

// m v (x) v summed over the atoms (kinetics.F90:218-262), after the second half kick of
// k_vv2 when hdw is given: a grid-stride loop, so each thread reduces its own atoms in
// registers and the FP64 sum over the grid runs once per thread rather than once per atom
// (the FP64 unit bounds it).  Its last block adds up the blocks' sums: one launch where
// the kick, the blocks' sums and their total took three (16 us at 4,096 atoms, now 8).
constexpr int KIN_NT = 256;
__global__ void __launch_bounds__(KIN_NT) k_kinstress(int n, const double* __restrict__ w,
                                                      const int* __restrict__ lfrzn, const double* __restrict__ hdw,
                                                      const double* __restrict__ fx, const double* __restrict__ fy,
                                                      const double* __restrict__ fz, double* __restrict__ vx,
                                                      double* __restrict__ vy, double* __restrict__ vz, double* part,
                                                      GridSum gs, StopIf stop, unsigned long long* t_ns) {
  double a[6] = {0, 0, 0, 0, 0, 0};
  stamp_time(t_ns);
  if (stop.set()) hdw = nullptr;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double m = w[i];
    double u = vx[i], v = vy[i], t = vz[i];
    const bool frozen = lfrzn[i] != 0;
    if (hdw) {
      const double tmp = hdw[i];
      if (tmp > 0.0) {
        u = u + tmp * fx[i]; v = v + tmp * fy[i]; t = t + tmp * fz[i];
        vx[i] = u; vy[i] = v; vz[i] = t;
      }
    }
    if (frozen) continue;
    a[0] += m * u * u; a[1] += m * u * v; a[2] += m * u * t;
    a[3] += m * v * v; a[4] += m * v * t; a[5] += m * t * t;
  }
  block_reduce_store<6>(a, part);
  grid_finish<6>(part, gs);
}

// largest |r - r_checkpoint|^2 with minimum image, over a grid-stride loop, after the first
// half kick and the drift of k_vv1 when hdw is given; the caller takes the square root of
// the maximum (the square root is monotone and correctly rounded, so it equals the largest
// of the per-atom square roots); doubles >= 0 order as their bits
__global__ void k_maxdisp(int n, const double* __restrict__ hdw, double tstep, const double* __restrict__ fx,
                          const double* __restrict__ fy, const double* __restrict__ fz, double* __restrict__ vx,
                          double* __restrict__ vy, double* __restrict__ vz, double* __restrict__ x,
                          double* __restrict__ y, double* __restrict__ z, const double* __restrict__ xb,
                          const double* __restrict__ yb, const double* __restrict__ zb, double c0, double a0,
                          unsigned long long* out, StopIf stop, unsigned long long* t_ns) {
  double r2 = 0.0;
  stamp_time(t_ns);
  if (stop.set()) hdw = nullptr;
  const long long quarter = __double_as_longlong(0.25 * c0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double px = x[i], py = y[i], pz = z[i];
    const double bx = xb[i], by = yb[i], bz = zb[i];
    if (hdw) {
      const double tmp = hdw[i];
      if (tmp > 0.0) {
        const double u = vx[i] + tmp * fx[i], v = vy[i] + tmp * fy[i], t = vz[i] + tmp * fz[i];
        vx[i] = u; vy[i] = v; vz[i] = t;
        px = px + tstep * u; py = py + tstep * v; pz = pz + tstep * t;
        x[i] = px; y[i] = py; z[i] = pz;
      }
    }
    const double dx = image_short(px - bx, quarter, c0, a0), dy = image_short(py - by, quarter, c0, a0),
                 dz = image_short(pz - bz, quarter, c0, a0);
    r2 = fmax(r2, dx * dx + dy * dy + dz * dz);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(r2));
}

__global__ void k_fix_to_fp64(int n, const long long* fixp, double* fx, double* fy, double* fz) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double s = 1.0 / 1099511627776.0;
  fx[i] = (double)fixp[3 * i] * s;
  fy[i] = (double)fixp[3 * i + 1] * s;
  fz[i] = (double)fixp[3 * i + 2] * s;
}

// constraints_tags: bond vectors at the start of the stage (min image)
__global__ void k_con_tags(int nc, const int* ci, const int* cj, const double* x, const double* y, const double* z,
                           double c0, double a0, double* dxx, double* dyy, double* dzz) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nc) return;
  int i = ci[k], j = cj[k];
  dxx[k] = image1(x[i] - x[j], c0, a0);
  dyy[k] = image1(y[i] - y[j], c0, a0);
  dzz[k] = image1(z[i] - z[j], c0, a0);
}

struct ConArgs {
  int nc, natms, maxit;
  const int *ci, *cj, *listot, *astart, *alist, *lfrzn;
  const double* d0;
  double *dxx, *dyy, *dzz, *dxt, *dyt, *dzt, *dt2, *gam;
  double *x, *y, *z, *vx, *vy, *vz;
  const double* w;
  double tstep, tol, c0, a0;
  int* flags;      // maxit+1 ints, zeroed
  GridSum gs;      // of k_constrain_small's stress
  bool tags;       // RATTLE of k_constrain_small: form the bond vectors from the positions (and store them)
  DevScalars* sc;
  double* blk;     // per-block stress partials (6)
  StopIf stop;
};

// constraints_shake_vv: Jacobi sweeps until every |d^2 - d0^2|/2 < tol*d0
__global__ void k_shake(ConArgs A) {
  if (A.stop.set()) return;
  cg::grid_group grid = cg::this_grid();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  const double tstep2 = A.tstep * A.tstep;
  double st[6] = {0, 0, 0, 0, 0, 0};
  int it = 0;
  bool safe = false;
  while (!safe && it < A.maxit) {
    ++it;
    for (int k = tid; k < A.nc; k += nth) {
      int i = A.ci[k], j = A.cj[k];
      double dx = image1(A.x[i] - A.x[j], A.c0, A.a0);
      double dy = image1(A.y[i] - A.y[j], A.c0, A.a0);
      double dz = image1(A.z[i] - A.z[j], A.c0, A.a0);
      A.dxt[k] = dx; A.dyt[k] = dy; A.dzt[k] = dz;
      double d0 = A.d0[k];
      double d2 = dx * dx + dy * dy + dz * dz - d0 * d0;
      A.dt2[k] = d2;
      if (!(0.5 * fabs(d2) < A.tol * d0)) A.flags[it] = 1;
    }
    grid.sync();
    safe = (A.flags[it] == 0);
    if (!safe) {
      for (int k = tid; k < A.nc; k += nth) {
        int i = A.ci[k], j = A.cj[k];
        double amti = tstep2 / A.w[i], amtj = tstep2 / A.w[j];
        if (A.lfrzn[i] != 0) amti = 0.0;
        if (A.lfrzn[j] != 0) amtj = 0.0;
        double gamma = A.dt2[k] / ((amti + amtj) * (A.dxx[k] * A.dxt[k] + A.dyy[k] * A.dyt[k] + A.dzz[k] * A.dzt[k]));
        A.gam[k] = gamma;
        st[0] -= gamma * A.dxx[k] * A.dxx[k]; st[1] -= gamma * A.dxx[k] * A.dyy[k];
        st[2] -= gamma * A.dxx[k] * A.dzz[k]; st[3] -= gamma * A.dyy[k] * A.dyy[k];
        st[4] -= gamma * A.dyy[k] * A.dzz[k]; st[5] -= gamma * A.dzz[k] * A.dzz[k];
      }
      grid.sync();
      for (int i = tid; i < A.natms; i += nth) {
        const int s = A.astart[i], e = A.astart[i + 1];
        if (s == e || A.lfrzn[i] != 0) continue;
        double xt = 0.0, yt = 0.0, zt = 0.0;
        const double amt = tstep2 / A.w[i];
        for (int t = s; t < e; ++t) {
          int code = A.alist[t];
          int k = code >> 1;
          double g = A.gam[k];
          double f = (code & 1) ? 0.5 * g * amt : -0.5 * g * amt;
          xt += A.dxx[k] * f; yt += A.dyy[k] * f; zt += A.dzz[k] * f;
        }
        const double dli = 1.0 / (double)A.listot[i];
        double px = A.x[i], py = A.y[i], pz = A.z[i];
        for (int r = 0; r < A.listot[i]; ++r) { px += xt * dli; py += yt * dli; pz += zt * dli; }
        A.x[i] = px; A.y[i] = py; A.z[i] = pz;
      }
      grid.sync();
    }
  }
  if (tid == 0) {
    A.sc->shake_iters = it;
    if (!safe) A.sc->status |= ST_SHAKE_FAIL;
  }
  block_reduce_store<6>(st, A.blk);
}

// constraints_rattle: normalise the bond vectors, then Jacobi sweeps on v
__global__ void k_rattle(ConArgs A) {
  if (A.stop.set()) return;
  cg::grid_group grid = cg::this_grid();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  for (int k = tid; k < A.nc; k += nth) {
    double dis = 1.0 / sqrt(A.dxx[k] * A.dxx[k] + A.dyy[k] * A.dyy[k] + A.dzz[k] * A.dzz[k]);
    A.dxx[k] *= dis; A.dyy[k] *= dis; A.dzz[k] *= dis;
  }
  grid.sync();
  int it = 0;
  bool safe = false;
  while (!safe && it < A.maxit) {
    ++it;
    for (int k = tid; k < A.nc; k += nth) {
      int i = A.ci[k], j = A.cj[k];
      double amti = A.tstep / A.w[i], amtj = A.tstep / A.w[j];
      if (A.lfrzn[i] != 0) amti = 0.0;
      if (A.lfrzn[j] != 0) amtj = 0.0;
      double gamma = A.dxx[k] * (A.vx[i] - A.vx[j]) + A.dyy[k] * (A.vy[i] - A.vy[j]) + A.dzz[k] * (A.vz[i] - A.vz[j]);
      if (!(0.5 * A.tstep * fabs(gamma) < A.tol)) A.flags[it] = 1;
      A.gam[k] = gamma / (amti + amtj);
    }
    grid.sync();
    safe = (A.flags[it] == 0);
    if (!safe) {
      for (int i = tid; i < A.natms; i += nth) {
        const int s = A.astart[i], e = A.astart[i + 1];
        if (s == e || A.lfrzn[i] != 0) continue;
        double xt = 0.0, yt = 0.0, zt = 0.0;
        const double amt = A.tstep / A.w[i];
        for (int t = s; t < e; ++t) {
          int code = A.alist[t];
          int k = code >> 1;
          double g = A.gam[k];
          double f = (code & 1) ? g * amt : -g * amt;
          xt += A.dxx[k] * f; yt += A.dyy[k] * f; zt += A.dzz[k] * f;
        }
        const double dli = 1.0 / (double)A.listot[i];
        double px = A.vx[i], py = A.vy[i], pz = A.vz[i];
        for (int r = 0; r < A.listot[i]; ++r) { px += xt * dli; py += yt * dli; pz += zt * dli; }
        A.vx[i] = px; A.vy[i] = py; A.vz[i] = pz;
      }
      grid.sync();
    }
  }
  if (tid == 0) {
    A.sc->rattle_iters = it;
    if (!safe) A.sc->status |= ST_RATTLE_FAIL;
  }
}

// ------------------------------------------------- cluster-local SHAKE/RATTLE
// When every connected group of constraints (a "cluster": a rigid water, a
// small molecule) has at most CL_MAXA atoms and CL_MAXC constraints, the
// Jacobi sweeps of different clusters are independent: sweep `it` of a cluster
// reads only that cluster's atoms.  One thread then owns a cluster and runs
// its sweeps in registers; the only global quantity is the convergence test,
// "every constraint of every cluster passes at sweep it".  Sweeps run in
// chunks of CL_CHUNK: each cluster records the sweeps at which it fails in a
// per-sweep flag word and applies every update of the chunk, saving the state
// after each sweep in a per-cluster ring; one grid barrier per chunk then gives
// the first sweep N at which nobody failed, and each cluster keeps the state
// saved after sweep N-1.  Every update uses the per-sweep kernel's arithmetic,
// so the result and the iteration count are those of the reference's global
// sweeps (constraints.F90:898-969 and 1032-1071).
//
// FP64 instructions are expensive on this part, so tests that need no
// arithmetic are done on the IEEE bit patterns: the minimum image of a bond
// shorter than a quarter cell is the bond itself (round(d/L) = 0 exactly), and
// the tolerance tests 0.5|x| < t are |x| < 2t, an integer compare of the
// magnitudes' bits.
constexpr int CL_MAXA = 4, CL_MAXC = 6, CL_CHUNK = 8;
constexpr int CL_RING = CL_CHUNK + 1;       // state at chunk start + after each sweep
constexpr int CL_SLOT = 3 * CL_MAXA + CL_MAXC;  // doubles per ring slot: state, then sweep gammas

struct ClusterTab {
  int atom[CL_MAXA];   // global atom ids, -1 padding
  int con[CL_MAXC];    // global constraint ids in ascending order, -1 padding
  int pair[CL_MAXC];   // local ends: li | lj << 4
  int alist[CL_MAXA];  // per local atom: count | entries (local constraint << 1 | j end) in 4-bit fields from bit 4
  int meta;            // na | nc << 4
};

__device__ __forceinline__ void warp_flag(bool fail, int* flag) {
  const unsigned m = __activemask();
  const unsigned b = __ballot_sync(m, fail);
  if (b && (threadIdx.x & 31) == __ffs(m) - 1) atomicOr(flag, 1);
}

// register-array reads with a runtime index, as selects (no local-memory copy)
template <int N>
__device__ __forceinline__ double sel(const double (&a)[N], int i) {
  double r = a[0];
#pragma unroll
  for (int k = 1; k < N; ++k) r = (i == k) ? a[k] : r;
  return r;
}

// per-cluster constants and state (positions for SHAKE, velocities for RATTLE)
template <int MA, int MC>
struct ClData {
  int na, nc;
  double x[MA], y[MA], z[MA];
  double bx[MC], by[MC], bz[MC];
  double d0sq[MC];          // SHAKE: d0^2
  long long tolb[MC];       // bits of the tolerance bound on |d2| (SHAKE) or |gamma| (RATTLE)
  double msum[MC];          // amt_i + amt_j
  double hm[MA];            // per-atom update factor: 0.5 amt (SHAKE) or amt (RATTLE)
  double dli[MA];           // 1 / listot
  bool active[MA];          // has constraints and is not frozen
};

template <int MA, int MC>
__device__ __forceinline__ void cl_load(const ConArgs& A, const ClusterTab& T, bool rattle, ClData<MA, MC>& D) {
  D.na = T.meta & 15;
  D.nc = (T.meta >> 4) & 15;
  const double amt_num = rattle ? A.tstep : A.tstep * A.tstep;
  double amt[MA];
#pragma unroll
  for (int a = 0; a < MA; ++a) {
    D.x[a] = D.y[a] = D.z[a] = 0.0;
    amt[a] = 0.0; D.hm[a] = 0.0; D.dli[a] = 1.0; D.active[a] = false;
    if (a < D.na) {
      const int i = T.atom[a];
      if (rattle) { D.x[a] = A.vx[i]; D.y[a] = A.vy[i]; D.z[a] = A.vz[i]; }
      else { D.x[a] = A.x[i]; D.y[a] = A.y[i]; D.z[a] = A.z[i]; }
      const bool frz = A.lfrzn[i] != 0;
      amt[a] = frz ? 0.0 : amt_num / A.w[i];
      const int cnt = T.alist[a] & 15;
      D.active[a] = !frz && cnt > 0;
      D.hm[a] = rattle ? amt[a] : 0.5 * amt[a];
      D.dli[a] = 1.0 / (double)(cnt > 0 ? cnt : 1);
    }
  }
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    D.bx[c] = D.by[c] = D.bz[c] = 0.0; D.d0sq[c] = 0.0; D.tolb[c] = 0; D.msum[c] = 1.0;
    if (c < D.nc) {
      const int k = T.con[c];
      const int li = T.pair[c] & 15, lj = T.pair[c] >> 4;
      double ux = A.dxx[k], uy = A.dyy[k], uz = A.dzz[k];
      if (rattle) {
        const double dis = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
        ux *= dis; uy *= dis; uz *= dis;
        // 0.5 tstep |gamma| < tol  <=>  |gamma| < (2 tol) / tstep, evaluated as the kernel does: 0.5*tstep*|g| < tol
        D.tolb[c] = 0;  // unused: RATTLE keeps the FP64 comparison (tstep scaling is not exact)
      } else {
        const double d0 = A.d0[k];
        D.d0sq[c] = d0 * d0;
        D.tolb[c] = __double_as_longlong(2.0 * (A.tol * d0));  // 0.5|d2| < tol d0  <=>  |d2| < 2 (tol d0)
      }
      D.bx[c] = ux; D.by[c] = uy; D.bz[c] = uz;
      D.msum[c] = sel(amt, li) + sel(amt, lj);
    }
  }
}

// one sweep: tests (returns true when a constraint fails), gammas, update of the state
template <int MA, int MC>
__device__ __forceinline__ bool cl_sweep(const ConArgs& A, const ClusterTab& T, bool rattle, long long quarter,
                                         ClData<MA, MC>& D, double (&gam)[MC]) {
  bool fail = false;
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    gam[c] = 0.0;
    if (c < D.nc) {
      const int li = T.pair[c] & 15, lj = T.pair[c] >> 4;
      if (rattle) {
        const double gamma = D.bx[c] * (sel(D.x, li) - sel(D.x, lj)) + D.by[c] * (sel(D.y, li) - sel(D.y, lj)) +
                             D.bz[c] * (sel(D.z, li) - sel(D.z, lj));
        if (!(0.5 * A.tstep * fabs(gamma) < A.tol)) fail = true;
        gam[c] = gamma / D.msum[c];
      } else {
        const double dx = image_short(sel(D.x, li) - sel(D.x, lj), quarter, A.c0, A.a0);
        const double dy = image_short(sel(D.y, li) - sel(D.y, lj), quarter, A.c0, A.a0);
        const double dz = image_short(sel(D.z, li) - sel(D.z, lj), quarter, A.c0, A.a0);
        const double d2 = dx * dx + dy * dy + dz * dz - D.d0sq[c];
        if (!(absbits(d2) < D.tolb[c])) fail = true;
        gam[c] = d2 / (D.msum[c] * (D.bx[c] * dx + D.by[c] * dy + D.bz[c] * dz));
      }
    }
  }
#pragma unroll
  for (int a = 0; a < MA; ++a) {
    if (!D.active[a]) continue;
    const int al = T.alist[a], cnt = al & 15;
    double xt = 0.0, yt = 0.0, zt = 0.0;
#pragma unroll
    for (int e = 0; e < MC; ++e) {
      if (e < cnt) {
        const int code = (al >> (4 + 4 * e)) & 15, c = code >> 1;
        const double gh = sel(gam, c) * D.hm[a];
        const double f = (code & 1) ? gh : -gh;
        xt += sel(D.bx, c) * f; yt += sel(D.by, c) * f; zt += sel(D.bz, c) * f;
      }
    }
    double px = D.x[a], py = D.y[a], pz = D.z[a];
    for (int r = 0; r < cnt; ++r) { px += xt * D.dli[a]; py += yt * D.dli[a]; pz += zt * D.dli[a]; }
    D.x[a] = px; D.y[a] = py; D.z[a] = pz;
  }
  return fail;
}

template <int MA, int MC>
__device__ __forceinline__ void ring_put(double* slot, const ClData<MA, MC>& D, const double (&gam)[MC]) {
#pragma unroll
  for (int a = 0; a < MA; ++a) { slot[3 * a] = D.x[a]; slot[3 * a + 1] = D.y[a]; slot[3 * a + 2] = D.z[a]; }
#pragma unroll
  for (int c = 0; c < MC; ++c) slot[3 * CL_MAXA + c] = gam[c];
}

// SHAKE (rattle = false) or RATTLE (rattle = true) over all clusters; gsum
// (MC doubles per cluster) holds the committed gamma sums of SHAKE for
// the constraint stress
template <int MA, int MC>
__global__ void __launch_bounds__(128) k_constrain_cl(ConArgs A, const ClusterTab* __restrict__ tabs, int ncl,
                                                      double* __restrict__ ring, double* __restrict__ gsum,
                                                      int rattle_i) {
  if (A.stop.set()) return;
  cg::grid_group grid = cg::this_grid();
  const bool rattle = rattle_i != 0;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  const long long quarter = __double_as_longlong(0.25 * A.c0);
  int it0 = 0, nfinal = -1;
  for (;;) {
    for (int cl = tid; cl < ncl; cl += nth) {
      const ClusterTab T = tabs[cl];
      ClData<MA, MC> D;
      cl_load(A, T, rattle, D);
      double* rg = ring + (size_t)cl * CL_RING * CL_SLOT;
      double gam[MC];
#pragma unroll
      for (int c = 0; c < MC; ++c) gam[c] = 0.0;
      ring_put(rg, D, gam);
      for (int s_ = 1; s_ <= CL_CHUNK; ++s_) {
        if (it0 + s_ > A.maxit) break;
        const bool fail = cl_sweep(A, T, rattle, quarter, D, gam);
        warp_flag(fail, &A.flags[it0 + s_]);
        ring_put(rg + s_ * CL_SLOT, D, gam);
      }
    }
    grid.sync();
    for (int s_ = 1; s_ <= CL_CHUNK && it0 + s_ <= A.maxit; ++s_)
      if (A.flags[it0 + s_] == 0) { nfinal = it0 + s_; break; }
    // committed sweeps of this chunk: all of them, or those before nfinal
    const int last = nfinal > 0 ? nfinal - 1 - it0 : (A.maxit - it0 < CL_CHUNK ? A.maxit - it0 : CL_CHUNK);
    for (int cl = tid; cl < ncl; cl += nth) {
      const ClusterTab T = tabs[cl];
      const int na = T.meta & 15, nc = (T.meta >> 4) & 15;
      const double* rg = ring + (size_t)cl * CL_RING * CL_SLOT;
      const double* fin = rg + last * CL_SLOT;
#pragma unroll
      for (int a = 0; a < MA; ++a) {
        if (a < na) {
          const int i = T.atom[a];
          if (rattle) { A.vx[i] = fin[3 * a]; A.vy[i] = fin[3 * a + 1]; A.vz[i] = fin[3 * a + 2]; }
          else { A.x[i] = fin[3 * a]; A.y[i] = fin[3 * a + 1]; A.z[i] = fin[3 * a + 2]; }
        }
      }
      if (!rattle) {
        for (int s_ = 1; s_ <= last; ++s_)
#pragma unroll
          for (int c = 0; c < MC; ++c)
            if (c < nc) gsum[(size_t)cl * CL_MAXC + c] += rg[s_ * CL_SLOT + 3 * CL_MAXA + c];
      }
    }
    if (nfinal > 0) break;
    it0 += CL_CHUNK;
    if (it0 >= A.maxit) break;
    // no barrier needed here: a cluster is always handled by the same thread
  }
  if (tid == 0) {
    if (rattle) {
      A.sc->rattle_iters = nfinal > 0 ? nfinal : A.maxit;
      if (nfinal < 0) A.sc->status |= ST_RATTLE_FAIL;
    } else {
      A.sc->shake_iters = nfinal > 0 ? nfinal : A.maxit;
      if (nfinal < 0) A.sc->status |= ST_SHAKE_FAIL;
    }
  }
  if (!rattle) {
    // constraint stress: every committed update adds -gamma b b^T, b fixed during SHAKE
    double st[6] = {0, 0, 0, 0, 0, 0};
    for (int cl = tid; cl < ncl; cl += nth) {
      const ClusterTab T = tabs[cl];
      const int nc = (T.meta >> 4) & 15;
#pragma unroll
      for (int c = 0; c < MC; ++c) {
        if (c >= nc) continue;
        const int k = T.con[c];
        const double g = gsum[(size_t)cl * CL_MAXC + c];
        const double bx = A.dxx[k], by = A.dyy[k], bz = A.dzz[k];
        st[0] -= g * bx * bx; st[1] -= g * bx * by; st[2] -= g * bx * bz;
        st[3] -= g * by * by; st[4] -= g * by * bz; st[5] -= g * bz * bz;
      }
    }
    block_reduce_store<6>(st, A.blk);
  }
}

// ------------------------------------ clusters of at most 3 constraints, in scalars
// The Jacobi sweeps of a small cluster only ever move its atoms along the cluster's own
// (fixed) bond vectors b_i, so the state of a cluster is one scalar per constraint, t_i
// = M_i/2 * sum(gamma_i) (SHAKE) or sum(b_i . dv) (RATTLE), M_i = amt_i + amt_j:
//   bond     d_c = u_c + sum_i K_ci b_i t_i,    K_ci = (s_ai amt_a - s_bi amt_b) / M_i, (a, b) the ends of c
//   atom     x_a = x_a(0) + sum_i W_ai b_i t_i,  W_ai = s_ai amt_a / M_i, s_ai = -1 / +1 / 0 (i end, j end, neither)
//   SHAKE    t_c += q_c / (2 p_c), q_c = |d_c|^2 - d0_c^2 a quadratic in t, p_c = b_c . d_c linear in t
//   RATTLE   t_c += g_c, g_c = b_c . (v_a - v_b) linear in t
// (constraints.F90:898-969 and 687-742 written in these variables; the sweeps, their tests
// and their number are the same).  The polynomials' constants are formed once per cluster
// and a sweep is double-float arithmetic on the FP32 pipes: |q| is a difference from
// |u|^2 - d0^2 (FP64) by terms of the size of the correction, so it is as exact as the FP64
// form's, whose coordinates carry the rounding of the box's size (7e-15 A at 50 A).
// An FP64 instruction takes 16 issue slots of an SM sub-partition here: the FP64 form of
// the sweep (~110 FP64 instructions with 3 divisions, k_constrain_cl) took 0.83 ms a call
// for 32,768 waters (~67 sweeps) and 0.52 ms for 2,197.
// A lane holds one constraint (3 lanes a cluster, 10 clusters a warp) and exchanges its
// scalar by shuffles: a sweep is a chain of dependent operations, which one lane per
// cluster ran at two warps a scheduler (0.133 and 0.090 ms).  q_c is evaluated as c0 +
// sum_i t_i (l_i + sum_j q_ij t_j); the inner sums run over an added constant
// (off_add_prod; it grows with the cluster's bonds where they start far from their lengths:
// sums that reach it lose their last bits, and SHAKE of molecules three times too large did
// not converge), and the scalars of a chunk's sweeps are kept in shared memory, so that none is
// repeated.  It takes 0.090 ms (SHAKE) and 0.053 ms (RATTLE, which forms the bond
// vectors too) for 32,768 waters, 0.047 and 0.027 ms for 2,197: the operations of a sweep in
// order, the FP64 set-up and epilogue, and five grid barriers.
// Sweeps run in chunks of CS_CHUNK between grid barriers (20 steps of 2,197 molecules:
// 8.6 ms with chunks of 8, 8.3 with 16 and with 31, which doubles the shared memory).
constexpr int CS_CHUNK = 16, CS_MAXC = 3, CS_PERWARP = 10;
// One block per SM, of as many warps as the clusters need, up to the most whose registers (80 a
// thread in SHAKE) it holds with the same number for each scheduler: 24, or 240 clusters a SM.  More
// clusters than that keep their polynomials in memory between chunks and repeat the last
// one (152 SMs, SHAKE and RATTLE: 35,937 clusters 0.094 and 0.061 ms, 39,304 0.172 and 0.101).
constexpr int CS_THREADS = 768;
constexpr int CS_POLY = 15;      // float2 of the polynomials of a lane

struct ClKind {        // clusters with equal masses, lengths and topology share one
  int na, nc;
  int li[CS_MAXC], lj[CS_MAXC];         // local ends of the constraints
  float2 K[CS_MAXC][CS_MAXC];           // double-float
  float2 tol_s[CS_MAXC], tol_r;         // bounds on |q| (2 tol d0) and |g| (2 tol / tstep)
  float off;                            // 8 max(d0^2) rounded up to a power of two
  double W[CL_MAXA][CS_MAXC];
  double d0sq[CS_MAXC];
  double two_m[CS_MAXC];                // gamma sum = two_m * t (SHAKE)
  double wh[CL_MAXA];                   // weight / hstep, 0: frozen
};

__device__ __forceinline__ df df_of(float2 a) { return df_make(a.x, a.y); }

__device__ __forceinline__ df df_dot(const df (&a)[3], const df (&b)[3]) {
  dacc s = {0.f, 0.f};
  dacc_add_prod(s, a[0], b[0]);
  dacc_add_prod(s, a[1], b[1]);
  dacc_add_prod(s, a[2], b[2]);
  return quick_two_sum(s.s, s.c);
}

// |a| < b; false for NaN
__device__ __forceinline__ bool df_abs_less(df a, float2 b) {
  const bool neg = a.hi < 0.f;
  const float h = neg ? -a.hi : a.hi, l = neg ? -a.lo : a.lo;
  return h < b.x || (h == b.x && l < b.y);
}

__device__ __forceinline__ df df_shfl(df a, int lane) {
  return df_make(__shfl_sync(0xffffffffu, a.hi, lane), __shfl_sync(0xffffffffu, a.lo, lane));
}

// The polynomials of a lane's constraint; index r is the constraint of the cluster r places
// after its own, cyclically; q in the order 00, 01, 02, 11, 12, 22.
struct ClPoly {
  float off;          // a power of two, at least 8/3 of the |l| (SHAKE)
  df c0, l[CS_MAXC];  // l over the constant off
  df q[6];
  df p0, p[CS_MAXC];
};

// c: constraint of the lane, on: it has one; n1, n2: lanes of the next two constraints
template <bool RATTLE>
__device__ __forceinline__ void cs_setup(const ConArgs& A, const ClusterTab& T, const ClKind& D, int c, bool on, int n1,
                                         int n2, long long quarter, ClPoly& P) {
  df b[CS_MAXC][3], u[3], B[6], K[CS_MAXC];
  P.c0 = df_make(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 3; ++k) b[0][k] = u[k] = P.c0;
  if (on) {
    const int k = T.con[c], i = T.atom[D.li[c]], j = T.atom[D.lj[c]];
    double bx, by, bz;
    if (RATTLE && A.tags) {
      bx = image_short(A.x[i] - A.x[j], quarter, A.c0, A.a0);
      by = image_short(A.y[i] - A.y[j], quarter, A.c0, A.a0);
      bz = image_short(A.z[i] - A.z[j], quarter, A.c0, A.a0);
      A.dxx[k] = bx; A.dyy[k] = by; A.dzz[k] = bz;
    } else {
      bx = A.dxx[k]; by = A.dyy[k]; bz = A.dzz[k];
    }
    if (RATTLE) {
      const double b2 = bx * bx + by * by + bz * bz;
      double r = rsqrt_seeded(b2);
      r = r * fma(-0.5 * b2 * r, r, 1.5);
      bx *= r; by *= r; bz *= r;
      const double dx = A.vx[i] - A.vx[j], dy = A.vy[i] - A.vy[j], dz = A.vz[i] - A.vz[j];
      P.c0 = dbl_split(bx * dx + by * dy + bz * dz);
    } else {
      const double dx = image_short(A.x[i] - A.x[j], quarter, A.c0, A.a0);
      const double dy = image_short(A.y[i] - A.y[j], quarter, A.c0, A.a0);
      const double dz = image_short(A.z[i] - A.z[j], quarter, A.c0, A.a0);
      u[0] = dbl_split(dx); u[1] = dbl_split(dy); u[2] = dbl_split(dz);
      P.c0 = dbl_split(dx * dx + dy * dy + dz * dz - D.d0sq[c]);
    }
    b[0][0] = dbl_split(bx); b[0][1] = dbl_split(by); b[0][2] = dbl_split(bz);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b[1][k] = df_shfl(b[0][k], n1);
    b[2][k] = df_shfl(b[0][k], n2);
  }
  const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
  K[0] = df_of(D.K[c][c]); K[1] = df_of(D.K[c][c1]); K[2] = df_of(D.K[c][c2]);
  B[0] = df_dot(b[0], b[0]);
  B[1] = df_dot(b[0], b[1]);
  B[2] = df_shfl(B[1], n2);  // 2 . 0
  B[3] = df_shfl(B[0], n1);
  B[4] = df_shfl(B[1], n1);  // 1 . 2
  B[5] = df_shfl(B[0], n2);
  if (!on) K[0] = K[1] = K[2] = df_make(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < CS_MAXC; ++k) P.p[k] = df_mul(K[k], B[k]);
  if (!RATTLE) {
    float m = 0.f;  // the largest |l|
#pragma unroll
    for (int k = 0; k < CS_MAXC; ++k) {
      P.l[k] = df_mul(K[k], df_dot(u, b[k]));
      m = fmaxf(m, 2.f * fabsf(P.l[k].hi));
    }
    P.off = D.off;
    if (m > 0.375f * P.off) P.off = __uint_as_float(min((__float_as_uint(m) >> 23) + 4u, 254u) << 23);
#pragma unroll
    for (int k = 0; k < CS_MAXC; ++k) {
      const df s = two_sum(P.off, 2.f * P.l[k].hi);
      P.l[k] = df_make(s.hi, s.lo + 2.f * P.l[k].lo);
    }
    P.p0 = on ? df_dot(u, b[0]) : df_make(1.f, 0.f);
    int i = 0;
#pragma unroll
    for (int k = 0; k < CS_MAXC; ++k)
#pragma unroll
      for (int n = k; n < CS_MAXC; ++n, ++i) {
        const df e = df_mul(df_mul(K[k], K[n]), B[i]);
        const float f = n == k ? 1.f : 2.f;
        P.q[i] = df_make(f * e.hi, f * e.lo);
      }
  }
}

// one sweep from the scalars t (own first): true when the constraint fails its test; the new
// scalars in t
template <bool RATTLE>
__device__ __forceinline__ bool cs_sweep(const ClPoly& P, float2 tol, int n1, int n2, df (&t)[CS_MAXC]) {
  dacc a = {P.c0.hi, P.c0.lo};
  df step;
  bool fail;
  if constexpr (RATTLE) {
#pragma unroll
    for (int i = 0; i < CS_MAXC; ++i) dacc_add_prod(a, P.p[i], t[i]);
    step = quick_two_sum(a.s, a.c);
    fail = !df_abs_less(step, tol);
  } else {
    dacc e = {P.p0.hi, P.p0.lo};  // p exceeds its corrections
#pragma unroll
    for (int i = 0; i < CS_MAXC; ++i) off_add_prod(e, P.p[i], t[i]);
    // 1/p: FP32 reciprocal and the first-order remainder (relative error about 2^-46)
    const float r = __frcp_rn(e.s);
    const float h = __fmaf_rn(-e.c, r, __fmaf_rn(-e.s, r, 1.f));
    int m = 0;
#pragma unroll
    for (int i = 0; i < CS_MAXC; ++i) {
      dacc v = {P.l[i].hi, P.l[i].lo};
#pragma unroll
      for (int j = i; j < CS_MAXC; ++j, ++m) off_add_prod(v, P.q[m], t[j]);
      dacc_add_prod(a, df_make(__fsub_rn(v.s, P.off), v.c), t[i]);
    }
    const df q = quick_two_sum(a.s, a.c);
    fail = !df_abs_less(q, tol);
    const df s = df_mul(q, df_make(r, r * h));
    step = df_make(0.5f * s.hi, 0.5f * s.lo);
  }
  t[0] = df_add(t[0], step);
  t[1] = df_shfl(t[0], n1);
  t[2] = df_shfl(t[0], n2);
  return fail;
}

// The polynomials of a lane to and from pbuf (more clusters than resident lanes).
template <bool RATTLE, bool STORE>
__device__ __forceinline__ void cs_poly_io(float2* __restrict__ pbuf, size_t ld, ClPoly& P) {
  auto io = [&](int slot, df& v) {
    if (STORE)
      pbuf[slot * ld] = make_float2(v.hi, v.lo);
    else
      v = df_of(pbuf[slot * ld]);
  };
  io(0, P.c0);
#pragma unroll
  for (int k = 0; k < 3; ++k) io(1 + k, P.p[k]);
  if (RATTLE) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) io(4 + k, P.l[k]);
#pragma unroll
  for (int k = 0; k < 6; ++k) io(7 + k, P.q[k]);
  io(13, P.p0);
  df off = df_make(P.off, 0.f);
  io(14, off);
  P.off = off.hi;
}

// SHAKE with its epilogue (apply_shake: v += dr/dt, f += dr/dt m/(dt/2)) or RATTLE.  pbuf: when
// there are more clusters than resident lanes, the polynomials of a lane and its scalar
// at the start and the end of the chunk ([CS_POLY + 2][3 ncl]; L2 traffic of a few microseconds
// a chunk); such a cluster repeats the last chunk's committed sweeps.
template <bool RATTLE>
__global__ void __launch_bounds__(CS_THREADS) k_constrain_small(ConArgs A, const ClusterTab* __restrict__ tabs,
                                                               const int* __restrict__ kind_of,
                                                               const ClKind* __restrict__ kinds, int ncl,
                                                               float2* __restrict__ pbuf, double rstep, double* fx,
                                                               double* fy, double* fz) {
  extern __shared__ float2 cs_hist[];  // [CS_CHUNK][blockDim.x]: the scalar before each sweep of the chunk
  if (A.stop.set()) return;
  cg::grid_group grid = cg::this_grid();
  const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int wstep = ((gridDim.x * blockDim.x) >> 5) * CS_PERWARP;
  const int sub = lane / 3, c = lane - 3 * sub;
  const int n1 = 3 * sub + (c == 2 ? 0 : c + 1), n2 = 3 * sub + (c == 0 ? 2 : c - 1);
  const long long quarter = __double_as_longlong(0.25 * A.c0);
  const bool multi = ncl > wstep;
  const size_t ld = 3 * (size_t)ncl;
  ClPoly P;
  df t[CS_MAXC];
#pragma unroll
  for (int r = 0; r < CS_MAXC; ++r) t[r] = df_make(0.f, 0.f);
  int it0 = 0, nfinal = -1, last = 0;
  bool done = false;
  for (int ch = 0;; ++ch) {
    unsigned bad = 0;
    const int n = min(CS_CHUNK, A.maxit - it0);
    for (int cl0 = warp * CS_PERWARP; cl0 < ncl; cl0 += wstep) {
      const bool in = lane < 3 * CS_PERWARP && cl0 + sub < ncl;
      const int cl = in ? cl0 + sub : cl0;
      const ClKind& D = kinds[kind_of[cl]];
      const bool on = in && c < D.nc;
      float2* pb = pbuf + (size_t)3 * cl + c;
      if (it0 == 0) {
        cs_setup<RATTLE>(A, tabs[cl], D, c, on, n1, n2, quarter, P);
        if (multi && in) cs_poly_io<RATTLE, true>(pb, ld, P);
        t[0] = t[1] = t[2] = df_make(0.f, 0.f);
      } else if (multi) {
        cs_poly_io<RATTLE, false>(pb, ld, P);
        t[0] = df_of(pb[(CS_POLY + 1) * ld]);
        t[1] = df_shfl(t[0], n1);
        t[2] = df_shfl(t[0], n2);
      }
      if (multi && in) pb[CS_POLY * ld] = make_float2(t[0].hi, t[0].lo);
      const float2 tol = RATTLE ? D.tol_r : D.tol_s[c];
      unsigned b = 0;
      for (int s = 0; s < n; ++s) {
        cs_hist[s * blockDim.x + threadIdx.x] = make_float2(t[0].hi, t[0].lo);
        if (cs_sweep<RATTLE>(P, tol, n1, n2, t)) b |= 1u << s;
      }
      if (on) bad |= b;
      if (multi && in) pb[(CS_POLY + 1) * ld] = make_float2(t[0].hi, t[0].lo);
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (bad && lane == 0) atomicOr(&A.flags[ch], (int)bad);
    grid.sync();
    const unsigned f = ~(unsigned)__ldcg(&A.flags[ch]) & ((1u << n) - 1u);
    last = n;  // committed sweeps of this chunk: all, or those before the first that nobody failed
    if (f) {
      last = __ffs((int)f) - 1;
      nfinal = it0 + last + 1;
      done = true;
    }
    if (done || it0 + n >= A.maxit) break;
    it0 += n;
  }
  if (warp == 0 && lane == 0) {
    (RATTLE ? A.sc->rattle_iters : A.sc->shake_iters) = nfinal > 0 ? nfinal : A.maxit;
    if (nfinal < 0) A.sc->status |= RATTLE ? ST_RATTLE_FAIL : ST_SHAKE_FAIL;
  }
  double st[6] = {0, 0, 0, 0, 0, 0};
  for (int cl0 = warp * CS_PERWARP; cl0 < ncl; cl0 += wstep) {
    const bool in = lane < 3 * CS_PERWARP && cl0 + sub < ncl;
    const int cl = in ? cl0 + sub : cl0;
    const ClusterTab& T = tabs[cl];
    const ClKind& D = kinds[kind_of[cl]];
    const bool on = in && c < D.nc;
    if (multi) {
      const float2* pb = pbuf + (size_t)3 * cl + c;
      cs_poly_io<RATTLE, false>(pbuf + (size_t)3 * cl + c, ld, P);
      t[0] = df_of(pb[CS_POLY * ld]);
      t[1] = df_shfl(t[0], n1);
      t[2] = df_shfl(t[0], n2);
      const float2 tol = RATTLE ? D.tol_r : D.tol_s[c];
      for (int s = 0; s < last; ++s) cs_sweep<RATTLE>(P, tol, n1, n2, t);
    } else if (done) {
      t[0] = df_of(cs_hist[last * blockDim.x + threadIdx.x]);
    }
    double v[3] = {0.0, 0.0, 0.0};  // t b of the lane's constraint
    if (on) {
      const int k = T.con[c];
      const double b[3] = {A.dxx[k], A.dyy[k], A.dzz[k]};
      double tt = df_to_double(t[0]);
      if (RATTLE) {
        const double b2 = b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
        double r = rsqrt_seeded(b2);
        r = r * fma(-0.5 * b2 * r, r, 1.5);
        tt *= r;  // unit bond vectors
      } else {
        const double g = D.two_m[c] * tt;
        int m = 0;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const double gb = -g * b[p];
#pragma unroll
          for (int q = p; q < 3; ++q, ++m) st[m] = fma(gb, b[q], st[m]);
        }
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) v[p] = tt * b[p];
    }
    double w[CS_MAXC][3];
#pragma unroll
    for (int k = 0; k < CS_MAXC; ++k)
#pragma unroll
      for (int p = 0; p < 3; ++p) w[k][p] = __shfl_sync(0xffffffffu, v[p], 3 * sub + k);
    if (!in) continue;
    for (int a = c; a < D.na; a += CS_MAXC) {
      if (__double_as_longlong(D.wh[a]) == 0) continue;
      double dx = 0.0, dy = 0.0, dz = 0.0;
#pragma unroll
      for (int k = 0; k < CS_MAXC; ++k) {
        const double f = D.W[a][k];
        if (__double_as_longlong(f) == 0) continue;
        dx = fma(f, w[k][0], dx); dy = fma(f, w[k][1], dy); dz = fma(f, w[k][2], dz);
      }
      const int i = T.atom[a];
      if (RATTLE) {
        A.vx[i] += dx; A.vy[i] += dy; A.vz[i] += dz;
      } else {
        const double x0 = A.x[i], y0 = A.y[i], z0 = A.z[i];
        const double x1 = x0 + dx, y1 = y0 + dy, z1 = z0 + dz;
        A.x[i] = x1; A.y[i] = y1; A.z[i] = z1;
        const double ux = (x1 - x0) * rstep, uy = (y1 - y0) * rstep, uz = (z1 - z0) * rstep;
        A.vx[i] += ux; A.vy[i] += uy; A.vz[i] += uz;
        fx[i] += ux * D.wh[a]; fy[i] += uy * D.wh[a]; fz[i] += uz * D.wh[a];
      }
    }
  }
  if (!RATTLE) {
    block_reduce_store<6>(st, A.blk);
    grid_finish<6>(A.blk, A.gs);
  }
}

// apply_shake epilogue: v += dr/dt, f += dr/dt * m/(dt/2) for constrained atoms
__global__ void k_shake_post(int n, const int* astart, const int* lfrzn, double rstep, double hstep, const double* w,
                             const double* x, const double* y, const double* z, const double* ox, const double* oy,
                             const double* oz, double* vx, double* vy, double* vz, double* fx, double* fy,
                             double* fz, StopIf stop) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || stop.set()) return;
  if (astart[i + 1] == astart[i] || lfrzn[i] != 0) return;
  double xt = (x[i] - ox[i]) * rstep, yt = (y[i] - oy[i]) * rstep, zt = (z[i] - oz[i]) * rstep;
  vx[i] += xt; vy[i] += yt; vz[i] += zt;
  double tmp = w[i] / hstep;
  fx[i] += xt * tmp; fy[i] += yt * tmp; fz[i] += zt * tmp;
}

__global__ void k_copy3(int n, const double* a, const double* b, const double* c, double* oa, double* ob, double* oc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { oa[i] = a[i]; ob[i] = b[i]; oc[i] = c[i]; }
}

int* d_flags = nullptr;
int coop_blocks_shake = 0, coop_blocks_rattle = 0;
// cluster-local path (used when every constraint cluster is small)
ClusterTab* d_cltab = nullptr;
double* d_clring = nullptr;  // per-cluster state ring (CL_RING slots of CL_SLOT doubles)
double* d_clgsum = nullptr;  // per-cluster committed SHAKE gamma sums
int n_clusters = 0, coop_blocks_cl = 0;
constexpr int CL_THREADS = 128;  // small blocks spread the clusters over every SM
// clusters of at most 3 constraints (k_constrain_small)
int* d_clkind = nullptr;     // kind of each cluster
ClKind* d_kinds = nullptr;
float2* d_clt = nullptr;     // polynomials and scalars, when there are more clusters than resident lanes
bool cl_small = false;
int coop_blocks_small = 0, cs_threads = 32;
const void* cl_kernel = nullptr;  // k_constrain_cl instantiation for the largest cluster

// The form by FP64 instructions keeps k_constrain_cl: it is there to check the others.
bool use_small() { return cl_small && !g.fp64_native; }

// connected constraint clusters; false when one exceeds CL_MAXA atoms or CL_MAXC constraints
bool build_clusters(const std::vector<int>& ci, const std::vector<int>& cj, std::vector<ClusterTab>& out) {
  const int n = g.natms, nc = (int)ci.size();
  std::vector<int> parent(n);
  for (int i = 0; i < n; ++i) parent[i] = i;
  auto find = [&](int a) {
    while (parent[a] != a) a = parent[a] = parent[parent[a]];
    return a;
  };
  for (int k = 0; k < nc; ++k) {
    const int a = find(ci[k]), b = find(cj[k]);
    if (a != b) parent[std::max(a, b)] = std::min(a, b);
  }
  std::vector<int> root_id(n, -1);
  out.clear();
  std::vector<std::vector<int>> atoms, cons;
  for (int k = 0; k < nc; ++k) {  // clusters in order of their first constraint; constraints ascending
    const int r = find(ci[k]);
    if (root_id[r] < 0) {
      root_id[r] = (int)atoms.size();
      atoms.emplace_back();
      cons.emplace_back();
    }
    cons[root_id[r]].push_back(k);
  }
  for (size_t c = 0; c < cons.size(); ++c) {
    for (int k : cons[c])
      for (int e : {ci[k], cj[k]})
        if (std::find(atoms[c].begin(), atoms[c].end(), e) == atoms[c].end()) atoms[c].push_back(e);
    if ((int)atoms[c].size() > CL_MAXA || (int)cons[c].size() > CL_MAXC) return false;
  }
  out.resize(cons.size());
  for (size_t c = 0; c < cons.size(); ++c) {
    ClusterTab& T = out[c];
    for (int a = 0; a < CL_MAXA; ++a) { T.atom[a] = -1; T.alist[a] = 0; }
    for (int q = 0; q < CL_MAXC; ++q) { T.con[q] = -1; T.pair[q] = 0; }
    const int na = (int)atoms[c].size(), ncl = (int)cons[c].size();
    for (int a = 0; a < na; ++a) T.atom[a] = atoms[c][a];
    auto local = [&](int gid) { return (int)(std::find(atoms[c].begin(), atoms[c].end(), gid) - atoms[c].begin()); };
    for (int q = 0; q < ncl; ++q) {
      const int k = cons[c][q];
      T.con[q] = k;
      const int li = local(ci[k]), lj = local(cj[k]);
      T.pair[q] = li | (lj << 4);
      // per-atom entries in constraint order, as the global per-atom table holds them
      for (int end = 0; end < 2; ++end) {
        const int la = end ? lj : li;
        const int cnt = T.alist[la] & 15;
        T.alist[la] = (T.alist[la] & ~15) | (cnt + 1);
        T.alist[la] |= ((q << 1) | end) << (4 + 4 * cnt);
      }
    }
    T.meta = na | (ncl << 4);
  }
  return true;
}

// Kinds of the clusters for k_constrain_small; false when a cluster has more than 3
// constraints, a constraint has no movable end (its gamma divides by zero) or a length
// that reaches the range where the minimum image of a moving bond can change.
bool build_kinds(const std::vector<ClusterTab>& tabs, const std::vector<double>& d0, std::vector<int>& kind_of,
                 std::vector<ClKind>& kinds) {
  std::vector<double> w(g.natms);
  std::vector<int> frz(g.natms);
  GB_CUDA(cudaMemcpy(w.data(), g.weight, sizeof(double) * g.natms, cudaMemcpyDeviceToHost));
  GB_CUDA(cudaMemcpy(frz.data(), g.lfrzn, sizeof(int) * g.natms, cudaMemcpyDeviceToHost));
  const double dt = g.p.tstep, tol = g.p.shake_tol;
  auto split = [](double v) {
    float2 r;
    df_split(v, &r.x, &r.y);
    return r;
  };
  std::map<std::string, int> seen;
  kind_of.resize(tabs.size());
  kinds.clear();
  for (size_t q = 0; q < tabs.size(); ++q) {
    const ClusterTab& T = tabs[q];
    ClKind D;
    std::memset((void*)&D, 0, sizeof(D));
    D.na = T.meta & 15;
    D.nc = (T.meta >> 4) & 15;
    if (D.nc > CS_MAXC || D.na > CL_MAXA) return false;
    double iw[CL_MAXA] = {0, 0, 0, 0};  // amt without its power of tstep
    for (int a = 0; a < D.na; ++a) {
      const int i = T.atom[a];
      iw[a] = frz[i] ? 0.0 : 1.0 / w[i];
      D.wh[a] = frz[i] ? 0.0 : w[i] / (0.5 * dt);
    }
    double W[CL_MAXA][CS_MAXC] = {};
    for (int c = 0; c < D.nc; ++c) {
      D.li[c] = T.pair[c] & 15;
      D.lj[c] = T.pair[c] >> 4;
      const double m = iw[D.li[c]] + iw[D.lj[c]], len = d0[T.con[c]];
      if (!(m > 0.0) || !std::isfinite(m) || !(len > 0.0 && len < 0.125 * g.cell[0]) || D.li[c] == D.lj[c]) return false;
      W[D.li[c]][c] -= iw[D.li[c]] / m;
      W[D.lj[c]][c] += iw[D.lj[c]] / m;
      D.d0sq[c] = len * len;
      D.two_m[c] = 2.0 / (m * dt * dt);
      D.off = std::max(D.off, std::ldexp(1.f, std::ilogb(len * len) + 4));
      D.tol_s[c] = split(2.0 * (tol * len));
    }
    D.tol_r = split(tol / (0.5 * dt));
    std::memcpy(D.W, W, sizeof(W));
    for (int c = 0; c < D.nc; ++c)
      for (int k = 0; k < D.nc; ++k) D.K[c][k] = split(W[D.li[c]][k] - W[D.lj[c]][k]);
    const std::string key((const char*)&D, sizeof(D));
    auto it = seen.find(key);
    if (it == seen.end()) {
      it = seen.emplace(key, (int)kinds.size()).first;
      kinds.push_back(D);
    }
    kind_of[q] = it->second;
  }
  return true;
}

}  // namespace

// ===================================================================== host
void integ_setup_constraints(const int32_t* listcon, const double* prmcon) {
  const int nc = g.ntcons;
  if (nc == 0) return;
  std::vector<int> ci(nc), cj(nc), lt(g.natms, 0);
  std::vector<double> d0(nc);
  for (int k = 0; k < nc; ++k) {
    ci[k] = listcon[3 * k + 1] - 1;
    cj[k] = listcon[3 * k + 2] - 1;
    d0[k] = prmcon[listcon[3 * k] - 1];
    lt[ci[k]]++; lt[cj[k]]++;
  }
  // per-atom constraint table in constraint order; bit 0 = atom is the j end
  std::vector<int> start(g.natms + 1, 0), list;
  for (int i = 0; i < g.natms; ++i) start[i + 1] = start[i] + lt[i];
  list.resize(start[g.natms]);
  std::vector<int> fill(g.natms, 0);
  for (int k = 0; k < nc; ++k) {
    list[start[ci[k]] + fill[ci[k]]++] = (k << 1) | 0;
    list[start[cj[k]] + fill[cj[k]]++] = (k << 1) | 1;
  }
  GB_CUDA(cudaMalloc(&g.con_i, sizeof(int) * nc));
  GB_CUDA(cudaMalloc(&g.con_j, sizeof(int) * nc));
  GB_CUDA(cudaMalloc(&g.con_d0, sizeof(double) * nc));
  GB_CUDA(cudaMalloc(&g.listot, sizeof(int) * g.natms));
  GB_CUDA(cudaMalloc(&g.acon_start, sizeof(int) * (g.natms + 1)));
  GB_CUDA(cudaMalloc(&g.acon_list, sizeof(int) * std::max<size_t>(1, list.size())));
  for (double** p : {&g.dxx, &g.dyy, &g.dzz, &g.dxt, &g.dyt, &g.dzt, &g.dt2, &g.gam})
    GB_CUDA(cudaMalloc(p, sizeof(double) * nc));
  GB_CUDA(cudaMemcpy(g.con_i, ci.data(), sizeof(int) * nc, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.con_j, cj.data(), sizeof(int) * nc, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.con_d0, d0.data(), sizeof(double) * nc, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.listot, lt.data(), sizeof(int) * g.natms, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.acon_start, start.data(), sizeof(int) * (g.natms + 1), cudaMemcpyHostToDevice));
  if (!list.empty())
    GB_CUDA(cudaMemcpy(g.acon_list, list.data(), sizeof(int) * list.size(), cudaMemcpyHostToDevice));
  if (d_flags) cudaFree(d_flags);
  GB_CUDA(cudaMalloc(&d_flags, sizeof(int) * (g.p.shake_maxit + CL_CHUNK + 2)));
  int bps = 0;
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_shake, 256, 0));
  coop_blocks_shake = std::max(1, std::min(bps * g.nsm, nblocks(std::max(nc, g.natms), 256)));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_rattle, 256, 0));
  coop_blocks_rattle = std::max(1, std::min(bps * g.nsm, nblocks(std::max(nc, g.natms), 256)));
  // cluster-local sweeps when every cluster is small (GB_SHAKE_GLOBAL=1 keeps the per-sweep kernels)
  if (d_cltab) { cudaFree(d_cltab); d_cltab = nullptr; }
  if (d_clring) { cudaFree(d_clring); d_clring = nullptr; }
  if (d_clgsum) { cudaFree(d_clgsum); d_clgsum = nullptr; }
  if (d_clkind) { cudaFree(d_clkind); d_clkind = nullptr; }
  if (d_kinds) { cudaFree(d_kinds); d_kinds = nullptr; }
  if (d_clt) { cudaFree(d_clt); d_clt = nullptr; }
  cl_small = false;
  n_clusters = 0;
  const char* env = std::getenv("GB_SHAKE_GLOBAL");
  std::vector<ClusterTab> tabs;
  if (!(env && env[0] == '1') && build_clusters(ci, cj, tabs)) {
    n_clusters = (int)tabs.size();
    GB_CUDA(cudaMalloc(&d_cltab, sizeof(ClusterTab) * tabs.size()));
    GB_CUDA(cudaMemcpy(d_cltab, tabs.data(), sizeof(ClusterTab) * tabs.size(), cudaMemcpyHostToDevice));
    std::vector<int> kind_of;
    std::vector<ClKind> kinds;
    // k_constrain_small where it applies (water: 0.83 ms a call in k_constrain_cl)
    cl_small = build_kinds(tabs, d0, kind_of, kinds);
    if (cl_small) {
      GB_CUDA(cudaMalloc(&d_clkind, sizeof(int) * kind_of.size()));
      GB_CUDA(cudaMemcpy(d_clkind, kind_of.data(), sizeof(int) * kind_of.size(), cudaMemcpyHostToDevice));
      GB_CUDA(cudaMalloc(&d_kinds, sizeof(ClKind) * kinds.size()));
      GB_CUDA(cudaMemcpy(d_kinds, kinds.data(), sizeof(ClKind) * kinds.size(), cudaMemcpyHostToDevice));
      // one block per SM (the fewest to meet at a grid barrier), wide enough for all clusters
      const int nwarp = (n_clusters + CS_PERWARP - 1) / CS_PERWARP;
      cs_threads = 32 * std::min((nwarp + g.nsm - 1) / g.nsm, CS_THREADS / 32);
      coop_blocks_small = std::min(g.nsm, nblocks(nwarp, cs_threads / 32));
      const int smem = (int)sizeof(float2) * CS_CHUNK * CS_THREADS;
      GB_CUDA(cudaFuncSetAttribute(k_constrain_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      GB_CUDA(cudaFuncSetAttribute(k_constrain_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (coop_blocks_small * (cs_threads / 32) < nwarp)
        GB_CUDA(cudaMalloc(&d_clt, sizeof(float2) * (CS_POLY + 2) * CS_MAXC * tabs.size()));
    }
    // and k_constrain_cl, for the other clusters and the FP64 form by instructions
    GB_CUDA(cudaMalloc(&d_clring, sizeof(double) * CL_RING * CL_SLOT * tabs.size()));
    GB_CUDA(cudaMalloc(&d_clgsum, sizeof(double) * CL_MAXC * tabs.size()));
    // rigid 3-site molecules get register arrays sized 3 x 3 (more resident warps)
    bool three = true;
    for (const ClusterTab& T : tabs)
      if ((T.meta & 15) > 3 || ((T.meta >> 4) & 15) > 3) three = false;
    cl_kernel = three ? (const void*)k_constrain_cl<3, 3> : (const void*)k_constrain_cl<CL_MAXA, CL_MAXC>;
    GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, cl_kernel, CL_THREADS, 0));
    coop_blocks_cl = std::max(1, std::min(bps * g.nsm, nblocks(n_clusters, CL_THREADS)));
  }
}

void integ_forces_to_fp64() {
  k_fix_to_fp64<<<nblocks(g.natms, 256), 256, 0, g.stream>>>(g.natms, g.fixp, g.fx, g.fy, g.fz);
  GB_LAUNCHED();
}

// The displacement check, with the NVE stage 1 in the same pass when stage1 is set.  The
// caller has cleared maxdisp.
static void launch_maxdisp(bool stage1) {
  k_maxdisp<<<std::min(nblocks(g.natms, 128), 4 * g.nsm), 128, 0, g.stream>>>(
      g.natms, stage1 ? g.hdw : nullptr, g.p.tstep, g.fx, g.fy, g.fz, g.vx, g.vy, g.vz, g.x, g.y, g.z, g.xbg, g.ybg,
      g.zbg, g.cell[0], 1.0 / g.cell[0], (unsigned long long*)&g.sc->maxdisp, stop_if(ST_STOP1), stamp_at(0));
  GB_LAUNCHED();
}

// NVE without constraints: stage 1 and the displacement check as one kernel
void integ_stage1_check() {
  GB_CUDA(cudaMemsetAsync(&g.sc->maxdisp, 0, sizeof(double), g.stream));
  prof_begin(P_VV);
  launch_maxdisp(true);
  prof_end(P_VV);
}

void integ_vnl_launch() {
  GB_CUDA(cudaMemsetAsync(&g.sc->maxdisp, 0, sizeof(double), g.stream));
  launch_maxdisp(false);
}

int integ_vnl_result() { return std::sqrt(g.hsc->maxdisp) >= std::nextafter(0.5, 0.0) * g.p.rpad ? 1 : 0; }

int integ_vnl_check() {
  integ_vnl_launch();
  gb_sync_scalars();
  return integ_vnl_result();
}

static void con_args(ConArgs& A, int stop) {
  A.nc = g.ntcons; A.natms = g.natms; A.maxit = g.p.shake_maxit;
  A.ci = g.con_i; A.cj = g.con_j; A.listot = g.listot; A.astart = g.acon_start; A.alist = g.acon_list;
  A.lfrzn = g.lfrzn; A.d0 = g.con_d0;
  A.dxx = g.dxx; A.dyy = g.dyy; A.dzz = g.dzz; A.dxt = g.dxt; A.dyt = g.dyt; A.dzt = g.dzt;
  A.dt2 = g.dt2; A.gam = g.gam;
  A.x = g.x; A.y = g.y; A.z = g.z; A.vx = g.vx; A.vy = g.vy; A.vz = g.vz; A.w = g.weight;
  A.tstep = g.p.tstep; A.tol = g.p.shake_tol; A.c0 = g.cell[0]; A.a0 = 1.0 / g.cell[0];
  A.flags = d_flags; A.sc = g.sc; A.blk = nullptr; A.gs = {nullptr, nullptr}; A.tags = false;
  A.stop = stop_if(stop);
}

template <bool RATTLE>
static void launch_small(ConArgs& A, double rstep) {
  const ClusterTab* tabs = d_cltab;
  const int* kind = d_clkind;
  const ClKind* kinds = d_kinds;
  int ncl = n_clusters;
  float2* tbuf = d_clt;
  double *fx = g.fx, *fy = g.fy, *fz = g.fz;
  void* args[] = {&A, &tabs, &kind, &kinds, &ncl, &tbuf, &rstep, &fx, &fy, &fz};
  GB_CUDA(cudaLaunchCooperativeKernel((void*)k_constrain_small<RATTLE>, coop_blocks_small, cs_threads, args,
                                      sizeof(float2) * CS_CHUNK * cs_threads, g.stream));
}

// constraints_tags (constraints.F90:438-586): old bond vectors from the current positions
void integ_con_tags() {
  if (g.ntcons <= 0) return;
  k_con_tags<<<nblocks(g.ntcons, 256), 256, 0, g.stream>>>(g.ntcons, g.con_i, g.con_j, g.x, g.y, g.z, g.cell[0],
                                                             1.0 / g.cell[0], g.dxx, g.dyy, g.dzz);
  GB_LAUNCHED();
}

// apply_shake (constraints.F90:1071-1200): the current positions are the unconstrained
// ones (oxt); SHAKE against the bond vectors of the last integ_con_tags, then the velocity
// and force corrections.  Throws GB_ERR_SHAKE when the iteration does not converge.
void integ_shake(int* iters, double* vircon, double* strcon) {
  if (iters) *iters = 0;
  if (g.ntcons <= 0) return;
  cudaStream_t st = g.stream;
  const bool small = use_small();
  const int n = g.natms;
  const double tstep = g.p.tstep, hstep = 0.5 * tstep, rstep = 1.0 / tstep;
  if (!small) {
    k_copy3<<<nblocks(n, 256), 256, 0, st>>>(n, g.x, g.y, g.z, g.ox, g.oy, g.oz);
    GB_LAUNCHED();
  }
  GB_CUDA(cudaMemsetAsync(d_flags, 0, sizeof(int) * (g.p.shake_maxit + CL_CHUNK + 2), st));
  ConArgs A;
  con_args(A, ST_STOP1);
  const int nbs = small ? coop_blocks_small : n_clusters ? coop_blocks_cl : coop_blocks_shake;
  A.blk = gb_blkacc(nbs * 6);
  if (small) A.gs = gb_grid_sum(nbs, cs_threads, 6, &g.sc->acc[A_STRCON]);
  prof_begin(P_SHAKE);
  if (small) {
    launch_small<false>(A, rstep);
  } else if (n_clusters) {
    const ClusterTab* tabs = d_cltab;
    int ncl = n_clusters, rattle = 0;
    double *ring = d_clring, *gsum = d_clgsum;
    GB_CUDA(cudaMemsetAsync(d_clgsum, 0, sizeof(double) * CL_MAXC * n_clusters, st));
    void* args[] = {&A, &tabs, &ncl, &ring, &gsum, &rattle};
    GB_CUDA(cudaLaunchCooperativeKernel(cl_kernel, nbs, CL_THREADS, args, 0, st));
  } else {
    void* args[] = {&A};
    GB_CUDA(cudaLaunchCooperativeKernel((void*)k_shake, nbs, 256, args, 0, st));
  }
  GB_LAUNCHED();
  prof_end(P_SHAKE);
  if (!A.gs.count) gb_reduce_blocks(A.blk, nbs, 6, &g.sc->acc[A_STRCON]);
  if (!small) {
    k_shake_post<<<nblocks(n, 256), 256, 0, st>>>(n, g.acon_start, g.lfrzn, rstep, hstep, g.weight, g.x, g.y, g.z,
                                                   g.ox, g.oy, g.oz, g.vx, g.vy, g.vz, g.fx, g.fy, g.fz,
                                                   stop_if(ST_STOP1));
    GB_LAUNCHED();
  }
  if (g.defer_scalars) return;  // the MD loop reads the sums and the status
  gb_sync_scalars();
  if (iters) *iters = g.hsc->shake_iters;
  con_scalars(g.hsc, vircon, strcon);
  if (g.hsc->status & ST_SHAKE_FAIL) throw (int)GB_ERR_SHAKE;
}

// apply_rattle with kit = 1 (constraints.F90:1032-1069 -> constraints_rattle :587-775) on
// the current velocities, against the bond vectors of the last integ_con_tags or, with
// tags, of the current positions (constraints_tags as part of the kernel).  The
// status is read by the caller (ST_RATTLE_FAIL).
void integ_rattle_launch(bool tags) {
  if (g.ntcons <= 0) return;
  cudaStream_t st = g.stream;
  const bool small = use_small();
  GB_CUDA(cudaMemsetAsync(d_flags, 0, sizeof(int) * (g.p.shake_maxit + CL_CHUNK + 2), st));
  ConArgs A;
  con_args(A, ST_STOP2);
  if (tags && !small) integ_con_tags();
  A.tags = tags;
  prof_begin(P_RATTLE);
  if (small) {
    launch_small<true>(A, 0.0);
  } else if (n_clusters) {
    const ClusterTab* tabs = d_cltab;
    int ncl = n_clusters, rattle = 1;
    double *ring = d_clring, *gsum = d_clgsum;
    void* args[] = {&A, &tabs, &ncl, &ring, &gsum, &rattle};
    GB_CUDA(cudaLaunchCooperativeKernel(cl_kernel, coop_blocks_cl, CL_THREADS, args, 0, st));
  } else {
    void* args[] = {&A};
    GB_CUDA(cudaLaunchCooperativeKernel((void*)k_rattle, coop_blocks_rattle, 256, args, 0, st));
  }
  GB_LAUNCHED();
  prof_end(P_RATTLE);
}

// kinetic stress into acc[A_STRKIN], after the second half kick when kick is set
static void launch_kinstress(bool kick) {
  const int nb = std::min(nblocks(g.natms, KIN_NT), 2 * g.nsm);
  const GridSum gs = gb_grid_sum(nb, KIN_NT, 6, &g.sc->acc[A_STRKIN]);
  double* part = gb_blkacc(nb * 6);
  k_kinstress<<<nb, KIN_NT, 0, g.stream>>>(g.natms, g.weight, g.lfrzn, kick ? g.hdw : nullptr, g.fx, g.fy, g.fz, g.vx,
                                           g.vy, g.vz, part, gs, stop_if(ST_STOP2), kick ? stamp_at(2) : nullptr);
  GB_LAUNCHED();
  gb_grid_sum_done(gs, part, nb, 6);
}

void integ_vv(int stage, double* strkin, double* engke, int* iters, double* vircon, double* strcon) {
  cudaStream_t st = g.stream;
  const int n = g.natms;
  const double tstep = g.p.tstep, hstep = 0.5 * tstep;
  if (iters) *iters = 0;
  if (stage == 1) {
    integ_con_tags();
    prof_begin(P_VV);
    if (!thermo_vv1(hstep, tstep)) {
      k_vv1<<<nblocks(n, 256), 256, 0, st>>>(n, g.hdw, tstep, g.fx, g.fy, g.fz, g.vx, g.vy, g.vz, g.x, g.y, g.z,
                                             stop_if(ST_STOP1));
      GB_LAUNCHED();
    }
    prof_end(P_VV);
    integ_shake(iters, vircon, strcon);
  } else {
    const bool fused = g.ntcons <= 0 && g.ens == GB_NVE;  // the kick and the kinetic stress in one pass
    prof_begin(P_VV);
    if (!fused) {
      k_vv2<<<nblocks(n, 256), 256, 0, st>>>(n, g.hdw, g.fx, g.fy, g.fz, g.vx, g.vy, g.vz, stop_if(ST_STOP2),
                                             stamp_at(2));
      GB_LAUNCHED();
    }
    if (fused) launch_kinstress(true);
    prof_end(P_VV);
    integ_rattle_launch(true);
    if (!thermo_vv2_finish(strkin, engke)) {
      if (!fused) launch_kinstress(false);
      if (g.defer_scalars) return;  // the MD loop reads the sums after its last step
      gb_sync_scalars();
      kin_scalars(g.hsc, strkin, engke);
    }
    if (g.defer_scalars) return;
    if (iters && g.ntcons > 0) *iters = g.hsc->rattle_iters;
    if (g.ntcons > 0 && (g.hsc->status & ST_RATTLE_FAIL)) throw (int)GB_ERR_RATTLE;
    if (g.hsc->status & ST_RNG) throw (int)GB_ERR_RNG;
    if (g.hsc->status & ST_DEVICE_WAIT) throw (int)GB_ERR_DEVICE_WAIT;
  }
}

// virial and stress (symmetric 3x3) of the SHAKE stage from the device sums
void con_scalars(const DevScalars* h, double* vircon, double* strcon) {
  const double* s = &h->acc[A_STRCON];
  const double str[9] = {s[0], s[1], s[2], s[1], s[3], s[4], s[2], s[4], s[5]};
  if (strcon) for (int k = 0; k < 9; ++k) strcon[k] = str[k];
  if (vircon) *vircon = -(str[0] + str[4] + str[8]);
}

// kinetic stress (symmetric 3x3) and kinetic energy from the device sums
void kin_scalars(const DevScalars* h, double* strkin, double* engke) {
  const double* s = &h->acc[A_STRKIN];
  double sk[9] = {s[0], s[1], s[2], s[1], s[3], s[4], s[2], s[4], s[5]};
  if (strkin) for (int k = 0; k < 9; ++k) strkin[k] = sk[k];
  if (engke) *engke = 0.5 * (sk[0] + sk[4] + sk[8]);
}
