// gb_metal.cu - tabulated embedded-atom (EAM) metal forces on the device: the
// two passes of the reference (local density, then forces) over the Verlet list.
//
// Follows:
//   metal_table_read          source/metal.F90:1489-1925 (tab = 1, 'eam': pair, dens, embe tables)
//   metal_table_derivatives   source/metal.F90:2807-2897 (five-point derivative of each table)
//   metal_ld_compute          source/metal.F90:897-1257 (embedding F(rho), F'(rho), error 507)
//   metal_ld_collect_eam      source/metal.F90:2207-2516 (density pass, error 506)
//   metal_ld_set_halo         source/metal.F90:3146 (F'(rho) on the halo images)
//   metal_forces              source/metal.F90:193-895 (tabulated EAM branch)
// in the serial build without HALF_HALO (the default), whose bookkeeping is: a
// pair across the cell boundary is listed from both sides; each side adds only
// to its own local atom, and its energy is counted from the side with the smaller
// global id.  Here such a pair is evaluated once, from that side, and applied to
// both atoms, which gives the same sums.
//
// Every table value is interpolated with the reference's three-point formula
// (the l-1, l, l+1 points, its branch on ppp < 0 and l == 5).  Forces are summed
// in FP64 (the FP64 form; metals are not offered in the mixed form).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "gb_common.cuh"
#include "gb_dfr.cuh"

namespace {

inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

__device__ __forceinline__ double interp3(const double* v, int l, double ppp);
__device__ __forceinline__ double interp3_raw(const double* v, int l, double ppp) { return interp3(v, l, ppp); }

struct MetTab {
  int n;          // Nint(buffer(1)) = ngrid + 4; 0 = no table
  int off;        // values at v[off + i], i = 1..n (Fortran index), derivatives at d[off + i]
  double r0;      // start - 5*dr
  double rmax;    // finish
  double dr;
  double rdr;     // 1/dr as the reference forms it
  int grid;       // tables with the same (r0, rdr, n) share a grid id: one index serves them all
  int listed;     // pair tables: the FIELD 'metal' directive lists this type pair (keypot 0)
  double nr0rdr;  // -r0 * rdr: x = r * rdr + nr0rdr
  long long b_lo, b_hi;  // r <= rmax decided on rsq bits outside [rmax^2 (1 -+ 1e-12)]
  // double-float kernels: r <= rmax decided on rsq outside [f_lo, f_hi] (1e-6 around
  // rmax^2; -1 without a table), and rdr, nr0rdr as double-floats
  float f_lo, f_hi, rdr_h, rdr_l, nr_h, nr_l;
};

// r <= rmax as the reference decides it (correctly rounded sqrt), from the bits of rsq
// except inside a narrow band around rmax^2
__device__ __forceinline__ bool within(long long rb, long long lo, long long hi, double rsq, double rmax) {
  return rb < lo || (rb <= hi && sqrt(rsq) <= rmax);
}

// The three-point formula is the quadratic through (l-1, l, l+1) in both of its
// ppp branches, so the force passes evaluate it from per-point coefficients
// c0 + p (c1 + p c2), c0 = v_l, c1 = (v_{l+1} - v_{l-1})/2, c2 = (v_{l+1} - 2 v_l + v_{l-1})/2
// (two FMAs).  Entry l = 5 holds the linear form the reference uses there for
// ppp >= 0; the rare l = 5, ppp < 0 case and the density's negative fall-back read
// the raw values.
struct Coef {
  double c0, c1, c2, pad;
};

__device__ __forceinline__ double qeval(const Coef* c, int l, double p) {
  const double2 a = *reinterpret_cast<const double2*>(&c[l].c0);
  const double b = c[l].c2;
  return fma(p, fma(p, b, a.y), a.x);
}

// l = Nint((r - r0) / dr) clamped to [5, n-1] and ppp: the nearest integer comes from
// adding 1.5*2^52 (no FP64 conversion); false if the reference's l < 5 guard fires
__device__ __forceinline__ bool qindex(const MetTab& t, double r, int* l, double* ppp) {
  const double x = fma(r, t.rdr, t.nr0rdr);
  const double big = 6755399441055744.0;
  const double tt = x + big;
  int k = __double2loint(tt);
  double kd = tt - big;
  bool ok = true;
  if (k > t.n - 1) { k = t.n - 1; kd = (double)k; }
  if (k < 5) { ok = false; k = 6; kd = 6.0; }
  *l = k;
  *ppp = x - kd;
  return ok;
}

__device__ __forceinline__ double qeval_full(const Coef* c, const double* raw, int l, double p) {
  if (l == 5 && p < 0.0) return interp3_raw(raw, l, p);
  return qeval(c, l, p);
}

// metal_ld_compute / metal_forces interpolation: index l and fraction ppp
__device__ __forceinline__ bool tab_index(const MetTab& t, double r, int* l, double* ppp) {
  const double rr1 = r - t.r0;
  int k = min((int)round(rr1 * t.rdr), t.n - 1);
  bool ok = true;
  if (k < 5) { ok = false; k = 6; }
  *l = k;
  *ppp = rr1 * t.rdr - (double)k;
  return ok;
}

__device__ __forceinline__ double interp3(const double* v, int l, double ppp) {
  const double vk0 = v[l - 1], vk1 = v[l], vk2 = v[l + 1];
  const double t1 = vk1 + ppp * (vk1 - vk0);
  const double t2 = vk1 + ppp * (vk2 - vk1);
  if (ppp < 0.0) return t1 + 0.5 * (t2 - t1) * (ppp + 1.0);
  if (l == 5) return t2;
  return t2 + 0.5 * (t2 - t1) * (ppp - 1.0);
}

// density: the same formula, but a negative result falls back to t1 / t2
__device__ __forceinline__ double interp3_density(const double* v, int l, double ppp) {
  const double vk0 = v[l - 1], vk1 = v[l], vk2 = v[l + 1];
  const double t1 = vk1 + ppp * (vk1 - vk0);
  const double t2 = vk1 + ppp * (vk2 - vk1);
  if (ppp < 0.0) {
    const double d = t1 + 0.5 * (t2 - t1) * (ppp + 1.0);
    return d < 0.0 ? t1 : d;
  }
  if (l == 5) return t2;
  const double d = t2 + 0.5 * (t2 - t1) * (ppp - 1.0);
  return d < 0.0 ? t2 : d;
}

struct MetArgs {
  const MetTab* tab;    // [nkey pair | ntypes density | ntypes embedding]
  const double* v;      // table values (column 1), Fortran-indexed from off
  const double* d;      // column 2: -r dV/dr, -r drho/dr, dF/drho
  const Coef* cv;       // quadratic coefficients of column 1 (same offsets)
  const Coef* cd;       // and of column 2
  const int* listed;    // per pair key: 1 if the FIELD lists it (keypot = 0), else 0 (keypot = -1)
  int nkey, ntypes, ntab;
  double rcut;
  long long b_rc_lo, b_rc_hi;   // rcut^2 band as bit patterns
};

constexpr int MAX_TAB = 64;  // tables staged in shared memory (ntypes <= 8)

__device__ __forceinline__ void stage_tables(const MetArgs& A, MetTab* st) {
  for (int k = threadIdx.x; k < A.ntab; k += blockDim.x) st[k] = A.tab[k];
  __syncthreads();
}

// density from one species table; a negative quadratic falls back to t1 / t2 (metal_ld_collect_eam)
__device__ __forceinline__ double density_at(const MetArgs& A, const MetTab& t, int l, double p) {
  double dens = qeval_full(A.cv + t.off, A.v + t.off, l, p);
  const long long db = __double_as_longlong(dens);
  if (db < 0 && db != (long long)0x8000000000000000ull) dens = interp3_density(A.v + t.off, l, p);  // < 0
  return dens;
}

// r from rsq: seeded 1/sqrt (exact sqrt for a zero or subnormal rsq, which the table
// guards then reject)
__device__ __forceinline__ double dist_from(double rsq, long long rb, double* rinv) {
  if (rb < DBL_MIN_BITS) { *rinv = 0.0; return sqrt(rsq); }
  *rinv = rsqrt_seeded(rsq);
  return rsq * (*rinv);
}

__global__ void __launch_bounds__(256) k_metal_density(int natms, const DevScalars* sc, const int* __restrict__ at_list,
                                                       const int* __restrict__ list, int ld, const double* __restrict__ x,
                                                       const double* __restrict__ y, const double* __restrict__ z,
                                                       const int* __restrict__ ltype, const int* __restrict__ ltg,
                                                       const int* __restrict__ src, MetArgs A, double* rho,
                                                       int* status) {
  __shared__ MetTab tabs[MAX_TAB];
  stage_tables(A, tabs);
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nlast = sc->nlast;
  bool bad = false;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nlast; w += nwarps) {
    const int i = at_list[w];
    if (i >= natms) continue;
    const double xi = x[i], yi = y[i], zi = z[i];
    const int ai = ltype[i], gi = ltg[i];
    const MetTab& ti = tabs[A.nkey + ai - 1];
    const int* li = list + (size_t)i * ld + 3;
    const int n = li[0];
    double rho_i = 0.0;
    for (int m = lane + 1; m <= n; m += 32) {
      const int j = li[m] - 1;
      int jf = j;
      if (j >= natms) {
        if (gi > ltg[j]) continue;  // counted from the other side
        jf = src[j];
      }
      const double dx = xi - x[j], dy = yi - y[j], dz = zi - z[j];
      const double rsq = dx * dx + dy * dy + dz * dz;
      const long long rb = __double_as_longlong(rsq);
      const int aj = ltype[j];
      const MetTab& tj = tabs[A.nkey + aj - 1];
      const bool in_j = tj.n > 5 && within(rb, tj.b_lo, tj.b_hi, rsq, tj.rmax);
      const bool in_i = ai != aj && ti.n > 5 && within(rb, ti.b_lo, ti.b_hi, rsq, ti.rmax);
      if (!in_j && !in_i) continue;
      double rinv;
      const double r = dist_from(rsq, rb, &rinv);
      // to i from j's species table, to j from i's (metal_ld_collect_eam)
      int l = 0;
      double p = 0.0;
      int gl = -1;
      double to_j = 0.0;
      if (in_j) {
        if (!qindex(tj, r, &l, &p)) bad = true;
        gl = tj.grid;
        const double dens = density_at(A, tj, l, p);
        rho_i += dens;
        if (ai == aj) to_j = dens;
      }
      if (in_i) {
        if (ti.grid != gl && !qindex(ti, r, &l, &p)) bad = true;
        to_j = density_at(A, ti, l, p);
      }
      if ((__double_as_longlong(to_j) & 0x7FFFFFFFFFFFFFFFll) != 0) atomicAdd(&rho[jf], to_j);
    }
    rho_i = warp_sum(rho_i);
    if (lane == 0 && rho_i != 0.0) atomicAdd(&rho[i], rho_i);
  }
  if (bad) atomicOr(status, ST_METAL_TABLE);
}

// embedding energy and F'(rho) (metal_ld_compute, tab > 0, rho grid)
__global__ void k_metal_embed(int natms, const int* ltype, MetArgs A, double* rho, double* blk, int* status, GridSum gs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double e[1] = {0.0};
  int st = 0;
  if (i < natms) {
    const MetTab& t = A.tab[A.nkey + A.ntypes + ltype[i] - 1];
    if (t.n > 0) {
      const double rhosqr = rho[i];
      if (rhosqr >= t.r0 + 5.0 * t.dr) {
        if (rhosqr <= t.rmax) {
          int l;
          double p;
          if (!tab_index(t, rhosqr, &l, &p)) st |= ST_METAL_DENSITY;
          e[0] = interp3(A.v + t.off, l, p);
          rho[i] = interp3(A.d + t.off, l, p);
        } else {  // beyond the table: F at its last point, F' = 0
          e[0] = A.v[t.off + t.n];
          rho[i] = 0.0;
        }
      } else {
        st |= ST_METAL_DENSITY;
      }
    }
  }
  if (st) atomicOr(status, st);
  block_reduce_store<1>(e, blk);
  grid_finish<1>(blk, gs);
}

// metal_ld_set_halo: images carry F'(rho) of their source atom
__global__ void k_metal_halo(int natms, const DevScalars* sc, const int* src, double* rho) {
  const int k = natms + blockIdx.x * blockDim.x + threadIdx.x;
  if (k < sc->nlast) rho[k] = rho[src[k]];
}

constexpr int MACC = 8;  // engmet, virmet, stress (6)

__global__ void __launch_bounds__(256, 3) k_metal_forces(int natms, const DevScalars* sc, const int* __restrict__ at_list,
                                                      const int* __restrict__ list, int ld, const double* __restrict__ x,
                                                      const double* __restrict__ y, const double* __restrict__ z,
                                                      const int* __restrict__ ltype, const int* __restrict__ ltg,
                                                      const int* __restrict__ src, MetArgs A,
                                                      const double* __restrict__ rho, double* fx, double* fy, double* fz,
                                                      double* blk, int* status, unsigned long long* cnt) {
  __shared__ MetTab tabs[MAX_TAB];
  stage_tables(A, tabs);
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nlast = sc->nlast;
  double acc[MACC];
#pragma unroll
  for (int k = 0; k < MACC; ++k) acc[k] = 0.0;
  bool bad = false;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nlast; w += nwarps) {
    const int i = at_list[w];
    if (i >= natms) continue;
    const double xi = x[i], yi = y[i], zi = z[i], rho_i = rho[i];
    const int ai = ltype[i], gi = ltg[i];
    const MetTab& ti = tabs[A.nkey + ai - 1];
    const int* li = list + (size_t)i * ld + 3;
    const int n = li[0];
    double fix = 0.0, fiy = 0.0, fiz = 0.0;
    int nrc = 0;
    for (int m = lane + 1; m <= n; m += 32) {
      const int j = li[m] - 1;
      int jf = j;
      if (j >= natms) {
        if (gi > ltg[j]) continue;
        jf = src[j];
      }
      const int aj = ltype[j];
      const int key = (ai > aj ? ai * (ai - 1) / 2 + aj : aj * (aj - 1) / 2 + ai) - 1;
      const MetTab& tp = tabs[key];
      if (!tp.listed) continue;  // keypot = -1
      const double dx = xi - x[j], dy = yi - y[j], dz = zi - z[j];
      const double rsq = dx * dx + dy * dy + dz * dz;
      const long long rb = __double_as_longlong(rsq);
      if (!within(rb, A.b_rc_lo, A.b_rc_hi, rsq, A.rcut)) continue;   // rrr <= met%rcut
      ++nrc;
      double rinv;
      const double rrr = dist_from(rsq, rb, &rinv);
      const double inv_rsq = rinv * rinv;
      double eng = 0.0, gamma1 = 0.0, gamma2 = 0.0, gamma3 = 0.0;
      int l = 0, gl = -1;
      double p = 0.0;
      if (tp.n > 0 && within(rb, tp.b_lo, tp.b_hi, rsq, tp.rmax)) {
        if (!qindex(tp, rrr, &l, &p)) bad = true;
        gl = tp.grid;
        gamma1 = qeval_full(A.cd + tp.off, A.d + tp.off, l, p);
        eng = qeval_full(A.cv + tp.off, A.v + tp.off, l, p);
      }
      const MetTab& tj = tabs[A.nkey + aj - 1];
      if (tj.n > 0 && ti.n > 5 && within(rb, tj.b_lo, tj.b_hi, rsq, tj.rmax)) {
        if (tj.grid != gl && !qindex(tj, rrr, &l, &p)) bad = true;
        gl = tj.grid;
        gamma2 = qeval_full(A.cd + tj.off, A.d + tj.off, l, p);
      }
      if (ai == aj) {
        gamma3 = gamma2;
      } else if (ti.n > 5 && within(rb, ti.b_lo, ti.b_hi, rsq, ti.rmax)) {
        if (ti.grid != gl && !qindex(ti, rrr, &l, &p)) bad = true;
        gamma3 = qeval_full(A.cd + ti.off, A.d + ti.off, l, p);
      }
      const double num = gamma1 + (gamma2 * rho_i + gamma3 * rho[j]);  // gamma * rsq
      const double gamma = num * inv_rsq;
      const double fxx = gamma * dx, fyy = gamma * dy, fzz = gamma * dz;
      fix += fxx; fiy += fyy; fiz += fzz;
      atomicAdd(&fx[jf], -fxx);
      atomicAdd(&fy[jf], -fyy);
      atomicAdd(&fz[jf], -fzz);
      acc[0] += eng;
      acc[1] -= num;
      acc[2] = fma(dx, fxx, acc[2]); acc[3] = fma(dx, fyy, acc[3]); acc[4] = fma(dx, fzz, acc[4]);
      acc[5] = fma(dy, fyy, acc[5]); acc[6] = fma(dy, fzz, acc[6]); acc[7] = fma(dz, fzz, acc[7]);
    }
    fix = warp_sum(fix); fiy = warp_sum(fiy); fiz = warp_sum(fiz);
    if (cnt) nrc = warp_sumi(nrc);
    if (lane == 0) {
      atomicAdd(&fx[i], fix);
      atomicAdd(&fy[i], fiy);
      atomicAdd(&fz[i], fiz);
      if (cnt) {  // list entries walked and pairs inside the cutoff, when no pair kernel counts them
        atomicAdd(&cnt[0], (unsigned long long)n);
        atomicAdd(&cnt[1], (unsigned long long)nrc);
      }
    }
  }
  if (bad) atomicOr(status, ST_METAL_TABLE);
  block_reduce_store<MACC>(acc, blk);
}

// ------------------------------------------------------- sorted-position kernels
// Both passes over the list's partners in cell order (spos, as the pair kernels walk it),
// in double-float on the FP32 pipes.  The FP64 kernels above are bound by the FP64 unit
// (1/64 of the FP32 rate): 95 FP64 instructions per 32 list entries, executed for whole
// warps although a fifth of the entries lie beyond the cutoff.  Here an FP32 test of the
// high parts queues the entries that may be inside, and 32 queued pairs at a time are
// evaluated with every lane busy.  256,000 atoms: density 1.97 -> 0.47 ms, forces 4.35 ->
// 0.97 ms (1.04 with 102 registers, two CTAs per SM; a fourth CTA spills and gains
// nothing); latency of the partners and tables, at a third of the issue slots.
//   positions   fixed point (PosRec): the separation is an exact integer difference
//   r           to 1.4e-15 (rms), and its fraction of a table interval from the r of the
//               table's point; an atom's force is summed in FP64 (rms errors against 64
//               bits, 8,788 and 256,000 atoms: forces 5.0e-14 and 5.4e-14, of the FP64 kernels
//               6.7e-14 and 7.4e-14; stress 1.6e-13 and 1.3e-13, theirs 1.6e-12 and 1.4e-12)
// A pair near a cutoff, at an end of its table, next to the middle of two points, with a
// negative density or outside the FP32 range takes the FP64 formulas of the kernels above (metal_density_slow,
// metal_force_slow).  Densities and forces are summed in FP64 per sorted position and
// folded onto the atoms (a halo image's onto its source) afterwards.
struct __align__(16) CoefF {
  float c0h, c0l, c1h, c1l;
  float c2h, c2l, rh, rl;  // r of the point (in the tables of the values)
};

struct MetSorted {
  int natms;
  const int *at_list, *loc_sp, *list, *spos;
  int ld, ldt;
  const float4* xhs;
  const PosRec* rec;
  float sh, sl;                    // scales of its coordinates (fix_diff)
  const double *x, *y, *z, *rho;   // FP64 by atom index, for the slow path
  const CoefF *fv, *fd;            // quadratic coefficients of the values and derivatives
  const float2* fp;                // F'(rho) per sorted position
  float f_pre, f_rc_lo, f_rc_hi;
  double *s0, *s1, *s2;            // sums per sorted position
  double* blk; GridSum gs;
  int* status;
  unsigned long long* cnt;
};

constexpr int MET_NT = 256, MET_U = 4;

// df_norm2 with the squares of the low parts
__device__ __forceinline__ df met_norm2(df x, df y, df z) {
  const df px = two_prod(x.hi, x.hi), py = two_prod(y.hi, y.hi), pz = two_prod(z.hi, z.hi);
  const float cx = __fmaf_rn(__fadd_rn(x.hi, x.hi), x.lo, __fmaf_rn(x.lo, x.lo, px.lo));
  const float cy = __fmaf_rn(__fadd_rn(y.hi, y.hi), y.lo, __fmaf_rn(y.lo, y.lo, py.lo));
  const float cz = __fmaf_rn(__fadd_rn(z.hi, z.hi), z.lo, __fmaf_rn(z.lo, z.lo, pz.lo));
  const df s1 = two_sum(px.hi, py.hi);
  const df s2 = two_sum(s1.hi, pz.hi);
  return quick_two_sum(s2.hi, __fadd_rn(__fadd_rn(__fadd_rn(cx, cy), __fadd_rn(cz, s1.lo)), s2.lo));
}

// r and 1/r^2 (relative error below 1e-14, rms 1.7e-15) of a double-float r^2 in the normal
// range.  The force of a metal pair is a difference of terms that changes forty times as fast as
// r, so r gets three words: the FP32 root to half an ulp (1/r refined from its seed), the
// remainder (r^2 - s^2) / 2s and what FP32 leaves of that quotient.
struct Root {
  float s, q, x;
};
__device__ __forceinline__ Root met_dist(df r2, df* inv) {
  const float rs = rsqrtf(r2.hi);
  const float q0 = __fmul_rn(rs, rs);
  const float g0 = __fmaf_rn(-r2.hi, q0, 1.f);
  const float h = __fmul_rn(0.5f, __fmaf_rn(rs, __fmul_rn(0.5f, g0), rs));  // 1 / 2r
  const float s0 = __fmul_rn(r2.hi, __fadd_rn(h, h));
  Root r;
  r.s = __fmaf_rn(h, __fmaf_rn(-s0, s0, r2.hi), s0);
  const df ss = two_prod(r.s, r.s);
  const df e = two_sum(__fsub_rn(r2.hi, ss.hi), __fsub_rn(r2.lo, ss.lo));
  r.q = __fmul_rn(h, e.hi);
  // (s + q + x)^2 = r^2: x = (e - 2 s q - q^2) / 2s
  r.x = __fmul_rn(h, __fmaf_rn(-r.q, r.q, __fadd_rn(__fmaf_rn(-r.q, __fadd_rn(r.s, r.s), e.hi), e.lo)));
  if (inv) {
    const float q = __fmaf_rn(q0, g0, q0);
    const float g = __fmaf_rn(-r2.lo, q, __fmaf_rn(-r2.hi, q, 1.f));  // 1 - r2 q
    *inv = quick_two_sum(q, __fmul_rn(q, __fmaf_rn(g, g, g)));
  }
  return r;
}

// table point l and fraction p in [-0.5, 0.5] of r; false at a table's ends and
// next to the middle of two points (|p| = 0.5 to FP32, one lookup in 10^7), where the
// interpolant jumps by an eighth of the third difference and FP64 decides which point is nearer.
// p = (r - r_l) / dr from the point's own r: the product r / dr would be rounded at 2^-48 of
// a coordinate of some thousand.
__device__ __forceinline__ bool met_coord(const MetTab& t, const CoefF* __restrict__ c, Root r, int* l, df* p) {
  float k = rintf(__fmaf_rn(r.s, t.rdr_h, t.nr_h));
  if (!(k > 5.f && k < (float)(t.n - 1))) return false;
  int i = (int)k;
  df d;
  for (;;) {
    const float2 rk = *reinterpret_cast<const float2*>(&c[i].rh);
    const df b = two_sum(r.q, -rk.y);
    const df s = two_sum(__fsub_rn(r.s, rk.x), b.hi);  // (neighbours: the difference is exact)
    const df q = quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(b.lo, r.x)));
    d = df_mul(q, df_make(t.rdr_h, t.rdr_l));
    // (the FP32 nearest integer may have been the other neighbour of a midpoint)
    if (d.hi > 0.5f && i + 1 == (int)k + 1) ++i;
    else if (d.hi < -0.5f && i - 1 == (int)k - 1) --i;
    else break;
  }
  *l = i;
  *p = d;
  return i > 5 && i < t.n - 1 && fabsf(d.hi) != 0.5f;
}

__device__ __forceinline__ df met_poly(const CoefF* __restrict__ c, int l, df p) {
  const float4 a = *reinterpret_cast<const float4*>(&c[l].c0h);
  const float2 b = *reinterpret_cast<const float2*>(&c[l].c2h);
  const df t = df_fma(p, df_make(b.x, b.y), df_make(a.z, a.w));
  return df_fma(p, t, df_make(a.x, a.y));
}

// +1 inside a table's reach, 0 beyond it, -1 too near its end for FP32
__device__ __forceinline__ int met_in(const MetTab& t, float r2) { return r2 < t.f_lo ? 1 : r2 > t.f_hi ? 0 : -1; }

__device__ __forceinline__ bool met_plain(float r2) { return r2 > 1e-10f && r2 < 1e10f; }

// FP64 terms of one pair, as the atom-index kernels form them
__device__ __noinline__ void metal_density_slow(const MetArgs& A, const MetTab& ti, const MetTab& tj, bool same, double dx,
                                                double dy, double dz, double* to_i, double* to_j, bool* bad) {
  const double rsq = dx * dx + dy * dy + dz * dz;
  const long long rb = __double_as_longlong(rsq);
  *to_i = *to_j = 0.0;
  const bool in_j = tj.n > 5 && within(rb, tj.b_lo, tj.b_hi, rsq, tj.rmax);
  const bool in_i = !same && ti.n > 5 && within(rb, ti.b_lo, ti.b_hi, rsq, ti.rmax);
  if (!in_j && !in_i) return;
  double rinv;
  const double r = dist_from(rsq, rb, &rinv);
  int l = 0;
  double p = 0.0;
  if (in_j) {
    if (!qindex(tj, r, &l, &p)) *bad = true;
    *to_i = density_at(A, tj, l, p);
    if (same) *to_j = *to_i;
  }
  if (in_i) {
    if (!qindex(ti, r, &l, &p)) *bad = true;
    *to_j = density_at(A, ti, l, p);
  }
}

// false beyond the cutoff; num = gamma r^2
__device__ __noinline__ bool metal_force_slow(const MetArgs& A, const MetTab& tp, const MetTab& ti, const MetTab& tj,
                                              bool same, double dx, double dy, double dz, double fi, double fj,
                                              double* num, double* gamma, double* eng, bool* bad) {
  const double rsq = dx * dx + dy * dy + dz * dz;
  const long long rb = __double_as_longlong(rsq);
  *num = *gamma = *eng = 0.0;
  if (!within(rb, A.b_rc_lo, A.b_rc_hi, rsq, A.rcut)) return false;
  double rinv, gamma1 = 0.0, gamma2 = 0.0, gamma3 = 0.0, p = 0.0;
  const double r = dist_from(rsq, rb, &rinv);
  int l = 0;
  if (tp.n > 0 && within(rb, tp.b_lo, tp.b_hi, rsq, tp.rmax)) {
    if (!qindex(tp, r, &l, &p)) *bad = true;
    gamma1 = qeval_full(A.cd + tp.off, A.d + tp.off, l, p);
    *eng = qeval_full(A.cv + tp.off, A.v + tp.off, l, p);
  }
  if (tj.n > 0 && ti.n > 5 && within(rb, tj.b_lo, tj.b_hi, rsq, tj.rmax)) {
    if (!qindex(tj, r, &l, &p)) *bad = true;
    gamma2 = qeval_full(A.cd + tj.off, A.d + tj.off, l, p);
  }
  if (same) {
    gamma3 = gamma2;
  } else if (ti.n > 5 && within(rb, ti.b_lo, ti.b_hi, rsq, ti.rmax)) {
    if (!qindex(ti, r, &l, &p)) *bad = true;
    gamma3 = qeval_full(A.cd + ti.off, A.d + ti.off, l, p);
  }
  *num = gamma1 + (gamma2 * fi + gamma3 * fj);
  *gamma = *num * (rinv * rinv);
  return true;
}

// The partners of the atom at sorted position p (list row i), 32 MET_U entries at a time
// through the FP32 test, then 32 at a time through eval(j).
template <typename Eval>
__device__ __forceinline__ void met_walk(const MetSorted& S, int i, float4 pi, int* q, Eval eval) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int n = S.list[(size_t)i * S.ld + 3];
  const int* sp = S.spos + (size_t)i * S.ldt;
  int nq = 0;
  for (int base = 0;; base += 32 * MET_U) {
    const bool more = base < n;
    if (more) {
      int jv[MET_U];
      float4 pv[MET_U];
#pragma unroll
      for (int u = 0; u < MET_U; ++u) {
        const int m = base + 32 * u + lane + 1;
        jv[u] = m <= n ? sp[m] : -1;
      }
#pragma unroll
      for (int u = 0; u < MET_U; ++u) pv[u] = jv[u] >= 0 ? S.xhs[jv[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < MET_U; ++u) {
        const float ex = pi.x - pv[u].x, ey = pi.y - pv[u].y, ez = pi.z - pv[u].z;
        const bool keep = jv[u] >= 0 && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= S.f_pre;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if (keep) q[nq + __popc(b & lt)] = jv[u];
        nq += __popc(b);
      }
      __syncwarp();
    }
    while (nq >= 32 || (!more && nq > 0)) {
      const int take = min(nq, 32);
      if (lane < take) eval(q[nq - take + lane]);
      nq -= take;
      __syncwarp();  // the taken slots are read before the next pass appends over them
    }
    if (!more) break;
  }
}

__device__ __forceinline__ dacc dacc_xor(dacc a, int o) {
  const float s = __shfl_xor_sync(0xffffffffu, a.s, o), c = __shfl_xor_sync(0xffffffffu, a.c, o);
  const df u = two_sum(a.s, s);
  dacc r;
  r.s = u.hi;
  r.c = __fadd_rn(__fadd_rn(a.c, c), u.lo);
  return r;
}

__global__ void __launch_bounds__(MET_NT) k_metal_density_sorted(MetSorted S, MetArgs A) {
  __shared__ MetTab tabs[MAX_TAB];
  __shared__ int queue[MET_NT / 32][32 * (MET_U + 1)];
  stage_tables(A, tabs);
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  bool bad = false;
  const int per = (S.natms + gridDim.x - 1) / gridDim.x;
  const int a_end = min(S.natms, (int)(blockIdx.x + 1) * per);
  for (int a = blockIdx.x * per + wq; a < a_end; a += MET_NT / 32) {
    const int p = S.loc_sp[a], i = S.at_list[p];
    const PosRec ri = S.rec[p];
    const int ai = ri.type;
    const MetTab& ti = tabs[A.nkey + ai - 1];
    dacc rho = {0.f, 0.f};
    met_walk(S, i, S.xhs[p], queue[wq], [&](int j) {
      const PosRec rj = S.rec[j];
      const bool same = rj.type == ai;
      const MetTab& tj = tabs[A.nkey + rj.type - 1];
      const df dx = fix_diff_full(ri.x, rj.x, S.sh, S.sl), dy = fix_diff_full(ri.y, rj.y, S.sh, S.sl),
               dz = fix_diff_full(ri.z, rj.z, S.sh, S.sl);
      const df r2 = met_norm2(dx, dy, dz);
      const int in_j = met_in(tj, r2.hi), in_i = same ? in_j : met_in(ti, r2.hi);
      if (in_j == 0 && in_i == 0) return;
      bool slow = in_j < 0 || in_i < 0 || !met_plain(r2.hi);
      df to_i = df_make(0.f, 0.f), to_j = to_i;
      if (!slow) {
        const Root r = met_dist(r2, nullptr);
        int l = 0;
        df f;
        if (in_j) {
          slow = !met_coord(tj, S.fv + tj.off, r, &l, &f);
          if (!slow) {
            to_i = met_poly(S.fv + tj.off, l, f);
            slow = to_i.hi < 0.f;
          }
          if (same) to_j = to_i;
        }
        if (!same && in_i && !slow) {
          if (!(in_j && ti.grid == tj.grid)) slow = !met_coord(ti, S.fv + ti.off, r, &l, &f);
          if (!slow) {
            to_j = met_poly(S.fv + ti.off, l, f);
            slow = to_j.hi < 0.f;
          }
        }
      }
      double dj;
      if (slow) {
        const int jj = S.at_list[j];
        double di;
        metal_density_slow(A, ti, tj, same, S.x[i] - S.x[jj], S.y[i] - S.y[jj], S.z[i] - S.z[jj], &di, &dj, &bad);
        df_split(di, &to_i.hi, &to_i.lo);
      } else {
        dj = flt_dbl(to_j.hi) + flt_dbl(to_j.lo);
      }
      dacc_add(rho, to_i);
      if (__double_as_longlong(dj) != 0) atomicAdd(&S.s0[j], dj);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rho = dacc_xor(rho, o);
    if (lane == 0) atomicAdd(&S.s0[p], dacc_value(rho));
  }
  if (bad) atomicOr(S.status, ST_METAL_TABLE);
}

// densities per sorted position onto the atoms
__global__ void k_metal_rho_fold(int natms, const DevScalars* sc, const int* __restrict__ at_list,
                                 const int* __restrict__ src, const double* __restrict__ s0, double* rho) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= sc->nlast) return;
  const double v = s0[p];
  if (__double_as_longlong(v) == 0) return;
  const int a = at_list[p];
  atomicAdd(&rho[a < natms ? a : src[a]], v);
}

// metal_ld_set_halo per sorted position: F'(rho) of the atom or of an image's source
__global__ void k_metal_fp(const DevScalars* sc, const int* __restrict__ src, const int* __restrict__ sorted_pos,
                           const double* __restrict__ rho, float2* __restrict__ fp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->nlast) return;
  float h, l;
  df_split(rho[src[i]], &h, &l);
  fp[sorted_pos[i]] = make_float2(h, l);
}

__global__ void __launch_bounds__(MET_NT, 3) k_metal_forces_sorted(MetSorted S, MetArgs A) {
  __shared__ MetTab tabs[MAX_TAB];
  __shared__ int queue[MET_NT / 32][32 * (MET_U + 1)];
  stage_tables(A, tabs);
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  dacc e_eng = {0.f, 0.f}, e_vir = {0.f, 0.f};
  bool bad = false;
  unsigned long long n_list = 0;
  int n_rc = 0;
  const int per = (S.natms + gridDim.x - 1) / gridDim.x;
  const int a_end = min(S.natms, (int)(blockIdx.x + 1) * per);
  for (int a = blockIdx.x * per + wq; a < a_end; a += MET_NT / 32) {
    const int p = S.loc_sp[a], i = S.at_list[p];
    const PosRec ri = S.rec[p];
    const int ai = ri.type;
    const float2 f2 = S.fp[p];
    const df fpi = df_make(f2.x, f2.y);
    const MetTab& ti = tabs[A.nkey + ai - 1];
    double fx = 0.0, fy = 0.0, fz = 0.0;
    n_list += (unsigned long long)S.list[(size_t)i * S.ld + 3];
    met_walk(S, i, S.xhs[p], queue[wq], [&](int j) {
      const PosRec rj = S.rec[j];
      const int aj = rj.type;
      const MetTab& tp = tabs[(ai > aj ? ai * (ai - 1) / 2 + aj : aj * (aj - 1) / 2 + ai) - 1];
      if (!tp.listed) return;  // keypot = -1
      const df dx = fix_diff_full(ri.x, rj.x, S.sh, S.sl), dy = fix_diff_full(ri.y, rj.y, S.sh, S.sl),
               dz = fix_diff_full(ri.z, rj.z, S.sh, S.sl);
      const df r2 = met_norm2(dx, dy, dz);
      if (r2.hi > S.f_rc_hi) return;
      const bool same = aj == ai;
      const MetTab& tj = tabs[A.nkey + aj - 1];
      const int in_p = met_in(tp, r2.hi), in_j = ti.n > 5 ? met_in(tj, r2.hi) : 0,
                in_i = same ? in_j : met_in(ti, r2.hi);
      bool slow = r2.hi > S.f_rc_lo || in_p < 0 || in_j < 0 || in_i < 0 || !met_plain(r2.hi);
      const float2 fq = S.fp[j];
      df gam = df_make(0.f, 0.f), num = gam, eng = gam;
      if (!slow) {
        df inv, f;
        const Root r = met_dist(r2, &inv);
        int l = 0, gl = -1;
        if (in_p) {
          slow = !met_coord(tp, S.fv + tp.off, r, &l, &f);
          gl = tp.grid;
          if (!slow) {
            num = met_poly(S.fd + tp.off, l, f);
            eng = met_poly(S.fv + tp.off, l, f);
          }
        }
        df g = df_make(0.f, 0.f);
        if (in_j && !slow) {
          if (tj.grid != gl) slow = !met_coord(tj, S.fv + tj.off, r, &l, &f);
          gl = tj.grid;
          if (!slow) {
            g = met_poly(S.fd + tj.off, l, f);
            // one table for both when the types are equal: g (F'_i + F'_j)
            num = df_fma(g, same ? df_add(fpi, df_make(fq.x, fq.y)) : fpi, num);
          }
        }
        if (!same && in_i && !slow) {
          if (ti.grid != gl) slow = !met_coord(ti, S.fv + ti.off, r, &l, &f);
          if (!slow) {
            g = met_poly(S.fd + ti.off, l, f);
            num = df_fma(g, df_make(fq.x, fq.y), num);
          }
        }
        gam = df_mul(num, inv);
        slow = slow || !(fabsf(num.hi) < 1e30f && fabsf(gam.hi) < 1e25f);
      }
      if (slow) {
        const int jj = S.at_list[j];
        double n64, g64, e64;
        const double x = S.x[i] - S.x[jj], y = S.y[i] - S.y[jj], z = S.z[i] - S.z[jj];
        if (!metal_force_slow(A, tp, ti, tj, same, x, y, z, S.rho[i],
                              (double)fq.x + (double)fq.y, &n64, &g64, &e64, &bad)) return;
        ++n_rc;
        // summed in FP64, whatever their size
        df_split(e64, &eng.hi, &eng.lo);
        df_split(n64, &num.hi, &num.lo);
        atomicAdd(&S.s0[p], g64 * x); atomicAdd(&S.s1[p], g64 * y); atomicAdd(&S.s2[p], g64 * z);
        atomicAdd(&S.s0[j], -g64 * x); atomicAdd(&S.s1[j], -g64 * y); atomicAdd(&S.s2[j], -g64 * z);
        dacc_add(e_eng, eng);
        dacc_add(e_vir, df_neg(num));
        return;
      }
      ++n_rc;
      dacc_add(e_eng, eng);
      dacc_add(e_vir, df_neg(num));
      // the products as an exact high part and the sum of the rest; summed in FP64 (the forces
      // of an atom's neighbours cancel to a small part of each)
      auto term = [&](df d, double& s, double* slot) {
        const df t = two_prod(gam.hi, d.hi);
        const double v = flt_dbl(t.hi) + flt_dbl(__fmaf_rn(gam.hi, d.lo, __fmaf_rn(gam.lo, d.hi, t.lo)));
        s += v;
        atomicAdd(&slot[j], -v);
      };
      term(dx, fx, S.s0);
      term(dy, fy, S.s1);
      term(dz, fz, S.s2);
    });
    {
      // reduce-scatter of three values over the warp: x in lane 0, y in 8, z in 16
      const bool up16 = lane & 16, up8 = lane & 8;
      double k0 = up16 ? fz : fx, k1 = up16 ? 0.0 : fy;
      k0 += __shfl_xor_sync(0xffffffffu, up16 ? fx : fz, 16);
      k1 += __shfl_xor_sync(0xffffffffu, up16 ? fy : 0.0, 16);
      double r = up8 ? k1 : k0;
      r += __shfl_xor_sync(0xffffffffu, up8 ? k0 : k1, 8);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
      if ((lane & 7) == 0 && lane < 24) atomicAdd(&(lane == 0 ? S.s0 : lane == 8 ? S.s1 : S.s2)[p], r);
    }
  }
  if (bad) atomicOr(S.status, ST_METAL_TABLE);
  if (S.cnt) {
    n_rc = warp_sumi(n_rc);
    if (lane == 0) {
      atomicAdd(&S.cnt[0], n_list);
      atomicAdd(&S.cnt[1], (unsigned long long)n_rc);
    }
  }
  dfr out[2] = {to_dfr(two_sum(e_eng.s, e_eng.c)), to_dfr(two_sum(e_vir.s, e_vir.c))};
  block_reduce_store<2>(out, S.blk);
  grid_finish<2>(S.blk, S.gs);
}

// stress (sum over slots of x (x) F, every halo image at its own position) and each slot's
// force onto its atom, as the pair kernels' k_slot_stress_fold
__global__ void k_metal_force_fold(int natms, const DevScalars* sc, const int* __restrict__ at_list,
                                   const int* __restrict__ src, const double* __restrict__ x,
                                   const double* __restrict__ y, const double* __restrict__ z,
                                   const double* __restrict__ s0, const double* __restrict__ s1,
                                   const double* __restrict__ s2, double* fx, double* fy, double* fz, double* blk, GridSum gs) {
  const int nlast = sc->nlast;
  double st[6] = {0, 0, 0, 0, 0, 0};
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nlast; p += gridDim.x * blockDim.x) {
    const double fa = s0[p], fb = s1[p], fc = s2[p];
    if ((__double_as_longlong(fa) | __double_as_longlong(fb) | __double_as_longlong(fc)) == 0) continue;
    const int a = at_list[p];
    const double xa = x[a], ya = y[a], za = z[a];
    st[0] = fma(xa, fa, st[0]); st[1] = fma(xa, fb, st[1]); st[2] = fma(xa, fc, st[2]);
    st[3] = fma(ya, fb, st[3]); st[4] = fma(ya, fc, st[4]); st[5] = fma(za, fc, st[5]);
    const int tgt = a < natms ? a : src[a];
    atomicAdd(&fx[tgt], fa);
    atomicAdd(&fy[tgt], fb);
    atomicAdd(&fz[tgt], fc);
  }
  block_reduce_store<6>(st, blk);
  grid_finish<6>(blk, gs);
}

// ------------------------------------------------------------------- host state
MetTab* d_tab = nullptr;
double* d_val = nullptr;
double* d_der = nullptr;
Coef* d_cv = nullptr;
Coef* d_cd = nullptr;
int* d_listed = nullptr;
double* d_rho = nullptr;
int n_key = 0, n_tab = 0, occ_dens = 0, occ_force = 0;
// sorted-position kernels
CoefF *d_fv = nullptr, *d_fd = nullptr;
float2* d_fp = nullptr;
double* d_slot = nullptr;     // 3 x mxatms: density or force sums per sorted position
int occ_dens_s = 0, occ_force_s = 0;
double max_rmax = 0.0;        // largest reach of a density table

// metal_table_derivatives: five-point derivative on the normalised neighbours
void table_derivatives(const std::vector<double>& buf, std::vector<double>& der) {
  // buf and der are Fortran-indexed (element 0 unused), buf(1..4) the header
  const double delmet = buf[4];
  const int v_end = (int)std::lround(buf[1]);
  const int i_start = 5 + 2, i_end = v_end - 2;
  for (int i = i_start; i <= i_end; ++i) {
    double aa0 = buf[i], f0, f1, f2, f3, f4;
    if (std::fabs(aa0) <= DBL_MIN) {
      f0 = f1 = f2 = f3 = f4 = 0.0;
    } else {
      f0 = buf[i - 2] / aa0;
      f1 = buf[i - 1] / aa0;
      f2 = 1.0;
      f3 = buf[i + 1] / aa0;
      f4 = buf[i + 2] / aa0;
    }
    const double d1y = (f1 - f0);
    const double d2y = (f2 - f1) - (f1 - f0);
    const double d3y = (f3 - f0) + 3.0 * (f1 - f2);
    const double d4y = (f4 - f3) + 3.0 * (f2 - f3) + 3.0 * (f2 - f1) + (f0 - f1);
    aa0 = aa0 / delmet;
    const double aa4 = d4y / 24.0;
    const double aa3 = (d3y + 12.0 * aa4) / 6.0;
    const double aa2 = (d2y + 6.0 * aa3 - 14.0 * aa4) / 2.0;
    const double aa1 = d1y + 3.0 * aa2 - 7.0 * aa3 + 15.0 * aa4;
    der[i] = aa1 * aa0;
    if (i == i_start) {
      der[i_start - 2] = (aa1 - 4.0 * aa2 + 12.0 * aa3 - 32.0 * aa4) * aa0;
      der[i_start - 1] = (aa1 - 2.0 * aa2 + 3.0 * aa3 - 4.0 * aa4) * aa0;
    } else if (i == i_end) {
      der[i_end + 1] = (aa1 + 2.0 * aa2 + 3.0 * aa3 + 4.0 * aa4) * aa0;
      der[i_end + 2] = (aa1 + 4.0 * aa2 + 12.0 * aa3 + 32.0 * aa4) * aa0;
    }
  }
}

}  // namespace

void metal_free() {
  void* p[] = {d_tab, d_val, d_der, d_cv, d_cd, d_listed, d_rho, d_fv, d_fd, d_fp, d_slot};
  for (void* q : p)
    if (q) cudaFree(q);
  d_tab = nullptr; d_val = nullptr; d_der = nullptr; d_cv = nullptr; d_cd = nullptr; d_listed = nullptr;
  d_rho = nullptr;
  d_fv = d_fd = nullptr; d_fp = nullptr; d_slot = nullptr;
  n_key = n_tab = 0;
  g.has_metal = false;
}

bool metal_active() { return g.has_metal; }

// kind[k] 1 = pair (types t1, t2), 2 = density (type t1), 3 = embedding (type t1);
// values in the units of the tables after the FIELD energy unit is applied
// (pair and embedding energies in internal units)
int metal_setup(int ntab, const int32_t* kind, const int32_t* t1, const int32_t* t2, const int32_t* ngrid,
                const double* start, const double* finish, const double* values, const int32_t* listed) {
  metal_free();
  max_rmax = 0.0;
  const int nt = g.p.ntypes;
  n_key = nt * (nt + 1) / 2;
  n_tab = n_key + 2 * nt;
  if (n_tab > 64) return GB_ERR_ARG;  // MAX_TAB tables (8 species)
  std::vector<MetTab> tab(n_tab);
  for (auto& t : tab) {
    t.n = 0; t.off = 0; t.r0 = t.rmax = t.dr = t.rdr = t.nr0rdr = 0.0; t.grid = -1; t.listed = 0;
    t.b_lo = t.b_hi = 0;
    t.f_lo = t.f_hi = -1.f;
    t.rdr_h = t.rdr_l = t.nr_h = t.nr_l = 0.f;
  }
  std::vector<double> val(1, 0.0), der(1, 0.0);
  size_t pos = 0;
  for (int k = 0; k < ntab; ++k) {
    const int ng = ngrid[k];
    if (ng < 5 || kind[k] < 1 || kind[k] > 3 || t1[k] < 1 || t1[k] > nt) return GB_ERR_ARG;
    int id;
    if (kind[k] == 1) {
      if (t2[k] < 1 || t2[k] > nt) return GB_ERR_ARG;
      const int a = std::max(t1[k], t2[k]), b = std::min(t1[k], t2[k]);
      id = a * (a - 1) / 2 + b - 1;
    } else {
      id = n_key + (kind[k] == 2 ? 0 : nt) + t1[k] - 1;
    }
    // metal_table_read: buffer(1) = ngrid + 4, buffer(4) = dr, buffer(2) = start - 5 dr, buffer(3) = finish
    std::vector<double> buf(ng + 5 + 1, 0.0), d(ng + 5 + 1, 0.0);
    buf[1] = (double)(ng + 4);
    buf[4] = (finish[k] - start[k]) / (double)(ng - 1);
    buf[2] = start[k] - 5.0 * buf[4];
    buf[3] = finish[k];
    for (int i = 0; i < ng; ++i) buf[5 + i] = values[pos + i];
    pos += ng;
    table_derivatives(buf, d);
    for (int i = 1; i <= 4; ++i) d[i] = kind[k] == 2 ? 0.0 : buf[i];  // header copies; zero for density
    if (kind[k] != 3)  // pair and density: column 2 holds -r d/dr
      for (int i = 5; i <= ng + 4; ++i) d[i] = -((double)i * buf[4] + buf[2]) * d[i];
    MetTab& t = tab[id];
    t.n = ng + 4;
    t.off = (int)val.size() - 1;
    t.r0 = buf[2];
    t.rmax = buf[3];
    t.dr = buf[4];
    t.rdr = 1.0 / buf[4];
    // entries 1..n+1 as the reference's arrays hold them: the header in 1..4 (an
    // interpolation at l = 5 reads entry 4), the values, then zeros
    for (int i = 1; i <= ng + 5; ++i) {
      val.push_back(buf[i]);
      der.push_back(d[i]);
    }
  }
  // quadratic coefficients per point (entry l = 5: the reference's linear form for ppp >= 0)
  std::vector<Coef> cv(val.size()), cd(der.size());
  for (auto& c : cv) c = Coef{0, 0, 0, 0};
  for (auto& c : cd) c = Coef{0, 0, 0, 0};
  for (int id = 0; id < n_tab; ++id) {
    const MetTab& t = tab[id];
    if (t.n == 0) continue;
    for (int l = 5; l <= t.n - 1; ++l) {
      for (int col = 0; col < 2; ++col) {
        const std::vector<double>& w = col ? der : val;
        const double v0 = w[t.off + l - 1], v1 = w[t.off + l], v2 = w[t.off + l + 1];
        Coef& c = col ? cd[t.off + l] : cv[t.off + l];
        if (l == 5) c = Coef{v1, v2 - v1, 0.0, 0.0};
        else c = Coef{v1, 0.5 * (v2 - v0), 0.5 * ((v2 - v1) - (v1 - v0)), 0.0};
      }
    }
  }
  // grid ids: tables on the same grid share one index computation
  int ngrid_ids = 0;
  for (int id = 0; id < n_tab; ++id) {
    if (tab[id].n == 0) continue;
    for (int o = 0; o < id && tab[id].grid < 0; ++o)
      if (tab[o].n == tab[id].n && tab[o].r0 == tab[id].r0 && tab[o].rdr == tab[id].rdr) tab[id].grid = tab[o].grid;
    if (tab[id].grid < 0) tab[id].grid = ngrid_ids++;
  }
  std::vector<int> lst(n_key, 0);
  for (int k = 0; k < n_key; ++k) lst[k] = listed ? listed[k] : 1;
  auto bits = [](double v) { long long b; std::memcpy(&b, &v, 8); return b; };
  for (int id = 0; id < n_tab; ++id) {
    MetTab& t = tab[id];
    if (id < n_key) t.listed = lst[id];
    if (t.n == 0) continue;
    t.nr0rdr = -t.r0 * t.rdr;
    t.b_lo = bits(t.rmax * t.rmax * (1.0 - 1e-12));
    t.b_hi = bits(t.rmax * t.rmax * (1.0 + 1e-12));
    if (id < n_key + nt) {  // tables of r
      t.f_lo = (float)(t.rmax * t.rmax * (1.0 - 1e-6));
      t.f_hi = (float)(t.rmax * t.rmax * (1.0 + 1e-6));
      df_split(t.rdr, &t.rdr_h, &t.rdr_l);
      df_split(t.nr0rdr, &t.nr_h, &t.nr_l);
      if (id >= n_key) max_rmax = std::max(max_rmax, t.rmax);
    }
  }
  auto split_coef = [](const std::vector<Coef>& c) {
    std::vector<CoefF> f(c.size());
    for (size_t k = 0; k < c.size(); ++k) {
      CoefF& o = f[k];
      df_split(c[k].c0, &o.c0h, &o.c0l);
      df_split(c[k].c1, &o.c1h, &o.c1l);
      df_split(c[k].c2, &o.c2h, &o.c2l);
      o.rh = o.rl = 0.f;
    }
    return f;
  };
  std::vector<CoefF> fv = split_coef(cv), fd = split_coef(cd);
  for (int id = 0; id < n_key + nt; ++id)
    for (int l = 5; l <= tab[id].n - 1; ++l) {
      CoefF& o = fv[tab[id].off + l];
      df_split(tab[id].r0 + (double)l / tab[id].rdr, &o.rh, &o.rl);
    }
  const size_t mx = std::max(g.mxatms, 1);
  GB_CUDA(cudaMalloc(&d_fv, sizeof(CoefF) * fv.size()));
  GB_CUDA(cudaMalloc(&d_fd, sizeof(CoefF) * fd.size()));
  GB_CUDA(cudaMemcpy(d_fv, fv.data(), sizeof(CoefF) * fv.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(d_fd, fd.data(), sizeof(CoefF) * fd.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMalloc(&d_fp, sizeof(float2) * mx));
  GB_CUDA(cudaMalloc(&d_slot, sizeof(double) * 3 * mx));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_dens_s, k_metal_density_sorted, MET_NT, 0));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_force_s, k_metal_forces_sorted, MET_NT, 0));
  GB_CUDA(cudaMalloc(&d_tab, sizeof(MetTab) * n_tab));
  GB_CUDA(cudaMalloc(&d_val, sizeof(double) * val.size()));
  GB_CUDA(cudaMalloc(&d_der, sizeof(double) * der.size()));
  GB_CUDA(cudaMalloc(&d_cv, sizeof(Coef) * cv.size()));
  GB_CUDA(cudaMalloc(&d_cd, sizeof(Coef) * cd.size()));
  GB_CUDA(cudaMemcpy(d_cv, cv.data(), sizeof(Coef) * cv.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(d_cd, cd.data(), sizeof(Coef) * cd.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMalloc(&d_listed, sizeof(int) * n_key));
  GB_CUDA(cudaMalloc(&d_rho, sizeof(double) * std::max(g.mxatms, 1)));
  GB_CUDA(cudaMemcpy(d_tab, tab.data(), sizeof(MetTab) * n_tab, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(d_val, val.data(), sizeof(double) * val.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(d_der, der.data(), sizeof(double) * der.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(d_listed, lst.data(), sizeof(int) * n_key, cudaMemcpyHostToDevice));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_dens, k_metal_density, 256, 0));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_force, k_metal_forces, 256, 0));
  g.has_metal = true;
  return GB_OK;
}

// The double-float kernels where the list pairs every halo entry with its backward copy;
// the FP64 form by instructions keeps the FP64 kernels.
static bool use_sorted_metal() { return g.spos_valid && g.use_sorted && !g.fp64_native; }

static void metal_forces_sorted(const MetArgs& A, unsigned long long* cnt) {
  cudaStream_t st = g.stream;
  const int T = 256, mx = g.mxatms, nbm = nblocks(mx, T);
  MetSorted S;
  S.natms = g.natms;
  S.at_list = g.at_list; S.loc_sp = g.loc_sp; S.list = g.list; S.spos = g.spos; S.ld = g.ld; S.ldt = g.ldt;
  S.xhs = g.xhs; S.rec = g.rec;
  S.sh = (float)(268435456.0 / g.pos_scale);
  S.sl = (float)(1.0 / g.pos_scale);
  S.x = g.x; S.y = g.y; S.z = g.z; S.rho = d_rho;
  S.fv = d_fv; S.fd = d_fd; S.fp = d_fp;
  S.s0 = d_slot; S.s1 = d_slot + mx; S.s2 = d_slot + 2 * (size_t)mx;
  S.status = &g.sc->status;
  const double rc2 = g.p.rcut * g.p.rcut;
  S.f_rc_lo = (float)(rc2 * (1.0 - 1e-6));
  S.f_rc_hi = (float)(rc2 * (1.0 + 1e-6));
  // the FP32 test of the high parts: coordinates below R have rounding errors below u
  auto pre = [](double r2) {
    const double u = std::ldexp(1.0, std::ilogb(1.5 * g.cell[0]) - 23), D = std::sqrt(r2) + 1.0;
    const double dlt = 2.0 * u + std::ldexp(1.0, -23) * (D + 2.0 * u);
    const double band = 4.0 * (2.0 * std::sqrt(3.0) * D * dlt + 3.0 * dlt * dlt) + 8.0 * std::ldexp(1.0, -23) * D * D;
    return std::nextafter((float)(r2 + band), 3.0e38f);
  };
  // short-lived CTAs of at most 16 atoms per warp, in runs of consecutive sorted positions;
  // a small system has at most one CTA per resident slot
  auto blocks = [&](int occ) {
    const int per = std::max(1, std::min(16, nblocks(g.natms, (MET_NT / 32) * std::max(1, occ) * g.nsm)));
    return std::max(1, nblocks(g.natms, (MET_NT / 32) * per));
  };
  const int nbd = blocks(occ_dens_s), nbf = blocks(occ_force_s), nbe = nblocks(g.natms, T),
            nbs = std::max(1, std::min(nbm, 4 * g.nsm));
  double* blk = gb_blkacc(nbe + 2 * nbf + 6 * nbs);
  double *blk2 = blk + nbe, *blk3 = blk2 + 2 * (size_t)nbf;
  S.blk = blk2;
  S.gs = gb_grid_sum(nbf, MET_NT, 2, &g.sc->acc[A_METAL]);
  const GridSum gss = gb_grid_sum(nbs, T, 6, &g.sc->acc[A_METAL + 2]);
  S.cnt = cnt;
  prof_begin(P_METAL_DENSITY);
  GB_CUDA(cudaMemsetAsync(d_slot, 0, sizeof(double) * (size_t)mx, st));
  GB_CUDA(cudaMemsetAsync(d_rho, 0, sizeof(double) * (size_t)g.natms, st));
  S.f_pre = pre(max_rmax * max_rmax * (1.0 + 1e-6));
  k_metal_density_sorted<<<nbd, MET_NT, 0, st>>>(S, A);
  GB_LAUNCHED();
  k_metal_rho_fold<<<nbm, T, 0, st>>>(g.natms, g.sc, g.at_list, g.src, d_slot, d_rho);
  GB_LAUNCHED();
  const GridSum gse = gb_grid_sum(nbe, T, 1, &g.sc->acc[A_METAL + 8]);
  k_metal_embed<<<nbe, T, 0, st>>>(g.natms, g.ltype, A, d_rho, blk, &g.sc->status, gse);
  GB_LAUNCHED();
  gb_grid_sum_done(gse, blk, nbe, 1);
  k_metal_fp<<<nbm, T, 0, st>>>(g.sc, g.src, g.sorted_pos, d_rho, d_fp);
  GB_LAUNCHED();
  prof_end(P_METAL_DENSITY);
  prof_begin(P_METAL_FORCES);
  GB_CUDA(cudaMemsetAsync(d_slot, 0, sizeof(double) * 3 * (size_t)mx, st));
  S.f_pre = pre(rc2 * (1.0 + 1e-6));
  k_metal_forces_sorted<<<nbf, MET_NT, 0, st>>>(S, A);
  GB_LAUNCHED();
  k_metal_force_fold<<<nbs, T, 0, st>>>(g.natms, g.sc, g.at_list, g.src, g.x, g.y, g.z, S.s0, S.s1, S.s2, g.fx, g.fy,
                                        g.fz, blk3, gss);
  GB_LAUNCHED();
  gb_grid_sum_done(S.gs, blk2, nbf, 2);
  gb_grid_sum_done(gss, blk3, nbs, 6);
  prof_end(P_METAL_FORCES);
}

static void metal_forces_fp64(const MetArgs& A, unsigned long long* cnt) {
  cudaStream_t st = g.stream;
  const int T = 256;
  GB_CUDA(cudaMemsetAsync(d_rho, 0, sizeof(double) * g.mxatms, st));
  prof_begin(P_METAL_DENSITY);
  int nb = std::max(1, std::min(nblocks((long long)g.mxatms * 32, T), occ_dens * g.nsm));
  k_metal_density<<<nb, T, 0, st>>>(g.natms, g.sc, g.at_list, g.list, g.ld, g.x, g.y, g.z, g.ltype, g.ltg, g.src, A,
                                    d_rho, &g.sc->status);
  GB_LAUNCHED();
  const int nbe = nblocks(g.natms, T);
  double* blk = gb_blkacc(std::max(nbe, 1) + MACC * std::max(1, occ_force * g.nsm));
  const GridSum gse = gb_grid_sum(nbe, T, 1, &g.sc->acc[A_METAL + 8]);
  k_metal_embed<<<nbe, T, 0, st>>>(g.natms, g.ltype, A, d_rho, blk, &g.sc->status, gse);
  GB_LAUNCHED();
  gb_grid_sum_done(gse, blk, nbe, 1);
  k_metal_halo<<<nblocks(std::max(g.mxatms - g.natms, 1), T), T, 0, st>>>(g.natms, g.sc, g.src, d_rho);
  GB_LAUNCHED();
  prof_end(P_METAL_DENSITY);
  prof_begin(P_METAL_FORCES);
  nb = std::max(1, std::min(nblocks((long long)g.mxatms * 32, T), occ_force * g.nsm));
  double* blk2 = blk + std::max(nbe, 1);
  k_metal_forces<<<nb, T, 0, st>>>(g.natms, g.sc, g.at_list, g.list, g.ld, g.x, g.y, g.z, g.ltype, g.ltg, g.src, A,
                                   d_rho, g.fx, g.fy, g.fz, blk2, &g.sc->status, cnt);
  GB_LAUNCHED();
  gb_reduce_blocks(blk2, nb, MACC, &g.sc->acc[A_METAL]);
  prof_end(P_METAL_FORCES);
}

// both passes; adds forces into g.fx/fy/fz and stress into stress9; returns
// engmet, virmet (pair part) and engden, virden (embedding part) in e4
void metal_forces(double* e4, double* stress9) {
  MetArgs A;
  A.tab = d_tab; A.v = d_val; A.d = d_der; A.cv = d_cv; A.cd = d_cd; A.listed = d_listed;
  A.nkey = n_key; A.ntypes = g.p.ntypes; A.ntab = n_tab; A.rcut = g.p.rcut;
  {
    const double rc2 = g.p.rcut * g.p.rcut, lo = rc2 * (1.0 - 1e-12), hi = rc2 * (1.0 + 1e-12);
    std::memcpy(&A.b_rc_lo, &lo, 8);
    std::memcpy(&A.b_rc_hi, &hi, 8);
  }
  unsigned long long* cnt = nullptr;
  if (!g.has_coul && !g.has_vdw) {  // the pair kernel did not run: count here
    GB_CUDA(cudaMemsetAsync(&g.sc->npairs_list, 0, 2 * sizeof(unsigned long long), g.stream));
    cnt = &g.sc->npairs_list;
  }
  if (use_sorted_metal()) metal_forces_sorted(A, cnt);
  else metal_forces_fp64(A, cnt);
  if (g.defer_scalars) return;  // the MD loop reads the sums and the status
  gb_sync_scalars();
  if (g.hsc->status & ST_METAL_DENSITY) throw (int)GB_ERR_METAL_DENSITY;
  if (g.hsc->status & ST_METAL_TABLE) throw (int)GB_ERR_METAL_TABLE;
  metal_scalars(g.hsc, e4, stress9);
}

// engmet, virmet, engden, virden and the stress from the device sums
void metal_scalars(const DevScalars* h, double* e4, double* stress9) {
  const double* a = &h->acc[A_METAL];
  e4[0] = a[0];
  e4[1] = a[1];
  e4[2] = a[8];
  e4[3] = 0.0;  // virden: no long-range density correction for tabulated EAM
  const double s[9] = {a[2], a[3], a[4], a[3], a[5], a[6], a[4], a[6], a[7]};
  for (int k = 0; k < 9; ++k) stress9[k] += s[k];
}

void metal_rho(double* out, int n) {
  GB_CUDA(cudaMemcpy(out, d_rho, sizeof(double) * std::min(n, g.natms), cudaMemcpyDeviceToHost));
}
