// gb_list.cu - halo images and the link-cell Verlet list on the device.
//
// Follows, in serial (one-domain) semantics:
//   pbcshift            source/numerics.F90:1851-1907
//   set_halo_particles  source/halo.F90:153-356 (+ export_atomic_data deport_data.F90:1673-1900)
//   refresh_halo_positions source/halo.F90:47-114
//   link_cell_pairs     source/neighbours.F90:356-1414
// Every quantity that decides membership (cell index, halo flag, rsq <= rcsq)
// is computed with explicitly rounded FP64 operations (no FMA contraction) in
// the reference's operation order, so the pair set is bit-identical to the
// FP64 oracle.  Distance tests run first in FP32 with a proven error margin;
// only candidates inside the margin band are re-tested in exact FP64.
#include <cfloat>
#include <cmath>
#include <cstring>

#include "gb_common.cuh"

namespace {

constexpr int MAX_SBC = 1024;  // semi-ball offsets capacity

// for the list kernels: per semi-ball cell its linear offset and
// (nix + 64) | (niy + 64) << 8 | (niz + 64) << 16 | nir << 24; and, as the semi-ball cells in
// the reference order form, tile row (dy, dz) by tile row, runs of consecutive cells along x
// (contiguous sorted positions), per run with one nir flag the linear offsets of its first
// and last cell, its row and the flag
__device__ int2 d_sbc[MAX_SBC];
__device__ int4 d_seg[MAX_SBC];

struct HaloGeom {
  double rc[9];
  double ecw[3], cw[3];
};

struct CellGeom {
  double rc[9];
  double xdc, ydc, zdc;
  int nlp, nlx, nly, nlz, NX, NY, NZ;
  double rcsq;
  float rcsq_lo, rcsq_hi;
  double half_plus;
};

HaloGeom h_halo;
CellGeom h_cg;
double h_add[6][3];  // export add vectors for mdir -1,1,-2,2,-3,3
int h_halo_blocks = 0;  // blocks of k_halo_count and k_halo_write (GB_HALO_BLOCKS; 0: by size)

// ---------------------------------------------------------------- kernels
// The reduced coordinate rc(d) x + rc(d+3) y + rc(d+6) z of the reference: gb_init takes
// cubic cells only, whose off-diagonal terms are zero and add nothing.
__device__ __forceinline__ double red_coord(const double* rc, int d, double xd) { return mul_rn(rc[4 * d], xd); }

// an integer that orders as the double does (an FP64 comparison takes the FP64 unit)
__device__ __forceinline__ long long ordered(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ bool is_nan(double v) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

// relocate_particles (pbcshift, numerics.F90:1886-1930), set_halo_particles (halo.F90:153-356)
// and vnl_set_check (neighbours.F90:305-343) in two launches.  The reference's images come
// from six ordered exports (-x, +x, -y, +y, -z, +z), each a stable compaction of the atoms
// and images so far, and an image is not exported again along its own dimension.  So an
// image is an atom and a class, ox + 3 oy + 9 oz with o = 0 (not exported), 1 (-) or 2 (+)
// per dimension, an atom has the classes that its three 2-bit codes allow, and the images
// stand in the order of their class, then of their atom.  One launch wraps the atoms and counts
// each class per block, the next sums the counts before its own and writes the images.
// As six compactions between the barriers of one cooperative kernel it took 0.055 ms at
// 4,096 atoms; the two launches take 0.016, latency of the dependent loads.
constexpr int HALO_NT = 256, HALO_NC = 27;
struct HaloArgs {
  int n, mxatms;
  double *x, *y, *z, *xb, *yb, *zb;
  double a[3], c[3], half_minus;   // 1/L and L per dimension
  HaloGeom hg;
  double add[6][3];
  int *code, *src, *shcode, *ltg, *ltype, *lfrzn;
  double *chge, *weight;
  int* cnt;                        // [HALO_NC][blocks]
  DevScalars* sc;
};

// code: the 2-bit codes of x, y, z (bit 0: exported by -, bit 1: by +)
__device__ __forceinline__ bool has_class(int code, int c) {
  const int ox = c % 3, oy = (c / 3) % 3, oz = c / 9;
  return (ox == 0 || (code >> (ox - 1)) & 1) && (oy == 0 || (code >> (oy + 1)) & 1) &&
         (oz == 0 || (code >> (oz + 3)) & 1);
}

__device__ __forceinline__ double wrap1(double x, double a, double c, double half_minus) {
  double s = mul_rn(a, x);
  // |s| below half_minus (its bits): round(s) = 0
  if ((__double_as_longlong(s) & 0x7fffffffffffffffll) >= __double_as_longlong(half_minus)) {
    s = sub_rn(s, round(s));
    if (s >= half_minus) s = -s;
  }
  return mul_rn(c, s);
}

__global__ void __launch_bounds__(HALO_NT) k_halo_count(HaloArgs A) {
  __shared__ int s_cnt[HALO_NC];
  const int lane = threadIdx.x & 31;
  long long lo_b[3], hi_b[3];
  for (int d = 0; d < 3; ++d) { lo_b[d] = ordered(A.hg.ecw[d]); hi_b[d] = ordered(A.hg.cw[d]); }
  if (threadIdx.x < HALO_NC) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int per = (A.n + gridDim.x - 1) / gridDim.x;
  const int lo = min(A.n, (int)blockIdx.x * per), hi = min(A.n, lo + per);
  int cnt = 0;  // lane c: class c
  for (int i0 = lo; i0 < hi; i0 += HALO_NT) {
    const int i = i0 + threadIdx.x;
    int v = 0;
    if (i < hi) {
      const double x = wrap1(A.x[i], A.a[0], A.c[0], A.half_minus), y = wrap1(A.y[i], A.a[1], A.c[1], A.half_minus),
                   z = wrap1(A.z[i], A.a[2], A.c[2], A.half_minus);
      A.x[i] = x; A.y[i] = y; A.z[i] = z;
      A.xb[i] = x; A.yb[i] = y; A.zb[i] = z;
      const double red[3] = {red_coord(A.hg.rc, 0, x), red_coord(A.hg.rc, 1, y), red_coord(A.hg.rc, 2, z)};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const long long o = ordered(red[d]);
        const int w = (o <= lo_b[d] ? 1 : 0) | (o >= hi_b[d] ? 2 : 0);
        if (!is_nan(red[d])) v |= w << (2 * d);  // (a NaN compares false: not exported)
      }
      A.code[i] = v;
      A.src[i] = i;
      A.shcode[i] = 13;
    }
    if (!__any_sync(0xffffffffu, v != 0)) continue;
#pragma unroll
    for (int c = 1; c < HALO_NC; ++c) {
      const int k = __popc(__ballot_sync(0xffffffffu, has_class(v, c)));
      if (lane == c) cnt += k;
    }
  }
  if (lane < HALO_NC && cnt) atomicAdd(&s_cnt[lane], cnt);
  __syncthreads();
  if (threadIdx.x < HALO_NC) A.cnt[threadIdx.x * gridDim.x + blockIdx.x] = s_cnt[threadIdx.x];
}

__global__ void __launch_bounds__(HALO_NT) k_halo_write(HaloArgs A) {
  constexpr int NW = HALO_NT / 32;
  __shared__ int s_before[HALO_NC], s_all[HALO_NC], s_w[NW][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = gridDim.x;
  for (int c = 1 + wid; c < HALO_NC; c += NW) {  // images of the class before this block's, and all of them
    int before = 0, all = 0;
    for (int b = lane; b < nb; b += 32) {
      const int k = A.cnt[c * nb + b];
      all += k;
      before += b < (int)blockIdx.x ? k : 0;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    all = __reduce_add_sync(0xffffffffu, all);
    if (lane == 0) { s_before[c] = before; s_all[c] = all; }
  }
  __syncthreads();
  const bool cls = lane >= 1 && lane < HALO_NC;
  const int all = cls ? s_all[lane] : 0;
  int inc = all;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  int base = A.n + (inc - all) + (cls ? s_before[lane] : 0);  // lane c: place of the next image of class c
  if (blockIdx.x == 0 && threadIdx.x == 31) {  // images beyond mxatms are neither written nor counted
    const int nlast = min(A.n + inc, A.mxatms);
    A.sc->nlast = nlast;
    A.sc->nlast_prev = nlast;
    if (A.n + inc > A.mxatms) A.sc->status |= ST_HALO_OVERFLOW;
  }
  const int per = (A.n + nb - 1) / nb;
  const int lo = min(A.n, (int)blockIdx.x * per), hi = min(A.n, lo + per);
  for (int i0 = lo; i0 < hi; i0 += HALO_NT) {
    const int i = i0 + threadIdx.x;
    const int v = i < hi ? A.code[i] : 0;
    unsigned present = 0;  // classes that an atom of the warp has
    int cnt = 0;
    if (__any_sync(0xffffffffu, v != 0)) {
#pragma unroll
      for (int c = 1; c < HALO_NC; ++c) {
        const int k = __popc(__ballot_sync(0xffffffffu, has_class(v, c)));
        if (lane == c) cnt = k;
      }
      present = __ballot_sync(0xffffffffu, cnt != 0);
    }
    s_w[wid][lane] = cnt;
    __syncthreads();
    int pre = base;
    for (int w = 0; w < NW; ++w) {
      const int k = s_w[w][lane];
      if (w < wid) pre += k;
      base += k;
    }
    __syncthreads();
    if (!present) continue;
    double x = 0.0, y = 0.0, z = 0.0, q = 0.0, wt = 0.0;
    int tg = 0, ty = 0, fr = 0;
    if (v) {
      x = A.x[i]; y = A.y[i]; z = A.z[i];
      q = A.chge[i]; wt = A.weight[i];
      tg = A.ltg[i]; ty = A.ltype[i]; fr = A.lfrzn[i];
    }
    for (unsigned m = present; m; m &= m - 1) {
      const int c = __ffs((int)m) - 1;
      const bool on = has_class(v, c);
      const unsigned bal = __ballot_sync(0xffffffffu, on);
      const int dst = __shfl_sync(0xffffffffu, pre, c) + __popc(bal & ((1u << lane) - 1u));
      if (!on || dst >= A.mxatms) continue;
      const int o[3] = {c % 3, (c / 3) % 3, c / 9};
      double xi = x, yi = y, zi = z;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (o[d] == 0) continue;
        const double* ad = A.add[2 * d + o[d] - 1];
        xi = add_rn(xi, ad[0]); yi = add_rn(yi, ad[1]); zi = add_rn(zi, ad[2]);
      }
      A.x[dst] = xi; A.y[dst] = yi; A.z[dst] = zi;
      A.src[dst] = i;
      A.shcode[dst] = 13 + (o[0] == 0 ? 0 : o[0] == 1 ? 1 : -1) + (o[1] == 0 ? 0 : o[1] == 1 ? 3 : -3) +
                      (o[2] == 0 ? 0 : o[2] == 1 ? 9 : -9);
      A.ltg[dst] = tg;
      A.ltype[dst] = ty;
      A.chge[dst] = q;
      A.weight[dst] = wt;
      A.lfrzn[dst] = fr;
    }
  }
}

// The list's kernels do nothing after a halo overflow: the last list stays (the MD loop enqueues
// them behind the halo without waiting for its status).
__device__ __forceinline__ bool halo_cut(const DevScalars* sc) { return sc->status & ST_HALO_OVERFLOW; }

// Exclusive scan of the cells' counts (block 0: all cells, into start; block 1: the domain's
// cells, which hold the local atoms, into lstart) and the zeros that the list's kernels
// count from.  A warp takes 1/32 of the cells, 32 at a time.
__global__ void __launch_bounds__(1024) k_cell_scan(int n, CellGeom cg, const int* __restrict__ count, int* start,
                                                    int* lstart, DevScalars* sc) {
  __shared__ int s_w[32];
  if (halo_cut(sc)) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->ibig = 0;
    sc->tile_over = sc->halo_fwd = sc->halo_bwd = 0;
  }
  const bool local = blockIdx.x == 1;
  const int per = ((n + 1023) / 1024) * 32, lo = min(n, wid * per), hi = min(n, lo + per);
  auto get = [&](int c) {
    if (c >= hi) return 0;
    if (local) {
      const int a = c - 1, iz = a / (cg.NX * cg.NY), iy = a / cg.NX - cg.NY * iz, ix = a % cg.NX;
      if (a < 0 || ix < cg.nlp || ix >= cg.nlp + cg.nlx || iy < cg.nlp || iy >= cg.nlp + cg.nly || iz < cg.nlp ||
          iz >= cg.nlp + cg.nlz)
        return 0;
    }
    return count[c];
  };
  int t = 0;
#pragma unroll 4
  for (int b = lo; b < hi; b += 32) t += get(b + lane);
  t = __reduce_add_sync(0xffffffffu, t);
  if (lane == 0) s_w[wid] = t;
  __syncthreads();
  int run = __reduce_add_sync(0xffffffffu, lane < wid ? s_w[lane] : 0);
  int* out = local ? lstart : start;
#pragma unroll 4
  for (int b = lo; b < hi; b += 32) {
    const int k = get(b + lane);
    int inc = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (b + lane < hi) out[b + lane] = run + inc - k;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
}

// refresh_halo_positions: the same export chain applied to the source position
__global__ void k_halo_refresh(int natms, const DevScalars* sc, const int* src, const int* shcode, double* x,
                               double* y, double* z, const double* adds /*6x3*/) {
  int i = natms + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->nlast) return;
  int s = src[i], c = shcode[i];
  int sx = c % 3 - 1, sy = (c / 3) % 3 - 1, sz = c / 9 - 1;
  double xx = x[s], yy = y[s], zz = z[s];
  // adds[0..2] is the -x export (image at +L), adds[3..5] the +x export (image at -L), etc.
  if (sx != 0) { const double* a = adds + 3 * (sx > 0 ? 0 : 1); xx = add_rn(xx, a[0]); yy = add_rn(yy, a[1]); zz = add_rn(zz, a[2]); }
  if (sy != 0) { const double* a = adds + 3 * (sy > 0 ? 2 : 3); xx = add_rn(xx, a[0]); yy = add_rn(yy, a[1]); zz = add_rn(zz, a[2]); }
  if (sz != 0) { const double* a = adds + 3 * (sz > 0 ? 4 : 5); xx = add_rn(xx, a[0]); yy = add_rn(yy, a[1]); zz = add_rn(zz, a[2]); }
  x[i] = xx; y[i] = yy; z[i] = zz;
}

// ----------------------------------------------------------------- binning
__global__ void k_bin(int natms, const DevScalars* sc, const double* x, const double* y, const double* z,
                      CellGeom cg, int* which_cell, int* count) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nlast = sc->nlast;
  if (i >= nlast || halo_cut(sc)) return;
  const double xx = red_coord(cg.rc, 0, x[i]);
  const double yy = red_coord(cg.rc, 1, y[i]);
  const double zz = red_coord(cg.rc, 2, z[i]);
  const int nlp = cg.nlp, jx0 = nlp, jy0 = nlp, jz0 = nlp;
  const int nlx0e = nlp - 1, nly0e = nlp - 1, nlz0e = nlp - 1;
  const int nlx1s = cg.nlx + nlp, nly1s = cg.nly + nlp, nlz1s = cg.nlz + nlp;
  const int nlx1e = cg.nlx + 2 * nlp - 1, nly1e = cg.nly + 2 * nlp - 1, nlz1e = cg.nlz + 2 * nlp - 1;
  int icell;
  if (i < natms) {
    int ix = __double2int_rz(mul_rn(cg.xdc, add_rn(xx, 0.5))) + jx0;
    int iy = __double2int_rz(mul_rn(cg.ydc, add_rn(yy, 0.5))) + jy0;
    int iz = __double2int_rz(mul_rn(cg.zdc, add_rn(zz, 0.5))) + jz0;
    ix = max(min(ix, nlx1s - 1), nlx0e + 1);
    iy = max(min(iy, nly1s - 1), nly0e + 1);
    iz = max(min(iz, nlz1s - 1), nlz0e + 1);
    icell = 1 + ix + cg.NX * (iy + cg.NY * iz);
  } else {
    double dx, dy, dz;
    int ix, iy, iz;
    if (xx > -cg.half_plus) { dx = mul_rn(cg.xdc, add_rn(xx, 0.5)); ix = __double2int_rz(dx) + jx0; }
    else { dx = mul_rn(cg.xdc, fabs(add_rn(xx, 0.5))); ix = -__double2int_rz(dx) + jx0 - 1; }
    if (yy > -cg.half_plus) { dy = mul_rn(cg.ydc, add_rn(yy, 0.5)); iy = __double2int_rz(dy) + jy0; }
    else { dy = mul_rn(cg.ydc, fabs(add_rn(yy, 0.5))); iy = -__double2int_rz(dy) + jy0 - 1; }
    if (zz > -cg.half_plus) { dz = mul_rn(cg.zdc, add_rn(zz, 0.5)); iz = __double2int_rz(dz) + jz0; }
    else { dz = mul_rn(cg.zdc, fabs(add_rn(zz, 0.5))); iz = -__double2int_rz(dz) + jz0 - 1; }
    if (ix >= 0 && iy >= 0 && iz >= 0) {
      bool lx0 = ix > nlx0e, lx1 = ix < nlx1s, ly0 = iy > nly0e, ly1 = iy < nly1s, lz0 = iz > nlz0e, lz1 = iz < nlz1s;
      if ((lx0 && lx1) && (ly0 && ly1) && (lz0 && lz1)) {
        double x0 = fabs(sub_rn(dx, 0.0)), x1 = fabs(sub_rn(dx, (double)cg.nlx));
        dx = fmin(x0, x1);
        double y0 = fabs(sub_rn(dy, 0.0)), y1 = fabs(sub_rn(dy, (double)cg.nly));
        dy = fmin(y0, y1);
        double z0 = fabs(sub_rn(dz, 0.0)), z1 = fabs(sub_rn(dz, (double)cg.nlz));
        dz = fmin(z0, z1);
        if (dx <= dy && dx <= dz) {
          ix = x0 < x1 ? nlx0e : nlx1s;
          if (fabs(sub_rn(dx, dy)) < DBL_EPSILON) iy = y0 < y1 ? nly0e : nly1s;
          if (fabs(sub_rn(dx, dz)) < DBL_EPSILON) iz = z0 < z1 ? nlz0e : nlz1s;
        } else if (dy <= dx && dy <= dz) {
          iy = y0 < y1 ? nly0e : nly1s;
          if (fabs(sub_rn(dy, dz)) < DBL_EPSILON) iz = z0 < z1 ? nlz0e : nlz1s;
        } else {
          iz = z0 < z1 ? nlz0e : nlz1s;
        }
      }
      bool out = ix < 0 || ix > nlx1e || iy < 0 || iy > nly1e || iz < 0 || iz > nlz1e;
      icell = out ? 0 : 1 + ix + cg.NX * (iy + cg.NY * iz);
    } else {
      icell = 0;
    }
  }
  which_cell[i] = icell;
  atomicAdd(&count[icell], 1);
}

// (counts the cells back down to zero, for the next build)
__global__ void k_cell_scatter(const DevScalars* sc, const int* which_cell, const int* start, int* count,
                               int* tmp) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->nlast || halo_cut(sc)) return;
  int c = which_cell[i];
  int slot = atomicSub(&count[c], 1) - 1;
  tmp[start[c] + slot] = i;
}

__device__ __forceinline__ void tile_row(int t, const TilePlan& tp, const CellGeom& cg, const int* __restrict__ start,
                                         int* __restrict__ tile_rows, int* __restrict__ tile_info, int cap,
                                         DevScalars* sc);

// Stable order inside each cell (ascending atom index, as the reference's
// counting sort over i = 1..nlast): rank of each member by counting.  A local atom's
// sorted position goes to loc_sp too, in sorted order (a domain cell holds local atoms only).
// The blocks after the cells' take the residual halo cell (one warp took 0.065 ms for it
// where it is large: 6,591-atom water; 0.006 so), the blocks after those the tiles' rows.
constexpr int SORT_NT = 256, RESID_BLOCKS = 32;
__global__ void __launch_bounds__(SORT_NT) k_cell_sort(int ncells_p1, int natms, const int* start, const int* lstart,
                                                       const int* tmp, int* at_list, int* sorted_pos, int* loc_sp,
                                                       const double* x, const double* y, const double* z,
                                                       double4_32a* xs, float4* xsf, TilePlan tp, CellGeom cg,
                                                       int* tile_rows, int* tile_info, int cap, DevScalars* sc) {
  if (halo_cut(sc)) return;
  const int ncb = (ncells_p1 + SORT_NT / 32 - 1) / (SORT_NT / 32);
  if ((int)blockIdx.x >= ncb) {
    const int rb = blockIdx.x - ncb;
    if (rb >= RESID_BLOCKS) {
      tile_row((rb - RESID_BLOCKS) * SORT_NT + threadIdx.x, tp, cg, start, tile_rows, tile_info, cap, sc);
      return;
    }
    // residual halo cell: never a neighbour cell, order irrelevant
    const int s = start[0], e = start[1];
    for (int a = s + rb * SORT_NT + threadIdx.x; a < e; a += RESID_BLOCKS * SORT_NT) {
      const int v = tmp[a];
      at_list[a] = v;
      sorted_pos[v] = a;
      const double xv = x[v], yv = y[v], zv = z[v];
      xs[a] = make_double4_32a(xv, yv, zv, 0.0);
      xsf[a] = make_float4((float)xv, (float)yv, (float)zv, __int_as_float(v));
    }
    return;
  }
  const int cell = (blockIdx.x * SORT_NT + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (cell >= ncells_p1 || cell == 0) return;
  const int s = start[cell], n = start[cell + 1] - s, ls = lstart[cell];
  for (int a = lane; a < n; a += 32) {
    int v = tmp[s + a];
    int r = 0;
    for (int b = 0; b < n; ++b) r += (tmp[s + b] < v);
    int pos = s + r;
    at_list[pos] = v;
    sorted_pos[v] = pos;
    if (v < natms) loc_sp[ls + r] = pos;
    double xv = x[v], yv = y[v], zv = z[v];
    xs[pos] = make_double4_32a(xv, yv, zv, 0.0);
    xsf[pos] = make_float4((float)xv, (float)yv, (float)zv, __int_as_float(v));
  }
}

// Row tables of the cell tiles: per row (dy, dz) the first sorted position of its x run
// of cells and its slot base in the tile's staged set; per tile the staged total and the
// sorted-position range of its own (i) atoms.  Tiles above the capacity are counted: the
// list then comes from k_list_lanes.
__device__ __forceinline__ void tile_row(int t, const TilePlan& tp, const CellGeom& cg, const int* __restrict__ start,
                                         int* __restrict__ tile_rows, int* __restrict__ tile_info, int cap,
                                         DevScalars* sc) {
  if (t >= tp.ntiles) return;
  const int tx = t % tp.ntx, ty = (t / tp.ntx) % tp.nty, tz = t / (tp.ntx * tp.nty);
  const int nlp = cg.nlp;
  const int x0 = nlp + tx * tp.m, x1 = min(x0 + tp.m, nlp + cg.nlx);  // own cells [x0, x1)
  const int y = nlp + ty, z = nlp + tz;
  int base = 0;
  for (int r = 0; r < tp.nrows; ++r) {
    const int plane = cg.NX * ((y + tp.dy[r]) + cg.NY * (z + tp.dz[r]));
    const int clo = 1 + (x0 + tp.dxlo[r]) + plane, chi = 1 + (x1 - 1 + tp.dxhi[r]) + plane;
    const int f = start[clo], e = start[chi + 1];
    tile_rows[2 * (t * tp.nrows + r)] = f;
    tile_rows[2 * (t * tp.nrows + r) + 1] = base;
    base += e - f;
  }
  const int plane = cg.NX * (y + cg.NY * z);
  tile_info[4 * t] = base;
  tile_info[4 * t + 1] = start[1 + x0 + plane];
  tile_info[4 * t + 2] = start[1 + (x1 - 1) + plane + 1];
  tile_info[4 * t + 3] = 0;
  if (base > cap) atomicAdd(&sc->tile_over, 1);
}

// Half-shell Verlet list (neighbours.F90:876-1184) of a small system, several CTAs per cell tile: the tile's
// forward half shell (FP32 positions and atom ids) is staged in shared memory and one
// warp per local atom walks it in the reference order (semi-ball cell by cell, each
// cell's members in ascending order), one run of consecutive cells at a time, with
// ballot compaction.  Beside list(k, i) the kernel writes spos(k, i): the partner's
// sorted position, or -1 for the entries of the backward halo pass (pass 2), whose
// pairs the partner atom's forward pass also lists, so that the pair kernels evaluate
// each pair once, from its forward copy.  Bound by issue in pass 1 and by the latency of
// its loads in pass 2, whose cells are read from global memory: 32 cells' bounds are loaded
// at once and their members taken as one sequence (0.048 ms for 1,536 atoms, where seven CTAs
// share a tile; k_list_lanes takes 0.061 there and 0.059 instead of 0.062 at 4,096).
__global__ void __launch_bounds__(256) k_list_tiles(int natms, CellGeom cg, TilePlan tp, int nsbcll, int nseg,
                                                    int cap,
                                                    const int* __restrict__ tile_rows, const int* __restrict__ tile_info,
                                                    const int* __restrict__ at_list, const int* __restrict__ which_cell,
                                                    const int* __restrict__ start, const double4_32a* __restrict__ xs,
                                                    const float4* __restrict__ xsf, int* list, int ld, int* spos,
                                                    int ldt, int max_list, DevScalars* sc) {
  extern __shared__ float4 s_x[];  // cap staged FP32 positions, then cap atom ids
  int* s_at = reinterpret_cast<int*>(s_x + cap);
  __shared__ int s_first[TILE_MAX_ROWS], s_base[TILE_MAX_ROWS + 1];
  const int t = blockIdx.x;
  const int nst = tile_info[4 * t];
  if (nst > cap || halo_cut(sc)) return;  // k_list_lanes then builds the list (uniform over the CTA)
  const int nrows = tp.nrows;
  if (threadIdx.x < nrows) {
    s_first[threadIdx.x] = tile_rows[2 * (t * nrows + threadIdx.x)];
    s_base[threadIdx.x] = tile_rows[2 * (t * nrows + threadIdx.x) + 1];
  }
  if (threadIdx.x == 0) s_base[nrows] = nst;
  __syncthreads();
  for (int r = 0; r < nrows; ++r) {
    const int b = s_base[r], cnt = s_base[r + 1] - b, f = s_first[r];
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
      s_x[b + e] = xsf[f + e];
      s_at[b + e] = at_list[f + e];
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int ip0 = tile_info[4 * t + 1], ip1 = tile_info[4 * t + 2];
  const int nlp = cg.nlp;
  const int nlx0e = nlp - 1, nly0e = nlp - 1, nlz0e = nlp - 1;
  const int nlx1s = cg.nlx + nlp, nly1s = cg.nly + nlp, nlz1s = cg.nlz + nlp;
  int ncand64 = 0, nfwd = 0, nbwd = 0;
  for (int p = ip0 + warp + nw * blockIdx.y; p < ip1; p += nw * gridDim.y) {
    const int i0s = s_base[tp.r00] - s_first[tp.r00];
    const int i = s_at[p + i0s];
    const int ic = which_cell[i];
    const int icm = ic - 1;
    const int ix = icm % cg.NX;
    const int iz = icm / (cg.NX * cg.NY);
    const int iy = icm / cg.NX - cg.NY * iz;
    const double4_32a xi = xs[p];
    const float4 xif = s_x[p + i0s];
    int* li = list + (size_t)i * ld + 3;  // li[k] == list(k, i)
    int* si = spos + (size_t)i * ldt;
    int count = 0;
    int l_s0 = 0, l_e = 0, l_sl = 0;
    unsigned l_nir = 0;
    // pass 1: the forward half shell, all of it staged, one run of cells at a time
    // (the bounds of 32 runs are loaded at once, a lane each)
    for (int q = 0; q < nseg; ++q) {
      if ((q & 31) == 0) {
        const int sg = q + lane;
        int row = 0, nr = 0;
        l_s0 = l_e = 0;
        if (sg < nseg) {
          const int4 d = d_seg[sg];
          l_s0 = sg == 0 ? p + 1 : start[ic + d.x];  // segment 0 starts with the own cell
          l_e = start[ic + d.y + 1];
          row = d.z;
          nr = d.w;
        }
        l_sl = s_base[row] - s_first[row];  // slot = sorted position + l_sl
        l_nir = __ballot_sync(0xffffffffu, nr != 0);
      }
      const int s0 = __shfl_sync(0xffffffffu, l_s0, q & 31), e = __shfl_sync(0xffffffffu, l_e, q & 31),
                sl0 = __shfl_sync(0xffffffffu, l_sl, q & 31);
      const bool nir = (l_nir >> (q & 31)) & 1u;
      for (int b = s0; b < e; b += 32) {
        const int jj = b + lane;
        bool acc = false;
        if (jj < e) {
          if (nir) {
            acc = true;
          } else {
            const float4 xj = s_x[jj + sl0];
            const float dx = xj.x - xif.x, dy = xj.y - xif.y, dz = xj.z - xif.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < cg.rcsq_lo) {
              acc = true;
            } else if (r2 <= cg.rcsq_hi) {
              const double4_32a xd = xs[jj];
              const double ddx = sub_rn(xd.x, xi.x), ddy = sub_rn(xd.y, xi.y), ddz = sub_rn(xd.z, xi.z);
              const double rsq = add_rn(add_rn(mul_rn(ddx, ddx), mul_rn(ddy, ddy)), mul_rn(ddz, ddz));
              acc = rsq <= cg.rcsq;
              ++ncand64;
            }
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, acc);
        if (acc) {
          const int k = count + __popc(m & lt) + 1;
          const int a = s_at[jj + sl0];
          nfwd += a >= natms;
          if (k <= max_list) {
            li[k] = a + 1;
            si[k] = jj;
          }
        }
        count += __popc(m);
      }
    }
    // pass 2: backward cells that are halo cells (border atoms only), from global memory
    const int ix1 = ix - nlx0e, ix2 = ix - nlx1s, iy1 = iy - nly0e, iy2 = iy - nly1s, iz1 = iz - nlz0e,
              iz2 = iz - nlz1s;
    const bool border = (ix1 >= 1 && ix1 <= nlp) || (ix2 <= -1 && ix2 >= -nlp) || (iy1 >= 1 && iy1 <= nlp) ||
                        (iy2 <= -1 && iy2 >= -nlp) || (iz1 >= 1 && iz1 <= nlp) || (iz2 <= -1 && iz2 >= -nlp);
    if (border) {
      // 32 cells at a time, a lane each: their bounds, then their members as one sequence
      // (lane L of a step takes the member q, of the last cell that starts at or before q);
      // cell by cell each step had a chain of two dependent loads for a dozen members
      for (int k0 = 1; k0 < nsbcll; k0 += 32) {
        int c_s0 = 0, c_n = 0, c_nr = 0;
        if (k0 + lane < nsbcll) {
          const int2 d = d_sbc[k0 + lane];
          const int jx = ix - ((d.y & 255) - 64), jy = iy - (((d.y >> 8) & 255) - 64), jz = iz - (((d.y >> 16) & 255) - 64);
          if (jx <= nlx0e || jx >= nlx1s || jy <= nly0e || jy >= nly1s || jz <= nlz0e || jz >= nlz1s) {
            const int jc = ic - d.x;
            c_s0 = start[jc];
            c_n = start[jc + 1] - c_s0;
            c_nr = d.y >> 24;
          }
        }
        int inc = c_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += v;
        }
        const int tot = __shfl_sync(0xffffffffu, inc, 31);
        const int c_off0 = c_s0 - (inc - c_n);  // sorted position of member q of the sequence: q + c_off0
        const unsigned nirs = __ballot_sync(0xffffffffu, c_nr != 0);
        for (int b = 0; b < tot; b += 32) {
          const int q = b + lane;
          int L = 0;  // cells whose members all precede q
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const int v = __shfl_sync(0xffffffffu, inc, L + o - 1);
            if (v <= q) L += o;
          }
          const int jj = q + __shfl_sync(0xffffffffu, c_off0, L & 31);
          bool acc = false;
          if (q < tot) {
            if ((nirs >> L) & 1u) {
              acc = true;
            } else {
              const float4 xj = xsf[jj];
              const float dx = xj.x - xif.x, dy = xj.y - xif.y, dz = xj.z - xif.z;
              const float r2 = dx * dx + dy * dy + dz * dz;
              if (r2 < cg.rcsq_lo) {
                acc = true;
              } else if (r2 <= cg.rcsq_hi) {
                const double4_32a xd = xs[jj];
                const double ddx = sub_rn(xd.x, xi.x), ddy = sub_rn(xd.y, xi.y), ddz = sub_rn(xd.z, xi.z);
                const double rsq = add_rn(add_rn(mul_rn(ddx, ddx), mul_rn(ddy, ddy)), mul_rn(ddz, ddz));
                acc = rsq <= cg.rcsq;
                ++ncand64;
              }
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, acc);
          if (acc) {
            const int k = count + __popc(m & lt) + 1;
            ++nbwd;
            if (k <= max_list) {
              li[k] = at_list[jj] + 1;
              si[k] = -1;
            }
          }
          count += __popc(m);
        }
      }
    }
    if (lane == 0) {
      // the stored length never exceeds max_list, so no later kernel can read
      // past the column even when the overflow status is ignored
      const int stored = min(count, max_list);
      li[0] = stored;
      li[-1] = stored;
      li[-2] = stored;
      li[-3] = stored;
      if (count > max_list) {
        atomicOr(&sc->status, ST_LIST_OVERFLOW);
        atomicMax(&sc->ibig, count);
      }
    }
  }
  ncand64 = warp_sumi(ncand64);
  nfwd = warp_sumi(nfwd);
  nbwd = warp_sumi(nbwd);
  if (lane == 0) {
    if (ncand64) atomicAdd(&sc->ncand_fp64, ncand64);
    if (nfwd) atomicAdd(&sc->halo_fwd, nfwd);
    if (nbwd) atomicAdd(&sc->halo_bwd, nbwd);
  }
}

// Half-shell Verlet list (neighbours.F90:876-1184), G lanes per local atom: the 32 / G
// consecutive local atoms of a warp (in sorted order: one or two cells) walk the reference's
// order of their own shells together, pass 1 run by run of consecutive cells, pass 2 (the backward
// cells that are halo cells) cell by cell.  The atoms of a cell read the same candidates, LANE_U
// consecutive ones per lane and step; an atom's lanes add up their accepted ones, which go to the
// atom's column in shared memory, and the warp writes the columns as rows of list(k, i) and
// spos(k, i) when one is nearly full.  A step with a candidate that FP32 cannot decide takes
// FP64 for that one.
// Beside list(k, i) the kernel writes spos(k, i): the partner's sorted position, or -1 for
// the entries of pass 2, whose pairs the partner atom's forward pass also lists, so that
// the pair kernels evaluate each pair once, from its forward copy.
// A warp per atom, its lanes over the candidates of a staged cell tile (k_list_tiles), spends 76
// instructions on 32 candidates, most of them on the compaction.  In ms, that kernel and this
// one (with G lanes per atom and U candidates per lane and step):
//                            tiles   2, 4    4, 4    8, 2    16, 2
//   4,096 ions               0.062   0.117   0.079   0.073   0.059
//   6,591-atom water         0.106   0.130   0.087   0.080   0.065
//   13,824 ions              0.105   0.110   0.079   0.077   0.091
//   46,656 ions              0.189   0.127   0.136   0.160   0.215
//   98,304-atom water        0.370   0.274   0.283   0.336   0.434
//   262,144 ions             0.697   0.445   0.509   0.632   0.891
// More lanes per atom shorten a warp's walk, which is what few warps wait for; fewer lanes
// waste fewer candidates at the ends of runs and cells.  Bound by issue and L1 reads at 262,144.
constexpr int LANE_NT = 64, LANE_CAP = 64, LANE_LD = LANE_CAP + 1;
template <int G, int LANE_U>
__global__ void __launch_bounds__(LANE_NT) k_list_lanes(int natms, CellGeom cg, int nsbcll, int nseg,
                                                        const int* __restrict__ loc_sp, const int* __restrict__ at_list,
                                                        const int* __restrict__ which_cell,
                                                        const int* __restrict__ start,
                                                        const double4_32a* __restrict__ xs,
                                                        const float4* __restrict__ xsf, int* __restrict__ list, int ld,
                                                        int* __restrict__ spos, int ldt, int max_list, DevScalars* sc) {
  constexpr int NA = 32 / G, STEP = G * LANE_U;  // atoms per warp, candidates per step
  static_assert(STEP <= LANE_CAP / 2, "a step fits the column");
  __shared__ int2 s_buf[LANE_NT / 32][NA * LANE_LD];
  const int lane = threadIdx.x & 31, r = lane % G, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w * NA >= natms || halo_cut(sc)) return;
  int2* buf = s_buf[threadIdx.x >> 5];
  int2* const col = buf + (lane / G) * LANE_LD;
  const bool on = w * NA + lane / G < natms;
  const int p = loc_sp[min(w * NA + lane / G, natms - 1)];
  const int i = at_list[p], ic = which_cell[i];
  const float4 xif = xsf[p];
  int cnt = 0, pend = 0;  // entries written, entries in the column
  int ncand64 = 0, nfwd = 0, nbwd = 0;

  auto flush = [&]() {
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int n = __shfl_sync(0xffffffffu, pend, a * G), il = __shfl_sync(0xffffffffu, i, a * G),
                k0 = __shfl_sync(0xffffffffu, cnt, a * G) + 1;
      for (int e = lane; e < n; e += 32) {
        const int2 v = buf[a * LANE_LD + e];
        const int k = k0 + e;
        if (v.y < 0) ++nbwd;
        else if (v.x >= natms) ++nfwd;
        if (k <= max_list) {
          list[(size_t)il * ld + 3 + k] = v.x + 1;
          spos[(size_t)il * ldt + k] = v.y;
        }
      }
    }
    __syncwarp();
    cnt += pend;
    pend = 0;
  };
  // the lines of the next candidates, a lane each, into L1
  auto touch = [&](int s0, int e) {
    const int jj = s0 + 8 * (lane & 7);
    float v;
    if (jj < e) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(&xsf[jj].x));
  };
  // the candidates [s0, e) of each atom, in step; back: pass 2, whose entries carry -1.  (Up
  // to LANE_U - 1 records beyond e are read, and not used: xsf has room for them.)
  const float mid = 0.5f * (cg.rcsq_lo + cg.rcsq_hi), half = 0.5f * (cg.rcsq_hi - cg.rcsq_lo);
  auto walk = [&](int s0, int e, bool nir, bool back) {
    const int len = __reduce_max_sync(0xffffffffu, e - s0);
    const float cut = nir ? 3.0e38f : mid, undecided = nir ? -1.f : 1.01f * half;
    float4 xn[LANE_U];
    auto load = [&](int jj) {
      const float4* q = xsf + (jj < e ? jj : p);
#pragma unroll
      for (int u = 0; u < LANE_U; ++u) xn[u] = q[u];
    };
    if (len > 0) load(s0 + r * LANE_U);
    for (int t = 0; t < len; t += STEP) {
      const int jj = s0 + t + r * LANE_U, rem = e - jj;
      float r2[LANE_U], b = 3.0e38f;
      int id[LANE_U];
#pragma unroll
      for (int u = 0; u < LANE_U; ++u) {
        const float dx = xn[u].x - xif.x, dy = xn[u].y - xif.y, dz = xn[u].z - xif.z;
        r2[u] = dx * dx + dy * dy + dz * dz;
        b = fminf(b, fabsf(r2[u] - cut));
        id[u] = __float_as_int(xn[u].w);
      }
      if (t + STEP < len) load(jj + STEP);
      unsigned m = 0;
#pragma unroll
      for (int u = 0; u < LANE_U; ++u)
        if (u < rem && r2[u] < cut) m |= 1u << u;
      if (__any_sync(0xffffffffu, b <= undecided)) {
#pragma unroll
        for (int u = 0; u < LANE_U; ++u)
          if (u < rem && r2[u] >= cg.rcsq_lo && r2[u] <= cg.rcsq_hi) {
            const double4_32a xi = xs[p], xd = xs[jj + u];
            const double ddx = sub_rn(xd.x, xi.x), ddy = sub_rn(xd.y, xi.y), ddz = sub_rn(xd.z, xi.z);
            const bool ok = add_rn(add_rn(mul_rn(ddx, ddx), mul_rn(ddy, ddy)), mul_rn(ddz, ddz)) <= cg.rcsq;
            m = (m & ~(1u << u)) | (nir || ok ? 1u << u : 0u);
            ++ncand64;
          }
        __syncwarp();
      }
      const int c = __popc(m);
      int inc = c;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o, G);
        if (r >= o) inc += v;
      }
      int2* at = col + (pend + inc - c);
#pragma unroll
      for (int u = 0; u < LANE_U; ++u)
        if ((m >> u) & 1u) *at++ = make_int2(id[u], back ? -1 : jj + u);
      pend += __shfl_sync(0xffffffffu, inc, G - 1, G);
      if (__any_sync(0xffffffffu, pend > LANE_CAP - STEP)) flush();
    }
  };

  // pass 1 (the bounds of the run after the next and the lines of the next are on their way
  // while this one is walked)
  {
    int s0 = p + 1, e = start[ic + d_seg[0].y + 1], s1 = 0, e1 = 0;  // segment 0 starts with the own cell
    if (nseg > 1) {
      s1 = start[ic + d_seg[1].x];
      e1 = start[ic + d_seg[1].y + 1];
    }
    touch(s0, e);
    for (int q = 0; q < nseg; ++q) {
      int s2 = 0, e2 = 0;
      if (q + 2 < nseg) {
        const int4 d = d_seg[q + 2];
        s2 = start[ic + d.x];
        e2 = start[ic + d.y + 1];
      }
      touch(s1, e1);
      walk(s0, on ? e : s0, d_seg[q].w != 0, false);
      s0 = s1; e = e1;
      s1 = s2; e1 = e2;
    }
  }
  // pass 2: backward cells that are halo cells (border atoms only)
  {
    const int icm = ic - 1, ix = icm % cg.NX, iz = icm / (cg.NX * cg.NY), iy = icm / cg.NX - cg.NY * iz;
    const int nlp = cg.nlp, nl0e = nlp - 1;
    const int nlx1s = cg.nlx + nlp, nly1s = cg.nly + nlp, nlz1s = cg.nlz + nlp;
    const int ix1 = ix - nl0e, ix2 = ix - nlx1s, iy1 = iy - nl0e, iy2 = iy - nly1s, iz1 = iz - nl0e, iz2 = iz - nlz1s;
    const bool border = on && ((ix1 >= 1 && ix1 <= nlp) || (ix2 <= -1 && ix2 >= -nlp) || (iy1 >= 1 && iy1 <= nlp) ||
                               (iy2 <= -1 && iy2 >= -nlp) || (iz1 >= 1 && iz1 <= nlp) || (iz2 <= -1 && iz2 >= -nlp));
    auto bounds = [&](int k, int& s0, int& e) {
      s0 = e = 0;
      if (!border || k >= nsbcll) return;
      const int2 d = d_sbc[k];
      const int jx = ix - ((d.y & 255) - 64), jy = iy - (((d.y >> 8) & 255) - 64), jz = iz - (((d.y >> 16) & 255) - 64);
      if (jx <= nl0e || jx >= nlx1s || jy <= nl0e || jy >= nly1s || jz <= nl0e || jz >= nlz1s) {
        s0 = start[ic - d.x];
        e = start[ic - d.x + 1];
      }
    };
    if (__any_sync(0xffffffffu, border)) {
      int s0, e, s1, e1, s2, e2, s3, e3, s4, e4;
      bounds(1, s0, e);
      bounds(2, s1, e1);
      bounds(3, s2, e2);
      bounds(4, s3, e3);
      touch(s0, e);
      touch(s1, e1);
      for (int k = 1; k < nsbcll; ++k) {
        bounds(k + 4, s4, e4);
        touch(s2, e2);
        walk(s0, e, d_sbc[k].y >> 24 != 0, true);
        s0 = s1; e = e1;
        s1 = s2; e1 = e2;
        s2 = s3; e2 = e3;
        s3 = s4; e3 = e4;
      }
    }
  }
  flush();
  if (on && r == 0) {
    // the stored length never exceeds max_list, so no later kernel can read
    // past the column even when the overflow status is ignored
    int* li = list + (size_t)i * ld + 3;
    const int stored = min(cnt, max_list);
    li[0] = stored;
    li[-1] = stored;
    li[-2] = stored;
    li[-3] = stored;
    if (cnt > max_list) {
      atomicOr(&sc->status, ST_LIST_OVERFLOW);
      atomicMax(&sc->ibig, cnt);
    }
  }
  ncand64 = warp_sumi(ncand64);
  nfwd = warp_sumi(nfwd);
  nbwd = warp_sumi(nbwd);
  if (lane == 0) {
    if (ncand64) atomicAdd(&sc->ncand_fp64, ncand64);
    if (nfwd) atomicAdd(&sc->halo_fwd, nfwd);
    if (nbwd) atomicAdd(&sc->halo_bwd, nbwd);
  }
}

// Frozen (neighbours.F90:1198-1225) and excluded (:1229-1306) reordering, one warp per
// atom.  The reference walks the list from its end and swaps each hit with the last entry
// of the kept part; every entry between the hit and that one has been kept, so only the
// hits act.  The warp finds them, 128 entries' loads in flight together, and lane 0 swaps
// them in descending order, spos following.  (One thread per atom took 0.30 ms for 1,536
// atoms and 0.36 ms for 98,304, a dependent load per entry; this takes 0.010 and 0.066 ms.)
template <typename Hit>
__device__ __forceinline__ int list_move_hits(int* li, int* ti, int n, Hit hit) {
  const int lane = threadIdx.x & 31;
  int m_end = n;
  for (int b = (n - 1) & ~127; b >= 0 && n > 0; b -= 128) {
    int j[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int kk = b + 32 * u + lane + 1;
      j[u] = kk <= n ? li[kk] : 0;
    }
    unsigned hits[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) hits[u] = __ballot_sync(0xffffffffu, j[u] != 0 && hit(j[u]));
#pragma unroll
    for (int u = 3; u >= 0; --u) {
      for (unsigned m = hits[u]; m; --m_end) {
        const int bit = 31 - __clz((int)m);
        m ^= 1u << bit;
        const int k = b + 32 * u + bit + 1;
        if (lane == 0 && k < m_end) {
          const int jk = li[k], tk = ti[k];
          li[k] = li[m_end]; li[m_end] = jk;
          ti[k] = ti[m_end]; ti[m_end] = tk;
        }
      }
    }
  }
  return m_end;
}

__global__ void __launch_bounds__(256) k_list_reorder(int natms, int* list, int ld, int* spos, int ldt,
                                                      const int* __restrict__ lfrzn, const int* __restrict__ ltg,
                                                      const int* __restrict__ list_excl, int ldx, int megfrz,
                                                      int lbook, const DevScalars* sc) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= natms || halo_cut(sc)) return;
  int* li = list + (size_t)i * ld + 3;
  int* ti = spos + (size_t)i * ldt;
  const int n0 = li[0];
  int n1 = n0;
  if (megfrz > 1 && lfrzn[i] > 0) n1 = list_move_hits(li, ti, n0, [&](int j) { return lfrzn[j - 1] > 0; });
  int n2 = n1;
  if (lbook) {
    const int* ex = list_excl + (size_t)i * ldx;
    const int ii = ex[0];
    if (ii > 0) {
      __syncwarp();  // lane 0's swaps above
      const int e1 = ex[1], e2 = ii > 1 ? ex[2] : e1;
      n2 = list_move_hits(li, ti, n1, [&](int j) {
        const int jj = j <= natms ? j : ltg[j - 1];  // a local atom's global id is its index
        bool h = e1 == jj || e2 == jj;
        for (int t = 3; t <= ii; ++t) h |= ex[t] == jj;
        return h;
      });
    }
  }
  __syncwarp();
  if (lane == 0) {
    li[-2] = n0;
    li[-1] = n1;
    li[0] = n2;
    li[-3] = n2;
  }
}

// FP32 copy of positions + charge (mixed path and prefilter helpers)
// FP32 positions as an unevaluated sum hi + lo: in a large box the FP32
// coordinate alone carries an absolute error of up to half an ulp of |x|
// (7.6e-6 A at 180 A), while hi_i - hi_j + (lo_i - lo_j) keeps pair
// separations to FP32 precision of the separation itself.
// FP32 hi parts with the charge, and the lo remainders with the atom type in the
// fourth word (bit pattern), so a pair reads everything about j in two 16-byte loads
// Both records in one pass over the atoms (the FP64 values converted once): by atom index
// (xf, xlo: the type in xlo.w) and, for the sorted-position pair kernels, per sorted
// position sorted_pos[i] (xhs, and rec or, in the mixed form, xlh).  The same pass clears the
// force sums of the evaluation that follows (one launch for up to four; at 4,096 ions a
// fill takes 2 us and a gap).
struct ForceZero {
  int natms, mxatms;
  double *fx, *fy, *fz;      // FP64 forces (null in the mixed form)
  long long *fixp, *fixs;    // fixed-point sums by atom and by sorted position, with the pool's counter (or null)
};
__global__ void k_pos_records(const DevScalars* sc, const int* __restrict__ sorted_pos, const double* __restrict__ x,
                              const double* __restrict__ y, const double* __restrict__ z, const double* __restrict__ q,
                              const int* __restrict__ ltype, double pos_scale, float4* xf, float4* xlo, float2* qdf,
                              float4* xhs, PosRec* rec, uint2* xlh, ForceZero Z, unsigned long long* t_ns) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  stamp_time(t_ns);
  if (i < Z.natms) {
    if (Z.fx) { Z.fx[i] = 0.0; Z.fy[i] = 0.0; Z.fz[i] = 0.0; }
    if (Z.fixp) { Z.fixp[3 * i] = 0; Z.fixp[3 * i + 1] = 0; Z.fixp[3 * i + 2] = 0; }
  }
  if (i >= sc->nlast) return;
  if (Z.fixs) {
    Z.fixs[i] = 0; Z.fixs[Z.mxatms + i] = 0; Z.fixs[2 * (size_t)Z.mxatms + i] = 0;
    if (i == 0) Z.fixs[3 * (size_t)Z.mxatms] = 0;
  }
  const double xa = x[i], ya = y[i], za = z[i], qa = q[i];
  const int ta = ltype[i];
  const float hx = (float)xa, hy = (float)ya, hz = (float)za, hq = (float)qa;
  const float lx = (float)(xa - (double)hx), ly = (float)(ya - (double)hy), lz = (float)(za - (double)hz);
  xf[i] = make_float4(hx, hy, hz, hq);
  xlo[i] = make_float4(lx, ly, lz, __int_as_float(ta));
  const float lq = (float)(qa - (double)hq);
  if (qdf) qdf[i] = make_float2(hq, lq);
  if (xhs) {
    const int p = sorted_pos[i];
    xhs[p] = make_float4(hx, hy, hz, hq);
    if (xlh) {  // the mixed form's 8-byte record (pair_lo_type decodes it)
      xlh[p] = pack_lo_type(lx, ly, lz, ta);
    } else {
      PosRec r;
      r.x = __double2ll_rn(xa * pos_scale);
      r.y = __double2ll_rn(ya * pos_scale);
      r.z = __double2ll_rn(za * pos_scale);
      r.ql = lq;
      r.type = ta;
      rec[p] = r;
    }
  }
}

inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// ====================================================================== host
extern void dcell_host(const double* aaa, double* bbb);
extern void invert_host(const double* a, double* b, double* d);

static void upload_adds();

void list_setup() {
  // set_halo_particles constants (halo.F90:184-247)
  double cut = g.rcutx + 1.0e-6;
  double cp[10];
  dcell_host(g.cell, cp);
  int nl[3];
  for (int d = 0; d < 3; ++d) nl[d] = (int)(cp[6 + d] / (cut * 1.0));
  double det;
  invert_host(g.cell, h_halo.rc, &det);
  for (int d = 0; d < 3; ++d) {
    double cw = 1.0 / (double)(nl[d] * 1);
    // SPME needs a wider negative-direction halo for its splines (halo.F90:218-231);
    // without electrostatics the link-cell width alone
    double ecw = g.has_coul ? std::max(cw, (double)g.p.spline_pad / (double)g.p.kmax[d]) : cw;
    h_halo.ecw[d] = std::nextafter((-0.5 + ecw) + 0.0 * 1.0, 2.0) + DBL_MIN;
    h_halo.cw[d] = std::nextafter((-0.5 - cw) + 1.0 * 1.0, -2.0) - DBL_MIN - (nl[d] == 1 ? cw * 1.0e-10 : 0.0);
  }
  // export add vectors (deport_data.F90:1790-1796)
  const double* c = g.cell;
  const double sh[6][3] = {{+1, 0, 0}, {-1, 0, 0}, {0, +1, 0}, {0, -1, 0}, {0, 0, +1}, {0, 0, -1}};
  for (int m = 0; m < 6; ++m) {
    double u = sh[m][0], v = sh[m][1], w = sh[m][2];
    h_add[m][0] = c[0] * u + c[3] * v + c[6] * w;
    h_add[m][1] = c[1] * u + c[4] * v + c[7] * w;
    h_add[m][2] = c[2] * u + c[5] * v + c[8] * w;
  }
  upload_adds();
  const char* hb = getenv("GB_HALO_BLOCKS");
  h_halo_blocks = hb ? std::max(0, atoi(hb)) : 0;
  // link-cell geometry (neighbours.F90:396-463)
  double cut2 = g.rcutx + 1.0e-6;
  double disp[3] = {1.0 * cp[6] / cut2, 1.0 * cp[7] / cut2, 1.0 * cp[8] / cut2};
  int nlx = (int)disp[0], nly = (int)disp[1], nlz = (int)disp[2];
  int nlp = 1;
  double nlr2 = (double)g.natms;
  double dd = (nlx * nly * nlz) ? nlr2 / (double)(nlx * nly * nlz) : 0.0;
  while (nlx * nly * nlz > 0 && dd > g.p.pdplnc) {
    nlp = nlp + 1;
    double rr = (double)nlp;
    nlx = (int)(disp[0] * rr); nly = (int)(disp[1] * rr); nlz = (int)(disp[2] * rr);
    dd = nlr2 / (double)(nlx * nly * nlz);
  }
  g.nlx = nlx; g.nly = nly; g.nlz = nlz; g.nlp = nlp;
  g.NX = nlx + 2 * nlp; g.NY = nly + 2 * nlp; g.NZ = nlz + 2 * nlp;
  g.ncells = g.NX * g.NY * g.NZ;
  std::vector<int> off, nix, niy, niz;
  std::vector<unsigned char> nir;
  int nlp2 = nlp * nlp, nlp3 = (nlp - 1) * (nlp - 1);
  for (int iz = 0; iz <= nlp; ++iz) {
    int iz1 = iz > 0 ? (iz - 1) * (iz - 1) : 0, jz = iz * iz;
    for (int iy = -nlp; iy <= nlp; ++iy) {
      if (iz == 0 && iy < 0) continue;
      int a = std::abs(iy), iy1 = a > 0 ? (a - 1) * (a - 1) : 0, ll = iz1 + iy1;
      if (ll > nlp2) continue;
      int jy = jz + iy * iy;
      for (int ix = -nlp; ix <= nlp; ++ix) {
        if (iz == 0 && iy == 0 && ix < 0) continue;
        int b = std::abs(ix), ix1 = b > 0 ? (b - 1) * (b - 1) : 0;
        if (ll + ix1 > nlp2) continue;
        int jx = jy + ix * ix;
        nix.push_back(ix); niy.push_back(iy); niz.push_back(iz);
        nir.push_back(jx < nlp3 ? 1 : 0);
        off.push_back(ix + g.NX * (iy + g.NY * iz));
      }
    }
  }
  g.nsbcll = (int)off.size();
  if (g.nsbcll > MAX_SBC) throw (int)GB_ERR_ARG;
  // cell tiles: the rows (dy, dz) of the forward half shell in the order they first
  // appear, each with the range of dx its cells take
  {
    TilePlan& tp = g.tp;
    tp = TilePlan{};
    std::vector<unsigned char> row(off.size());
    for (size_t k = 0; k < off.size(); ++k) {
      int r = 0;
      while (r < tp.nrows && !(tp.dy[r] == niy[k] && tp.dz[r] == niz[k])) ++r;
      if (r == tp.nrows) {
        if (tp.nrows == TILE_MAX_ROWS) throw (int)GB_ERR_ARG;
        tp.dy[r] = niy[k]; tp.dz[r] = niz[k]; tp.dxlo[r] = nix[k]; tp.dxhi[r] = nix[k];
        ++tp.nrows;
      }
      tp.dxlo[r] = std::min(tp.dxlo[r], nix[k]);
      tp.dxhi[r] = std::max(tp.dxhi[r], nix[k]);
      row[k] = (unsigned char)r;
    }
    tp.r00 = row[0];  // offset (0, 0, 0) comes first; its row starts at dx = 0
    if (nix[0] != 0 || niy[0] != 0 || niz[0] != 0 || tp.dxlo[tp.r00] != 0) throw (int)GB_ERR_ARG;
    // segments: consecutive semi-ball cells of one row, adjacent along x, with one nir flag
    std::vector<int4> seg;
    std::vector<int2> sbc(off.size());
    for (size_t k = 0; k < off.size(); ++k) {
      sbc[k] = make_int2(off[k], (nix[k] + 64) | (niy[k] + 64) << 8 | (niz[k] + 64) << 16 | (int)nir[k] << 24);
      const bool joins = k > 0 && row[k] == row[k - 1] && nix[k] == nix[k - 1] + 1 && nir[k] == nir[k - 1];
      if (joins) seg.back().y = off[k];
      else seg.push_back(make_int4(off[k], off[k], row[k], nir[k]));
    }
    if (nlp > 63) throw (int)GB_ERR_ARG;  // beyond MAX_SBC long before
    g.nseg = (int)seg.size();
    GB_CUDA(cudaMemcpyToSymbol(d_seg, seg.data(), sizeof(int4) * seg.size()));
    GB_CUDA(cudaMemcpyToSymbol(d_sbc, sbc.data(), sizeof(int2) * sbc.size()));
    // tile width: the widest run of cells whose staged set stays near the capacity the
    // pair kernel's shared memory allows at two CTAs per SM
    const double apc = (double)g.natms / ((double)nlx * nly * nlz);
    auto cells_of = [&](int m) {
      int c = 0;
      for (int r = 0; r < tp.nrows; ++r) c += m + tp.dxhi[r] - tp.dxlo[r];
      return c;
    };
    int m = 1;
    const char* em = getenv("GB_TILE_M");
    if (em && atoi(em) > 0) {
      m = std::min(atoi(em), nlx);
    } else {
      for (int t = 2; t <= std::min(nlx, 8); ++t)
        if (1.3 * cells_of(t) * apc + 64.0 <= (double)TILE_CAP_TARGET) m = t;
    }
    tp.m = m;
    tp.ntx = (nlx + m - 1) / m; tp.nty = nly; tp.ntz = nlz;
    tp.ntiles = tp.ntx * tp.nty * tp.ntz;
    int cap = (int)(1.3 * cells_of(m) * apc) + 64;
    const char* ec = getenv("GB_TILE_CAP");  // this capacity, and the tile kernel at any size
    g.tiles_any = ec && atoi(ec) > 0;
    if (g.tiles_any) cap = atoi(ec);
    g.tile_cap_list = std::min(((cap + 31) / 32) * 32, (int)TILE_CAP_MAX);
    g.n_tile_over = 0;
    GB_CUDA(cudaFuncSetAttribute(k_list_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, 20 * TILE_CAP_MAX));
    if (g.tiles_alloc < tp.ntiles) {
      cudaFree(g.tile_rows); cudaFree(g.tile_info);
      GB_CUDA(cudaMalloc(&g.tile_rows, sizeof(int) * 2 * (size_t)tp.ntiles * TILE_MAX_ROWS));
      GB_CUDA(cudaMalloc(&g.tile_info, sizeof(int) * 4 * (size_t)tp.ntiles));
      g.tiles_alloc = tp.ntiles;
    }
  }
  for (int k = 0; k < 9; ++k) h_cg.rc[k] = h_halo.rc[k];
  h_cg.xdc = (double)(nlx * 1); h_cg.ydc = (double)(nly * 1); h_cg.zdc = (double)(nlz * 1);
  h_cg.nlp = nlp; h_cg.nlx = nlx; h_cg.nly = nly; h_cg.nlz = nlz;
  h_cg.NX = g.NX; h_cg.NY = g.NY; h_cg.NZ = g.NZ;
  h_cg.rcsq = g.rcutx * g.rcutx;
  // FP32 prefilter band: the FP32 rsq of a pair differs from the exact FP64
  // one by < 4e-4 A^2 for |coordinates| < 300 A and r ~ rc (rounding of the
  // coordinates to FP32 plus the FP32 arithmetic); take 25x that bound, scaled
  // with the box size.
  double Lmax = std::max(std::max(cp[0], cp[1]), cp[2]) + 2.0 * g.rcutx;
  double band = 0.01 * std::max(1.0, Lmax / 300.0) * std::max(1.0, g.rcutx / 13.0);
  h_cg.rcsq_lo = (float)(h_cg.rcsq - band);
  h_cg.rcsq_hi = (float)(h_cg.rcsq + band);
  h_cg.half_plus = std::nextafter(0.5, 1.0);
  if (g.cells_alloc < g.ncells + 2) {
    cudaFree(g.cell_count); cudaFree(g.cell_start); cudaFree(g.cell_lstart);
    GB_CUDA(cudaMalloc(&g.cell_count, sizeof(int) * (g.ncells + 2)));
    GB_CUDA(cudaMalloc(&g.cell_start, sizeof(int) * (g.ncells + 2)));
    GB_CUDA(cudaMalloc(&g.cell_lstart, sizeof(int) * (g.ncells + 2)));
    GB_CUDA(cudaMemset(g.cell_count, 0, sizeof(int) * (g.ncells + 2)));
    g.cells_alloc = g.ncells + 2;
  }
}

int list_relocate_and_halo(bool wait) {
  const int n = g.natms;
  g.spos_valid = false;  // new halo images: the sorted positions of the list are stale until the next build
  prof_begin(P_HALO);
  HaloArgs A;
  A.n = n; A.mxatms = g.mxatms;
  A.x = g.x; A.y = g.y; A.z = g.z; A.xb = g.xbg; A.yb = g.ybg; A.zb = g.zbg;
  for (int d = 0; d < 3; ++d) {
    const int k = g.cubic ? 0 : 4 * d;
    A.a[d] = 1.0 / g.cell[k];
    A.c[d] = g.cell[k];
  }
  A.half_minus = std::nextafter(0.5, 0.0);
  A.hg = h_halo;
  std::memcpy(A.add, h_add, sizeof(h_add));
  A.code = g.ixyz; A.src = g.src; A.shcode = g.shcode; A.ltg = g.ltg; A.ltype = g.ltype; A.lfrzn = g.lfrzn;
  A.chge = g.chge; A.weight = g.weight;
  A.sc = g.sc;
  const int nb = std::max(1, h_halo_blocks ? h_halo_blocks : std::min(nblocks(n, HALO_NT), 2 * g.nsm));
  A.cnt = gb_scan_scratch(HALO_NC * nb);
  k_halo_count<<<nb, HALO_NT, 0, g.stream>>>(A);
  GB_LAUNCHED();
  k_halo_write<<<nb, HALO_NT, 0, g.stream>>>(A);
  GB_LAUNCHED();
  prof_end(P_HALO);
  if (!wait) return GB_OK;  // list_build, which follows, reports ST_HALO_OVERFLOW
  gb_sync_scalars();
  if (g.hsc->status & ST_HALO_OVERFLOW) return GB_ERR_HALO;
  return GB_OK;
}

// the image shifts on the device for the halo refresh: allocated and written where the
// list geometry is set up, copied again only when they change (a step captured into a CUDA
// graph then holds neither an allocation nor a copy from pageable host memory)
static double* d_adds = nullptr;
static double d_adds_host[18];
static void upload_adds() {
  if (!d_adds) GB_CUDA(cudaMalloc(&d_adds, sizeof(double) * 18));
  GB_CUDA(cudaMemcpy(d_adds, h_add, sizeof(double) * 18, cudaMemcpyHostToDevice));
  std::memcpy(d_adds_host, h_add, sizeof(d_adds_host));
}

int list_refresh_halo() {
  if (!d_adds || std::memcmp(d_adds_host, h_add, sizeof(d_adds_host)) != 0) upload_adds();
  k_halo_refresh<<<nblocks(g.mxatms - g.natms, 256), 256, 0, g.stream>>>(g.natms, g.sc, g.src, g.shcode, g.x, g.y,
                                                                          g.z, d_adds);
  GB_LAUNCHED();
  return GB_OK;
}

int list_build() {
  const int T = 256;
  cudaStream_t st = g.stream;
  const int mx = g.mxatms;
  const TilePlan& tp = g.tp;
  const int cap = g.tile_cap_list;
  bool tiles = (g.natms / 2 < 12 * g.nsm || g.tiles_any) && g.n_tile_over == 0;
  prof_begin(P_BIN);
  k_bin<<<nblocks(mx, T), T, 0, st>>>(g.natms, g.sc, g.x, g.y, g.z, h_cg, g.which_cell, g.cell_count);
  GB_LAUNCHED();
  k_cell_scan<<<2, 1024, 0, st>>>(g.ncells + 2, h_cg, g.cell_count, g.cell_start, g.cell_lstart, g.sc);
  GB_LAUNCHED();
  int* tmp = gb_scan_scratch(mx + 1);
  k_cell_scatter<<<nblocks(mx, T), T, 0, st>>>(g.sc, g.which_cell, g.cell_start, g.cell_count, tmp);
  GB_LAUNCHED();
  k_cell_sort<<<nblocks(g.ncells + 1, SORT_NT / 32) + RESID_BLOCKS + (tiles ? nblocks(tp.ntiles, SORT_NT) : 0), SORT_NT,
                0, st>>>(
      g.ncells + 1, g.natms, g.cell_start, g.cell_lstart, tmp, g.at_list, g.sorted_pos, g.loc_sp, g.x, g.y, g.z, g.xs,
      g.xsf, tp, h_cg, g.tile_rows, g.tile_info, cap, g.sc);
  GB_LAUNCHED();
  prof_end(P_BIN);
  // The lanes per atom by the warps per SM that they give (the table at k_list_lanes); below
  // 12 with the most lanes the tiles' CTAs, which share a tile's atoms, are faster.
  const int n = g.natms, nsm = g.nsm;
  const int G = n / 16 >= 10 * nsm ? 2 : n / 4 >= 16 * nsm ? 8 : 16;
  auto lanes = G == 2 ? k_list_lanes<2, 4> : G == 8 ? k_list_lanes<8, 2> : k_list_lanes<16, 2>;
  for (;;) {
    prof_begin(P_LIST);
    if (tiles) {
      // several CTAs share a tile's atoms (each stages its whole shell), so that the device has
      // about three CTAs per SM
      const int split = std::max(1, std::min(8, 3 * nsm / std::max(tp.ntiles, 1)));
      k_list_tiles<<<dim3(tp.ntiles, split), 256, (size_t)cap * 20, st>>>(
          n, h_cg, tp, g.nsbcll, g.nseg, cap, g.tile_rows, g.tile_info, g.at_list, g.which_cell, g.cell_start, g.xs,
          g.xsf, g.list, g.ld, g.spos, g.ldt, g.p.max_list, g.sc);
    } else {
      lanes<<<nblocks((long long)n * G, LANE_NT), LANE_NT, 0, st>>>(
          n, h_cg, g.nsbcll, g.nseg, g.loc_sp, g.at_list, g.which_cell, g.cell_start, g.xs, g.xsf, g.list, g.ld, g.spos,
          g.ldt, g.p.max_list, g.sc);
    }
    GB_LAUNCHED();
    if (g.lbook || g.megfrz > 1) {  // (lists of tiles left out hold valid older entries, or none)
      k_list_reorder<<<nblocks((long long)n * 32, 256), 256, 0, st>>>(n, g.list, g.ld, g.spos, g.ldt, g.lfrzn, g.ltg,
                                                                      g.list_excl, g.p.max_exclude + 1, g.megfrz,
                                                                      g.lbook ? 1 : 0, g.sc);
      GB_LAUNCHED();
    }
    prof_end(P_LIST);
    gb_sync_scalars();  // (resolves the timings)
    if (g.hsc->status & ST_HALO_OVERFLOW) return GB_ERR_HALO;  // (list_relocate_and_halo without its wait)
    if (!tiles || g.hsc->tile_over == 0) break;
    g.n_tile_over = g.hsc->tile_over;  // denser tiles than planned: this list and the later ones from the other kernel
    tiles = false;
    GB_CUDA(cudaMemsetAsync(&g.sc->ibig, 0, sizeof(int), st));
    GB_CUDA(cudaMemsetAsync(&g.sc->halo_fwd, 0, 2 * sizeof(int), st));  // halo_fwd, halo_bwd
  }
  if (g.hsc->status & ST_LIST_OVERFLOW) return GB_ERR_LIST_OVERFLOW;
  // every pair across the periodic boundary is listed from both of its atoms, once in a
  // forward pass and once in the backward halo pass; the sorted-position pair kernels
  // evaluate the forward copy (else the atom-index kernels run, by the smaller global id)
  g.spos_valid = g.hsc->halo_fwd == g.hsc->halo_bwd;
  ++g.list_gen;  // the learned-MTS short list is rebuilt from this list on demand
  return GB_OK;
}

void list_pos_records(bool sorted) {
  const bool f64 = g.precision == GB_FP64;
  const ForceZero Z = {g.natms, g.mxatms, f64 ? g.fx : nullptr, g.fy, g.fz, !f64 || sorted ? g.fixp : nullptr,
                       sorted ? g.fixs : nullptr};
  k_pos_records<<<nblocks(g.mxatms, 256), 256, 0, g.stream>>>(
      g.sc, g.sorted_pos, g.x, g.y, g.z, g.chge, g.ltype, g.pos_scale, g.xf, g.xlo, f64 ? g.qdf : nullptr,
      sorted ? g.xhs : nullptr, g.rec, f64 ? nullptr : g.xlh, Z, stamp_at(1));
  GB_LAUNCHED();
}


