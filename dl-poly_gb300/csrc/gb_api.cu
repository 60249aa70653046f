// gb_api.cu - the C-ABI of the GB300 DL_POLY force/update path
// (include/gb300_dlpoly.h): device context, interpolation tables, the
// exported entry points and the resident md_vv step loop.
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "gb_common.cuh"
#include "gb_df64.cuh"

Dev g;

namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double kR4pie0 = 138935.4835;  // constants.F90:100

inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

// -------------------------------------------------------------- reductions
__global__ void k_reduce_blocks(const double* blk, int nb, int nv, double* out) {
  // one warp per value; fixed order -> deterministic
  int v = blockIdx.x;
  if (v >= nv) return;
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += blk[(size_t)b * nv + v];
  __shared__ double red[32];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) out[v] = t;
  }
}

__global__ void k_scan_excl(const int* in, int* out, int n) {
  __shared__ int part[1024];
  const int T = blockDim.x;
  const int per = (n + T - 1) / T;
  const int b = threadIdx.x * per;
  int s = 0;
  for (int k = 0; k < per; ++k) if (b + k < n) s += in[b + k];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < T; o <<= 1) {
    int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = part[threadIdx.x] - s;
  for (int k = 0; k < per; ++k)
    if (b + k < n) { out[b + k] = run; run += in[b + k]; }
}

__global__ void k_gather_parts(int n, const unsigned char* parts, double* x, double* y, double* z) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* r = reinterpret_cast<const double*>(parts + (size_t)i * 64);
  x[i] = r[0]; y[i] = r[1]; z[i] = r[2];
}

__global__ void k_nonfinite(int n, const double* a, const double* b, const double* c, int* status) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (!isfinite(a[i]) || !isfinite(b[i]) || !isfinite(c[i])) atomicOr(status, ST_NONFINITE);
}

// State transfer between the device arrays and caller buffers in pinned, mapped host
// memory: each thread moves element i of every array, so one launch replaces one copy per
// array.  Positions are checked for non-finite values on the way in; any thread that finds
// one stores ST_NONFINITE to the flag (the host clears it before the launch).
struct HostArrays {
  const double* h[9];
  double* d[9];
  int n;
};

__global__ void k_upload_state(HostArrays a, int narr, int* flag) {
  const int stride = gridDim.x * blockDim.x;
  int bad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += stride) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (k < narr) {
        const double v = a.h[k][i];
        a.d[k][i] = v;
        if (k < 3 && !isfinite(v)) bad = 1;
      }
    }
  }
  if (bad) *flag = ST_NONFINITE;
}

__global__ void k_download_state(HostArrays a) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += stride) {
#pragma unroll
    for (int k = 0; k < 9; ++k)
      if (a.d[k]) const_cast<double*>(a.h[k])[i] = a.d[k][i];
  }
}

// The device-side address of a caller buffer of n doubles when the whole buffer lies in
// pinned host memory mapped into the device's address space, else nullptr.
static double* mapped_span(const double* p, size_t n) {
  if (!p || n == 0) return nullptr;
  cudaPointerAttributes a0, a1;
  if (cudaPointerGetAttributes(&a0, p) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  if (a0.type != cudaMemoryTypeHost || !a0.devicePointer) return nullptr;
  const double* last = p + (n - 1);
  if (cudaPointerGetAttributes(&a1, last) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  if (a1.type != cudaMemoryTypeHost || !a1.devicePointer) return nullptr;
  double* d0 = static_cast<double*>(a0.devicePointer);
  if (static_cast<double*>(a1.devicePointer) != d0 + (n - 1)) return nullptr;
  return d0;
}

static int copy_grid(int n) { return std::max(1, std::min(nblocks(n, 256), 152 * 8)); }

std::vector<double> h_tmp;
int* d_scratch = nullptr;
size_t d_scratch_n = 0;
int* d_scratch_s = nullptr;  // the side stream's
size_t d_scratch_s_n = 0;

template <typename T>
void dalloc(T** p, size_t n) {
  GB_CUDA(cudaMalloc(p, sizeof(T) * std::max<size_t>(n, 1)));
  GB_CUDA(cudaMemset(*p, 0, sizeof(T) * std::max<size_t>(n, 1)));
}

// Captures the work body() issues on the main stream (and on the side stream it forks
// and joins) into *exec: a new graph, or the update of the existing one when its topology
// is unchanged.  Nothing runs during a capture.  *nk: the kernels of one launch (the launch
// counter is restored: graph launches add them).  Returns false, with nothing captured and
// the stream out of capture, when the body does something a capture cannot hold.
template <typename F>
static bool capture_graph(cudaGraphExec_t* exec, int64_t* nk, F&& body) {
  const int64_t l0 = g.launches;
  GB_CUDA(cudaStreamBeginCapture(g.main_stream, cudaStreamCaptureModeThreadLocal));
  bool ok = true;
  try {
    body();
  } catch (int) {
    ok = false;
  }
  cudaGraph_t graph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(g.main_stream, &graph);
  *nk = g.launches - l0;
  g.launches = l0;
  g.stream = g.main_stream;
  g.side = false;
  g.join_pending = false;
  if (!ok || e != cudaSuccess || !graph) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return false;
  }
  if (*exec) {
    cudaGraphExecUpdateResultInfo info;
    if (cudaGraphExecUpdate(*exec, graph, &info) != cudaSuccess) {
      cudaGetLastError();
      cudaGraphExecDestroy(*exec);
      *exec = nullptr;
    }
  }
  cudaError_t ei = cudaSuccess;
  if (!*exec) ei = cudaGraphInstantiate(exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ei != cudaSuccess) {
    cudaGetLastError();
    *exec = nullptr;
    return false;
  }
  return true;
}

static void launch_graph(cudaGraphExec_t exec, int64_t nk) {
  GB_CUDA(cudaGraphLaunch(exec, g.main_stream));
  g.launches += nk;
}

void free_graphs() {
  if (g.gx_vv1) cudaGraphExecDestroy(g.gx_vv1);
  if (g.gx_step) cudaGraphExecDestroy(g.gx_step);
  g.gx_vv1 = g.gx_step = nullptr;
}

void free_all() {
  void* ptrs[] = {g.x, g.y, g.z, g.xf, g.xlo, g.fx, g.fy, g.fz, g.fixp, g.vx, g.vy, g.vz, g.hdw, g.chge, g.weight, g.ltype, g.ltg,
                  g.lfrzn, g.ixyz, g.src, g.shcode, g.xbg, g.ybg, g.zbg, g.ox, g.oy, g.oz, g.which_cell,
                  g.cell_count, g.cell_start, g.cell_lstart, g.at_list, g.sorted_pos, g.xs, g.xsf, g.list, g.blk,
                  g.list_excl, g.erfc_coef, g.erfc_coef_f, g.vdw_coef, g.vdw_coef_f,
                  g.vdw_kind, g.vdw_eps, g.vdw_sig, g.erfc_df, g.vdw_df, g.qdf, g.spos, g.xhs, g.rec, g.xlh, g.fixs, g.eat, g.loc_sp,
                  g.tile_rows, g.tile_info, g.blkacc, g.con_i, g.con_j, g.con_d0, g.dxx, g.dyy,
                  g.dzz, g.dxt, g.dyt, g.dzt, g.dt2, g.gam, g.listot, g.acon_start, g.acon_list, g.sc, d_scratch,
                  d_scratch_s, g.blkacc_s};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  free_graphs();
  mts_free();
  spme_free();
  metal_free();
  if (g.hsc) cudaFreeHost(g.hsc);
  if (g.ring) cudaFreeHost(g.ring);
  if (g.hflag) cudaFreeHost(g.hflag);
  if (g.main_stream) {
    for (int k = 0; k < 8; ++k) cudaEventDestroy(g.ev[k]);
    cudaEventDestroy(g.ev_fork);
    cudaEventDestroy(g.ev_join);
    cudaStreamDestroy(g.main_stream);
    cudaStreamDestroy(g.side_stream);
  }
  d_scratch = nullptr;
  d_scratch_n = 0;
  d_scratch_s = nullptr;
  d_scratch_s_n = 0;
  g = Dev();
}

// quadratic coefficients of the 3-point interpolant over points k, k+1, k+2
inline void quad_coef(double p1, double p2, double p3, double* c) {
  double c2 = 0.5 * (p3 - 2.0 * p2 + p1);
  c[0] = p1;
  c[1] = (p2 - p1) - c2;
  c[2] = c2;
}

double calc_erfc_n(double x) {  // numerics.F90:3647-3667
  const double a1 = 0.254829592, a2 = -0.284496736, a3 = 1.421413741, a4 = -1.453152027, a5 = 1.061405429,
               pp = 0.3275911;
  double tt = 1.0 / (1.0 + pp * x);
  return tt * (a1 + tt * (a2 + tt * (a3 + tt * (a4 + tt * a5)))) * std::exp(-(x * x));
}

void build_tables(const double* vdw_prm) {
  const double rcut = g.p.rcut, alpha = g.p.alpha;
  // erfc(ar)/r and derivative tables, table(i) = f(i*h), i = 1..n (electrostatic.F90:88-127)
  const int n = g.nsamples;
  std::vector<double> te(n + 3, 0.0), td(n + 3, 0.0);
  const double h = rcut / (double)(n - 4);
  g.erfc_rdr = 1.0 / h;
  const double rsqrpi = 1.0 / std::sqrt(kPi);
  for (int i = 1; i <= n; ++i) {
    double r = (double)i * h;
    te[i] = calc_erfc_n(alpha * r) / r;
    td[i] = (calc_erfc_n(alpha * r) / r + alpha * (2.0 * std::exp(-((alpha * r) * (alpha * r))) * rsqrpi)) / (r * r);
  }
  std::vector<double> ec((size_t)(n + 1) * 6, 0.0);
  for (int k = 0; k + 2 <= n; ++k) {
    quad_coef(te[k], te[k + 1], te[k + 2], &ec[(size_t)k * 6]);
    quad_coef(td[k], td[k + 1], td[k + 2], &ec[(size_t)k * 6 + 3]);
  }
  // vdW tables (vdw.F90:1397-1460): tab(i) = lj(i*dlr), i = 1..max_grid
  const int mg = g.max_grid;
  const double dl = g.p.rvdw / (double)(mg - 4);
  g.vdw_rdr = 1.0 / dl;
  g.nkey = g.p.ntypes * (g.p.ntypes + 1) / 2;
  const int vstride = (mg + 3) * 6;
  std::vector<double> vc((size_t)g.nkey * vstride, 0.0);
  g.h_vdw_kind.assign(g.nkey, 0);
  g.h_vdw_eps.assign(g.nkey, 0.0);
  g.h_vdw_sig.assign(g.nkey, 0.0);
  for (int key = 0; key < g.nkey; ++key) {
    g.h_vdw_kind[key] = (int)vdw_prm[3 * key];
    g.h_vdw_eps[key] = vdw_prm[3 * key + 1];
    g.h_vdw_sig[key] = vdw_prm[3 * key + 2];
    if (g.h_vdw_kind[key] != 1) continue;
    std::vector<double> tf(mg + 3, 0.0), tp(mg + 3, 0.0);
    for (int i = 1; i <= mg; ++i) {
      double r = (double)i * dl;
      double sor = g.h_vdw_sig[key] / r;
      double sor6 = sor * sor * sor * sor * sor * sor;
      tp[i] = 4.0 * g.h_vdw_eps[key] * sor6 * (sor6 - 1.0);
      tf[i] = 24.0 * g.h_vdw_eps[key] * sor6 * (2.0 * sor6 - 1.0);
    }
    for (int k = 1; k + 2 <= mg; ++k) {
      quad_coef(tf[k], tf[k + 1], tf[k + 2], &vc[(size_t)key * vstride + (size_t)k * 6]);
      quad_coef(tp[k], tp[k + 1], tp[k + 2], &vc[(size_t)key * vstride + (size_t)k * 6 + 3]);
    }
  }
  dalloc(&g.erfc_coef, ec.size());
  dalloc(&g.erfc_coef_f, ec.size());
  dalloc(&g.vdw_coef, vc.size());
  dalloc(&g.vdw_coef_f, vc.size());
  GB_CUDA(cudaMemcpy(g.erfc_coef, ec.data(), sizeof(double) * ec.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.vdw_coef, vc.data(), sizeof(double) * vc.size(), cudaMemcpyHostToDevice));
  // double-float copies for the FP64 form's pair loop: per interval (c0, c1) of the first
  // and of the second polynomial as hi/lo pairs, then (c2 first, c2 second) as hi/lo pairs
  {
    auto pack = [](const double* c, float4* o) {  // c: first c0..c2, second c3..c5
      float h0, l0, h1, l1;
      df_split(c[0], &h0, &l0); df_split(c[1], &h1, &l1);
      o[0] = make_float4(h0, l0, h1, l1);
      df_split(c[3], &h0, &l0); df_split(c[4], &h1, &l1);
      o[1] = make_float4(h0, l0, h1, l1);
      df_split(c[2], &h0, &l0); df_split(c[5], &h1, &l1);
      o[2] = make_float4(h0, l0, h1, l1);
    };
    std::vector<float4> edf((size_t)(n + 1) * 3), vdf((size_t)g.nkey * (mg + 3) * 3);
    for (size_t k = 0; k < (size_t)(n + 1); ++k) pack(&ec[k * 6], &edf[k * 3]);
    for (size_t k = 0; k < (size_t)g.nkey * (mg + 3); ++k) pack(&vc[k * 6], &vdf[k * 3]);
    dalloc(&g.erfc_df, edf.size());
    dalloc(&g.vdw_df, vdf.size());
    GB_CUDA(cudaMemcpy(g.erfc_df, edf.data(), sizeof(float4) * edf.size(), cudaMemcpyHostToDevice));
    GB_CUDA(cudaMemcpy(g.vdw_df, vdf.data(), sizeof(float4) * vdf.size(), cudaMemcpyHostToDevice));
  }
  std::vector<float> ecf(ec.begin(), ec.end()), vcf(vc.begin(), vc.end());
  GB_CUDA(cudaMemcpy(g.erfc_coef_f, ecf.data(), sizeof(float) * ecf.size(), cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.vdw_coef_f, vcf.data(), sizeof(float) * vcf.size(), cudaMemcpyHostToDevice));
  dalloc(&g.vdw_kind, g.nkey);
  dalloc(&g.vdw_eps, g.nkey);
  dalloc(&g.vdw_sig, g.nkey);
  GB_CUDA(cudaMemcpy(g.vdw_kind, g.h_vdw_kind.data(), sizeof(int) * g.nkey, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.vdw_eps, g.h_vdw_eps.data(), sizeof(double) * g.nkey, cudaMemcpyHostToDevice));
  GB_CUDA(cudaMemcpy(g.vdw_sig, g.h_vdw_sig.data(), sizeof(double) * g.nkey, cudaMemcpyHostToDevice));
}

template <typename F>
int guarded(F&& f) {
  if (!g.init) return GB_ERR_NOT_INIT;
  try {
    return f();
  } catch (int e) {
    return e;
  }
}

// forces for the current positions: SPME then the pair loop (drivers.F90:655-786)
// md_step: the evaluation belongs to an MD step, where the learned-MTS form
// (when configured) may replace SPME by the surrogate; *full_out tells which ran.
int compute_forces(double* eng8, double* stress9, bool do_spme, bool do_real, bool md_step = false,
                   bool* full_out = nullptr) {
  double st[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  double strec[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  double erc = 0, vrc = 0;
  double e6[6] = {0, 0, 0, 0, 0, 0};
  // FP32 hi + lo positions by atom index and, for the sorted-position pair kernels, the same
  // per sorted position, and cleared force sums (one pass)
  list_pos_records(do_real && g.spos_valid && g.use_sorted && !(g.precision == GB_FP64 && g.fp64_native));
  const bool mts = md_step && do_spme && mts_active();
  const bool full = mts ? mts_step_needs_spme() : (do_spme && g.has_coul);
  // a learned-MTS inner step: the coarse grid, the network's inputs and inference go to the
  // side stream once the pair kernel is launched, and run beside it
  const bool mts_side = mts && !full && g.use_overlap && do_real && !g.has_metal;
  if (mts && !mts_side) mts_coarse();
  // SPME on the side stream while the pair kernel runs (the plain FP64 form keeps one
  // stream: its kernels are bound by the FP64 unit both sides share).  One stream / two, NaCl in
  // the double-float form, us per step: 32,768 ions 436 / 433, 85,184 863 / 856, 110,592 1108 /
  // 1097, 262,144 2130 / 2122; cutoff 9 A and a finer grid, 110,592 1216 / 1208.
  const bool overlap = g.use_overlap && full && !mts && do_real && !g.has_metal &&
                       !(g.precision == GB_FP64 && g.fp64_native);
  if (overlap) {
    const bool deferred = g.defer_scalars;
    g.defer_scalars = true;  // both sides leave their sums on the device; read once below
    GB_CUDA(cudaEventRecord(g.ev_fork, g.main_stream));
    GB_CUDA(cudaStreamWaitEvent(g.side_stream, g.ev_fork, 0));
    struct SideGuard {
      bool defer;
      ~SideGuard() {
        g.stream = g.main_stream;
        g.side = false;
        g.defer_scalars = defer;
        if (g.join_pending) {  // left by an error between the fork and the join
          cudaStreamWaitEvent(g.main_stream, g.ev_join, 0);
          g.join_pending = false;
        }
      }
    } guard{deferred};
    g.stream = g.side_stream;
    g.side = true;
    spme_forces(&erc, &vrc, strec);
    GB_CUDA(cudaEventRecord(g.ev_join, g.side_stream));
    g.stream = g.main_stream;
    g.side = false;
    g.join_pending = true;
    pair_forces(e6, st);  // waits for the side stream before it folds the pair forces
    side_join();
    g.defer_scalars = deferred;
    if (!deferred) {
      gb_sync_scalars();
      spme_scalars(g.hsc, &erc, &vrc, strec);
      for (int k = 0; k < 9; ++k) st[k] += strec[k];
      pair_scalars(g.hsc, e6, st);
    }
  } else if (mts_side) {
    struct SideWork {
      double *erc, *vrc, *strec, *st;
    } work{&erc, &vrc, strec, st};
    struct SideGuard {
      ~SideGuard() {
        g.stream = g.main_stream;
        g.side = false;
        g.side_hook = nullptr;
        if (g.join_pending) {  // left by an error between the fork and the join
          cudaStreamWaitEvent(g.main_stream, g.ev_join, 0);
          g.join_pending = false;
        }
      }
    } guard;
    GB_CUDA(cudaEventRecord(g.ev_fork, g.main_stream));
    g.side_hook_arg = &work;
    g.side_hook = [](void* a) {
      SideWork* w = static_cast<SideWork*>(a);
      GB_CUDA(cudaStreamWaitEvent(g.side_stream, g.ev_fork, 0));
      g.stream = g.side_stream;
      g.side = true;
      mts_coarse();
      mts_inner(w->erc, w->vrc, w->strec);
      for (int k = 0; k < 9; ++k) w->st[k] += w->strec[k];  // before the pair stress joins st
      GB_CUDA(cudaEventRecord(g.ev_join, g.side_stream));
      g.stream = g.main_stream;
      g.side = false;
      g.join_pending = true;
    };
    if (do_real && (g.has_coul || g.has_vdw)) pair_forces(e6, st);
    run_side_hook();  // (when pair_forces had nothing to launch)
    side_join();
  } else {
    if (full) spme_forces(&erc, &vrc, strec);
    else if (mts) mts_inner(&erc, &vrc, strec);
    for (int k = 0; k < 9; ++k) st[k] += strec[k];
    if (do_real && (g.has_coul || g.has_vdw)) pair_forces(e6, st);
  }
  for (int k = 0; k < 4; ++k) g.metal_e4[k] = 0.0;
  if (do_real && g.has_metal) metal_forces(g.metal_e4, st);  // metal_ld_compute + metal_forces
  if (g.precision == GB_MIXED) integ_forces_to_fp64();
  if (mts && full) mts_after_full(erc, vrc, strec);
  if (full_out) *full_out = mts ? full : true;
  if (eng8) {
    eng8[0] = erc; eng8[1] = vrc;
    eng8[2] = e6[0]; eng8[3] = e6[1]; eng8[4] = e6[2]; eng8[5] = e6[3]; eng8[6] = e6[4]; eng8[7] = e6[5];
  }
  if (stress9) for (int k = 0; k < 9; ++k) stress9[k] = st[k];
  return GB_OK;
}

// build_follows: the caller builds the list when *update is set
int do_refresh(int32_t* update, bool build_follows = false) {
  int upd = integ_vnl_check();
  if (update) *update = upd;
  if (upd) return list_relocate_and_halo(!build_follows);
  return list_refresh_halo();
}

}  // namespace

// ---------------------------------------------------------- shared helpers
void dcell_host(const double* aaa, double* bbb) {
  bbb[0] = std::sqrt(aaa[0] * aaa[0] + aaa[1] * aaa[1] + aaa[2] * aaa[2]);
  bbb[1] = std::sqrt(aaa[3] * aaa[3] + aaa[4] * aaa[4] + aaa[5] * aaa[5]);
  bbb[2] = std::sqrt(aaa[6] * aaa[6] + aaa[7] * aaa[7] + aaa[8] * aaa[8]);
  bbb[3] = (aaa[0] * aaa[3] + aaa[1] * aaa[4] + aaa[2] * aaa[5]) / (bbb[0] * bbb[1]);
  bbb[4] = (aaa[0] * aaa[6] + aaa[1] * aaa[7] + aaa[2] * aaa[8]) / (bbb[0] * bbb[2]);
  bbb[5] = (aaa[3] * aaa[6] + aaa[4] * aaa[7] + aaa[5] * aaa[8]) / (bbb[1] * bbb[2]);
  double axb1 = aaa[1] * aaa[5] - aaa[2] * aaa[4], axb2 = aaa[2] * aaa[3] - aaa[0] * aaa[5],
         axb3 = aaa[0] * aaa[4] - aaa[1] * aaa[3];
  double bxc1 = aaa[4] * aaa[8] - aaa[5] * aaa[7], bxc2 = aaa[5] * aaa[6] - aaa[3] * aaa[8],
         bxc3 = aaa[3] * aaa[7] - aaa[4] * aaa[6];
  double cxa1 = aaa[7] * aaa[2] - aaa[8] * aaa[1], cxa2 = aaa[8] * aaa[0] - aaa[6] * aaa[2],
         cxa3 = aaa[6] * aaa[1] - aaa[7] * aaa[0];
  bbb[9] = std::fabs(aaa[0] * bxc1 + aaa[1] * bxc2 + aaa[2] * bxc3);
  double d[3] = {bbb[9] / std::sqrt(bxc1 * bxc1 + bxc2 * bxc2 + bxc3 * bxc3),
                 bbb[9] / std::sqrt(cxa1 * cxa1 + cxa2 * cxa2 + cxa3 * cxa3),
                 bbb[9] / std::sqrt(axb1 * axb1 + axb2 * axb2 + axb3 * axb3)};
  double x[3] = {std::fabs(aaa[0]) / bbb[0], std::fabs(aaa[3]) / bbb[1], std::fabs(aaa[6]) / bbb[2]};
  double y[3] = {std::fabs(aaa[1]) / bbb[0], std::fabs(aaa[4]) / bbb[1], std::fabs(aaa[7]) / bbb[2]};
  if (x[0] >= x[1] && x[0] >= x[2]) {
    bbb[6] = d[0];
    if (y[1] >= y[2]) { bbb[7] = d[1]; bbb[8] = d[2]; } else { bbb[7] = d[2]; bbb[8] = d[1]; }
  } else if (x[1] >= x[0] && x[1] >= x[2]) {
    bbb[6] = d[1];
    if (y[0] >= y[2]) { bbb[7] = d[0]; bbb[8] = d[2]; } else { bbb[7] = d[2]; bbb[8] = d[0]; }
  } else {
    bbb[6] = d[2];
    if (y[0] >= y[1]) { bbb[7] = d[0]; bbb[8] = d[1]; } else { bbb[7] = d[1]; bbb[8] = d[0]; }
  }
}

void invert_host(const double* a, double* b, double* d) {
  b[0] = a[4] * a[8] - a[5] * a[7]; b[1] = a[2] * a[7] - a[1] * a[8]; b[2] = a[1] * a[5] - a[2] * a[4];
  b[3] = a[5] * a[6] - a[3] * a[8]; b[4] = a[0] * a[8] - a[2] * a[6]; b[5] = a[2] * a[3] - a[0] * a[5];
  b[6] = a[3] * a[7] - a[4] * a[6]; b[7] = a[1] * a[6] - a[0] * a[7]; b[8] = a[0] * a[4] - a[1] * a[3];
  *d = a[0] * b[0] + a[3] * b[1] + a[6] * b[2];
  double r = 0.0;
  if (std::fabs(*d) > 0.0) r = 1.0 / *d;
  for (int i = 0; i < 9; ++i) b[i] = r * b[i];
}

// ----------------------------------------------------------- event timers
static const char* kProfNames[P_NPROF] = {"halo",        "bin_sort",   "list_pairs", "short_list", "pair_forces",
                                          "excl_forces", "spme_prep",  "spme_spread", "fft_x_fwd", "fft_y",
                                          "fft_z_conv",  "fft_x_inv",  "spme_gather", "vv",        "shake",
                                          "rattle",      "mlp_infer",  "mts_inputs", "mlp_train",  "coarse_prep",
                                          "coarse_spread", "coarse_fft", "coarse_gather", "metal_density", "metal_forces"};

static int prof_event() {
  if (g.ev_used >= (int)g.evpool.size()) {
    cudaEvent_t e;
    GB_CUDA(cudaEventCreate(&e));
    g.evpool.push_back(e);
  }
  return g.ev_used++;
}

void prof_begin(int id) {
  if (!g.prof_on) return;
  int e = prof_event();
  GB_CUDA(cudaEventRecord(g.evpool[e], g.stream));
  g.open_ev[id] = e;
}

void prof_end(int id) {
  if (!g.prof_on) return;
  int e = prof_event();
  GB_CUDA(cudaEventRecord(g.evpool[e], g.stream));
  g.pend.push_back(id);
  g.pend.push_back(g.open_ev[id]);
  g.pend.push_back(e);
}

// resolve recorded event pairs (the stream has been synchronised)
static void prof_resolve() {
  for (size_t k = 0; k + 2 < g.pend.size(); k += 3) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g.evpool[g.pend[k + 1]], g.evpool[g.pend[k + 2]]);
    g.prof_ms[g.pend[k]] += ms;
    g.prof_n[g.pend[k]] += 1;
  }
  g.pend.clear();
  g.ev_used = 0;
}

void gb_sync_scalars() {
  GB_CUDA(cudaMemcpyAsync(g.hsc, g.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, g.stream));
  GB_CUDA(cudaStreamSynchronize(g.stream));
  if (g.prof_on && !g.pend.empty()) prof_resolve();
}

// register-resident DFMA chains: 8 independent accumulators per thread
__global__ void k_dfma_peak(int iters, double a, double b, double* out) {
  double r0 = threadIdx.x * 1e-9, r1 = r0 + 1e-9, r2 = r0 + 2e-9, r3 = r0 + 3e-9, r4 = r0 + 4e-9, r5 = r0 + 5e-9,
         r6 = r0 + 6e-9, r7 = r0 + 7e-9;
  for (int k = 0; k < iters; ++k) {
    r0 = fma(r0, a, b); r1 = fma(r1, a, b); r2 = fma(r2, a, b); r3 = fma(r3, a, b);
    r4 = fma(r4, a, b); r5 = fma(r5, a, b); r6 = fma(r6, a, b); r7 = fma(r7, a, b);
  }
  double s = r0 + r1 + r2 + r3 + r4 + r5 + r6 + r7;
  if (s == 12345.678) out[0] = s;  // keeps the loop alive
}

double* gb_blkacc(int n) {
  double*& buf = g.side ? g.blkacc_s : g.blkacc;
  int& cap = g.side ? g.blkacc_s_n : g.blkacc_n;
  if (n > cap) {
    if (buf) {
      GB_CUDA(cudaDeviceSynchronize());
      cudaFree(buf);
    }
    cap = n + 4096;
    GB_CUDA(cudaMalloc(&buf, sizeof(double) * cap));
  }
  return buf;
}

void run_side_hook() {
  if (!g.side_hook) return;
  void (*h)(void*) = g.side_hook;
  g.side_hook = nullptr;
  h(g.side_hook_arg);
}

void side_join() {
  if (!g.join_pending) return;
  GB_CUDA(cudaStreamWaitEvent(g.stream, g.ev_join, 0));
  g.join_pending = false;
}

void gb_reduce_blocks(const double* blk, int nblocks_, int nv, double* out_dev) {
  k_reduce_blocks<<<nv, 256, 0, g.stream>>>(blk, nblocks_, nv, out_dev);
  GB_LAUNCHED();
}

// Up to 20 block sums per lane of the last block: it adds about 3 us to the kernel, where the
// launch behind it takes 3.6 and a gap; a lane with 42 (336 blocks of 64 threads) adds 6 us.
GridSum gb_grid_sum(int nb, int nt, int nv, double* out_dev) {
  const int rows = nt / (nv <= 1 ? 1 : nv <= 2 ? 2 : nv <= 4 ? 4 : nv <= 8 ? 8 : 16);
  return {nb <= 20 * std::max(rows, 1) ? (g.side ? &g.sc->count_s : &g.sc->count) : nullptr, out_dev};
}

unsigned long long* stamp_at(int k) { return g.time_regions ? &g.sc->t_ns[k] : nullptr; }

// (a mask of 0, and no load, for bits that this system's kernels never set)
StopIf stop_if(int mask) {
  const int can = (g.ntcons > 0 ? ST_RATTLE_FAIL : 0) | (g.has_metal ? ST_STOP2 : 0);
  return {&g.sc->status, g.defer_scalars ? mask & can : 0};
}

void gb_grid_sum_done(const GridSum& gs, const double* blk, int nb, int nv) {
  if (!gs.count) gb_reduce_blocks(blk, nb, nv, gs.out);
}

int* gb_scan_scratch(int n) {
  int*& buf = g.side ? d_scratch_s : d_scratch;
  size_t& cap = g.side ? d_scratch_s_n : d_scratch_n;
  if ((size_t)n > cap) {
    if (buf) {
      GB_CUDA(cudaDeviceSynchronize());
      cudaFree(buf);
    }
    cap = (size_t)n + 4096;
    GB_CUDA(cudaMalloc(&buf, sizeof(int) * cap));
  }
  return buf;
}

void scan_exclusive(const int* in, int* out, int n) {
  k_scan_excl<<<1, 1024, 0, g.stream>>>(in, out, n);
  GB_LAUNCHED();
}

// ================================================================== C-ABI
extern "C" {

int gb_init(const gb_params* prm, int natms, const int32_t* ltype, const double* chge, const double* weight,
            const int32_t* lfrzn, const double* vdw_prm, int ntcons, const int32_t* listcon, const double* prmcon,
            const int32_t* list_excl) {
  if (!prm || natms <= 0 || !ltype || !chge || !weight || !vdw_prm) return GB_ERR_ARG;
  if (g.init) free_all();
  try {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return GB_ERR_NO_DEVICE;
    if (prm->device < 0 || prm->device >= ndev) return GB_ERR_ARG;
    if (prm->mxnode > 1) return GB_ERR_MULTI_RANK;  // one rank, one GPU: no domain decomposition
    GB_CUDA(cudaSetDevice(prm->device));
    cudaDeviceProp prop;
    GB_CUDA(cudaGetDeviceProperties(&prop, prm->device));
    g.nsm = prop.multiProcessorCount;
    g.p = *prm;
    g.natms = natms;
    g.mxatms = std::max(prm->mxatms, natms);
    if (prm->precision < GB_FP64 || prm->precision > GB_FP64_NATIVE) return GB_ERR_ARG;
    if (!(prm->tstep > 0.0)) return GB_ERR_ARG;
    g.precision = prm->precision == GB_MIXED ? GB_MIXED : GB_FP64;
    g.fp64_native = prm->precision == GB_FP64_NATIVE;
    std::memcpy(g.cell, prm->cell, sizeof(g.cell));
    double det;
    invert_host(g.cell, g.rcell, &det);
    dcell_host(g.cell, g.celprp);
    g.volm = g.celprp[9];
    {
      // the box with its halo within 62 bits, listed separations within 52 (fix_diff)
      const int box = (int)std::ceil(std::log2(1.5 * std::max(g.cell[0], 1.0)));
      const int sep = (int)std::ceil(std::log2(prm->rcut + 2.0 * prm->rpad + 1.0));
      g.pos_scale = std::ldexp(1.0, std::min(48, std::min(62 - box, 52 - sep)));
    }
    g.cubic = (g.cell[0] == g.cell[4] && g.cell[0] == g.cell[8]);
    bool ortho = g.cell[1] == 0 && g.cell[2] == 0 && g.cell[3] == 0 && g.cell[5] == 0 && g.cell[6] == 0 && g.cell[7] == 0;
    if (!ortho || !g.cubic) { free_all(); return GB_ERR_ARG; }  // cubic cells (imcon 1) only
    g.rcutx = prm->rcut + prm->rpad;
    if (g.rcutx >= std::min(g.celprp[6], std::min(g.celprp[7], g.celprp[8])) / 2.0) { free_all(); return GB_ERR_CUTOFF_CELL; }
    {
      int lo = 0, hi = 0;
      GB_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
      GB_CUDA(cudaStreamCreateWithPriority(&g.main_stream, cudaStreamNonBlocking, lo));
      GB_CUDA(cudaStreamCreateWithPriority(&g.side_stream, cudaStreamNonBlocking, hi));
      g.stream = g.main_stream;
      GB_CUDA(cudaEventCreateWithFlags(&g.ev_fork, cudaEventDisableTiming));
      GB_CUDA(cudaEventCreateWithFlags(&g.ev_join, cudaEventDisableTiming));
    }
    for (int k = 0; k < 8; ++k) GB_CUDA(cudaEventCreate(&g.ev[k]));
    const int mx = g.mxatms;
    dalloc(&g.x, mx); dalloc(&g.y, mx); dalloc(&g.z, mx);
    dalloc(&g.xf, mx);
    dalloc(&g.xlo, mx);
    dalloc(&g.qdf, mx);
    dalloc(&g.fx, natms); dalloc(&g.fy, natms); dalloc(&g.fz, natms);
    dalloc(&g.fixp, 3 * (size_t)mx);  // the double-float pair kernel also holds halo-image forces here
    dalloc(&g.vx, natms); dalloc(&g.vy, natms); dalloc(&g.vz, natms);
    dalloc(&g.chge, mx); dalloc(&g.weight, mx);
    dalloc(&g.ltype, mx); dalloc(&g.ltg, mx); dalloc(&g.lfrzn, mx);
    dalloc(&g.ixyz, mx); dalloc(&g.src, mx); dalloc(&g.shcode, mx);
    dalloc(&g.xbg, natms); dalloc(&g.ybg, natms); dalloc(&g.zbg, natms);
    dalloc(&g.ox, natms); dalloc(&g.oy, natms); dalloc(&g.oz, natms);
    dalloc(&g.which_cell, mx); dalloc(&g.at_list, mx); dalloc(&g.sorted_pos, mx);
    dalloc(&g.xs, mx); dalloc(&g.xsf, mx + 8);
    g.ld = prm->max_list + 4;
    dalloc(&g.list, (size_t)g.ld * natms);
    g.ldt = ((prm->max_list + 1 + 3) / 4) * 4;  // spos(k, i), k = 1..max_list, rows 16-byte aligned
    dalloc(&g.spos, (size_t)g.ldt * natms);
    dalloc(&g.xhs, mx); dalloc(&g.rec, mx); dalloc(&g.xlh, mx);
    dalloc(&g.loc_sp, natms);
    dalloc(&g.fixs, 3 * (size_t)mx + 1);
    dalloc(&g.eat, 4 * (size_t)natms);
    dalloc(&g.sc, 1);
    GB_CUDA(cudaMallocHost(&g.hsc, sizeof(DevScalars)));
    std::memset(g.hsc, 0, sizeof(DevScalars));
    GB_CUDA(cudaHostAlloc(&g.hflag, sizeof(int), cudaHostAllocMapped));
    GB_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&g.dflag), g.hflag, 0));
    *g.hflag = 0;
    // topology
    std::vector<int> ltg(natms);
    g.megfrz = 0;
    for (int i = 0; i < natms; ++i) { ltg[i] = i + 1; if (lfrzn && lfrzn[i]) g.megfrz++; }
    GB_CUDA(cudaMemcpy(g.ltg, ltg.data(), sizeof(int) * natms, cudaMemcpyHostToDevice));
    GB_CUDA(cudaMemcpy(g.ltype, ltype, sizeof(int) * natms, cudaMemcpyHostToDevice));
    GB_CUDA(cudaMemcpy(g.chge, chge, sizeof(double) * natms, cudaMemcpyHostToDevice));
    GB_CUDA(cudaMemcpy(g.weight, weight, sizeof(double) * natms, cudaMemcpyHostToDevice));
    {
      std::vector<double> hdw(natms);
      const double hstep = 0.5 * prm->tstep;
      for (int i = 0; i < natms; ++i) hdw[i] = weight[i] > 1.0e-6 ? hstep / weight[i] : 0.0;
      dalloc(&g.hdw, natms);
      GB_CUDA(cudaMemcpy(g.hdw, hdw.data(), sizeof(double) * natms, cudaMemcpyHostToDevice));
    }
    if (lfrzn) GB_CUDA(cudaMemcpy(g.lfrzn, lfrzn, sizeof(int) * natms, cudaMemcpyHostToDevice));
    const int ldx = prm->max_exclude + 1;
    dalloc(&g.list_excl, (size_t)ldx * natms);
    g.lbook = false;
    if (list_excl) {
      GB_CUDA(cudaMemcpy(g.list_excl, list_excl, sizeof(int) * (size_t)ldx * natms, cudaMemcpyHostToDevice));
      for (int i = 0; i < natms; ++i) if (list_excl[(size_t)i * ldx] > 0) { g.lbook = true; break; }
    }
    // tables and constants
    g.nsamples = std::max(1004, (int)std::lround(prm->rcut / 0.01) + 4);   // bounds.F90:811
    g.max_grid = std::max(1004, (int)std::lround(prm->rvdw / 0.01) + 4);   // bounds.F90:820
    build_tables(vdw_prm);
    pair_setup();
    g.scaling = kR4pie0 / prm->epsq;
    double sq2 = 0.0, qmax = 0.0;
    for (int i = 0; i < natms; ++i) {
      sq2 += chge[i] * chge[i];
      qmax = std::max(qmax, std::fabs(chge[i]));
    }
    // an atom's exclusion forces within a quarter of the sums' range, 2^63 units of 2^-40
    g.excl_fixed = 0.43 * std::fabs(g.scaling) * prm->alpha * prm->alpha * qmax * qmax *
                       std::max(prm->max_exclude, 1) < 2097152.0;
    g.self_interaction = -sq2 * (g.scaling * prm->alpha * (1.0 / 1.7724538509055161040) / 1.0);  // spme.F90:159-231
    g.ntcons = ntcons;
    if (ntcons > 0) integ_setup_constraints(listcon, prmcon);
    mts_set_topology(ntcons, listcon, weight);
    g.has_coul = sq2 > 0.0;   // SPME on (electro%key == ELECTROSTATIC_SPME) only with charges
    list_setup();
    g.has_coul = sq2 > 0.0;
    g.has_vdw = false;
    for (int k = 0; k < g.nkey; ++k) g.has_vdw = g.has_vdw || g.h_vdw_kind[k] != 0;
    g.has_metal = false;
    if (g.has_coul) spme_setup();  // an uncharged system has no electrostatics to set up
    g.nstep = 0;
    {
      const char* e = getenv("GB_PAIR_SORTED");
      g.use_sorted = !(e && e[0] == '0');
      const char* d = getenv("GB_MD_DEFER");  // 0: the MD loop reads every step's sums at the step
      g.use_deferred = !(d && d[0] == '0');
      const char* m = getenv("GB_MAPPED_COPY");  // 0: state transfers by cudaMemcpyAsync only
      g.use_mapped = !(m && m[0] == '0');
      const char* o = getenv("GB_OVERLAP");  // 0: SPME and the pair kernel on one stream
      g.use_overlap = !(o && o[0] == '0');
      const char* gr = getenv("GB_GRAPHS");  // 0: the MD loop's kernels launched one by one
      g.use_graphs = !(gr && gr[0] == '0');
      const char* t = getenv("GB_PAIR_NT");  // 256 / 1024: CTA size of the sorted pair kernels (else by form)
      g.pair_nt = t ? ((atoi(t) == 256) ? 256 : 1024) : 0;
      const char* w = getenv("GB_PAIR_APW");
      g.pair_apw = w ? std::max(0, atoi(w)) : -1;
    }
    thermo_setup(GB_NVE, 0.0, 0.0, 0.0, nullptr, 0.0);
    g.init = true;
    g.launches = 0;
    return GB_OK;
  } catch (int e) {
    free_all();
    return e;
  }
}

int gb_upload_state(const double* x, const double* y, const double* z, const double* vx, const double* vy,
                    const double* vz) {
  return guarded([&]() {
    const size_t b = sizeof(double) * g.natms;
    if (!x || !y || !z) return (int)GB_ERR_ARG;
    const bool with_v = vx && vy && vz;
    const int narr = with_v ? 6 : 3;
    const double* src[6] = {x, y, z, vx, vy, vz};
    double* dst[6] = {g.x, g.y, g.z, g.vx, g.vy, g.vz};
    HostArrays a{};
    a.n = g.natms;
    bool mapped = g.use_mapped && g.natms > 0;
    for (int k = 0; k < narr && mapped; ++k) {
      a.h[k] = mapped_span(src[k], g.natms);
      a.d[k] = dst[k];
      mapped = a.h[k] != nullptr;
    }
    *g.hflag = 0;
    if (mapped) {
      k_upload_state<<<copy_grid(g.natms), 256, 0, g.stream>>>(a, narr, g.dflag);
      GB_LAUNCHED();
    } else {
      for (int k = 0; k < narr; ++k)
        GB_CUDA(cudaMemcpyAsync(dst[k], src[k], b, cudaMemcpyHostToDevice, g.stream));
      if (g.natms > 0) {
        k_nonfinite<<<nblocks(g.natms, 256), 256, 0, g.stream>>>(g.natms, g.x, g.y, g.z, g.dflag);
        GB_LAUNCHED();
      }
    }
    GB_CUDA(cudaStreamSynchronize(g.stream));
    if (*static_cast<volatile int*>(g.hflag) & ST_NONFINITE) return (int)GB_ERR_NONFINITE;
    return (int)GB_OK;
  });
}

int gb_upload_parts(const void* parts, const double* vx, const double* vy, const double* vz) {
  return guarded([&]() {
    if (!parts) return (int)GB_ERR_ARG;
    unsigned char* d = nullptr;
    GB_CUDA(cudaMalloc(&d, (size_t)64 * g.natms));
    GB_CUDA(cudaMemcpy(d, parts, (size_t)64 * g.natms, cudaMemcpyHostToDevice));
    k_gather_parts<<<nblocks(g.natms, 256), 256, 0, g.stream>>>(g.natms, d, g.x, g.y, g.z);
    GB_LAUNCHED();
    GB_CUDA(cudaStreamSynchronize(g.stream));
    cudaFree(d);
    const size_t b = sizeof(double) * g.natms;
    if (vx && vy && vz) {
      GB_CUDA(cudaMemcpy(g.vx, vx, b, cudaMemcpyHostToDevice));
      GB_CUDA(cudaMemcpy(g.vy, vy, b, cudaMemcpyHostToDevice));
      GB_CUDA(cudaMemcpy(g.vz, vz, b, cudaMemcpyHostToDevice));
    }
    return (int)GB_OK;
  });
}

int gb_download_state(double* x, double* y, double* z, double* vx, double* vy, double* vz, double* fx, double* fy,
                      double* fz) {
  return guarded([&]() {
    const size_t b = sizeof(double) * g.natms;
    double* dst[9] = {x, y, z, vx, vy, vz, fx, fy, fz};
    double* src[9] = {g.x, g.y, g.z, g.vx, g.vy, g.vz, g.fx, g.fy, g.fz};
    HostArrays a{};
    a.n = g.natms;
    bool mapped = g.use_mapped && g.natms > 0;
    for (int k = 0; k < 9 && mapped; ++k) {
      if (!dst[k]) continue;
      a.h[k] = mapped_span(dst[k], g.natms);
      a.d[k] = src[k];
      mapped = a.h[k] != nullptr;
    }
    if (mapped) {
      k_download_state<<<copy_grid(g.natms), 256, 0, g.stream>>>(a);
      GB_LAUNCHED();
    } else {
      for (int k = 0; k < 9; ++k)
        if (dst[k]) GB_CUDA(cudaMemcpyAsync(dst[k], src[k], b, cudaMemcpyDeviceToHost, g.stream));
    }
    GB_CUDA(cudaStreamSynchronize(g.stream));
    return (int)GB_OK;
  });
}

int gb_download_parts(void* parts, double* vx, double* vy, double* vz) {
  return guarded([&]() {
    if (!parts) return (int)GB_ERR_ARG;
    const int n = g.natms;
    std::vector<double> a(7 * (size_t)n);
    double* p[7] = {&a[0], &a[n], &a[2 * (size_t)n], &a[3 * (size_t)n], &a[4 * (size_t)n], &a[5 * (size_t)n],
                    &a[6 * (size_t)n]};
    const size_t b = sizeof(double) * n;
    GB_CUDA(cudaMemcpy(p[0], g.x, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[1], g.y, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[2], g.z, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[3], g.fx, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[4], g.fy, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[5], g.fz, b, cudaMemcpyDeviceToHost));
    GB_CUDA(cudaMemcpy(p[6], g.chge, b, cudaMemcpyDeviceToHost));
    unsigned char* out = static_cast<unsigned char*>(parts);
    for (int i = 0; i < n; ++i) {
      double* r = reinterpret_cast<double*>(out + (size_t)i * 64);
      for (int k = 0; k < 7; ++k) r[k] = p[k][i];
    }
    if (vx) GB_CUDA(cudaMemcpy(vx, g.vx, b, cudaMemcpyDeviceToHost));
    if (vy) GB_CUDA(cudaMemcpy(vy, g.vy, b, cudaMemcpyDeviceToHost));
    if (vz) GB_CUDA(cudaMemcpy(vz, g.vz, b, cudaMemcpyDeviceToHost));
    return (int)GB_OK;
  });
}

int gb_relocate(void) {
  return guarded([&]() { return list_relocate_and_halo(); });
}

int gb_list_build(int32_t* list_out, int ldlist, int32_t* max_list_io) {
  return guarded([&]() {
    GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
    int st = list_build();
    if (st == GB_ERR_LIST_OVERFLOW) {
      if (max_list_io) *max_list_io = g.hsc->ibig;
      return st;
    }
    if (st) return st;
    if (list_out) {
      if (ldlist != g.ld) return (int)GB_ERR_ARG;
      GB_CUDA(cudaMemcpy(list_out, g.list, sizeof(int) * (size_t)g.ld * g.natms, cudaMemcpyDeviceToHost));
    }
    return (int)GB_OK;
  });
}

int gb_vnl_check(int32_t* update) {
  return guarded([&]() {
    int u = integ_vnl_check();
    if (update) *update = u;
    return (int)GB_OK;
  });
}

int gb_refresh(int32_t* update) {
  return guarded([&]() { return do_refresh(update); });
}

int gb_forces(double* eng_out, double* stress_out) {
  return guarded([&]() { return compute_forces(eng_out, stress_out, true, true); });
}

int gb_spme(double* eng_rc, double* vir_rc, double* stress_out) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    double e8[8], s9[9];
    int st = compute_forces(e8, s9, true, false);
    if (eng_rc) *eng_rc = e8[0];
    if (vir_rc) *vir_rc = e8[1];
    if (stress_out) for (int k = 0; k < 9; ++k) stress_out[k] = s9[k];
    return st;
  });
}

int gb_real(double* eng_out, double* stress_out) {
  return guarded([&]() {
    double e8[8], s9[9];
    int st = compute_forces(e8, s9, false, true);
    if (eng_out) for (int k = 0; k < 6; ++k) eng_out[k] = e8[2 + k];
    if (stress_out) for (int k = 0; k < 9; ++k) stress_out[k] = s9[k];
    return st;
  });
}

int gb_vv(int stage, double* strkin, double* engke, int32_t* iters, double* vircon, double* strcon) {
  return guarded([&]() {
    if (stage != 1 && stage != 2) return (int)GB_ERR_ARG;
    GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
    int it = 0;
    integ_vv(stage, strkin, engke, &it, vircon, strcon);
    if (iters) *iters = it;
    return (int)GB_OK;
  });
}

int gb_constraints_tags(void) {
  return guarded([&]() {
    integ_con_tags();
    return (int)GB_OK;
  });
}

int gb_shake(int32_t* iters, double* vircon, double* strcon) {
  return guarded([&]() {
    GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
    int it = 0;
    integ_shake(&it, vircon, strcon);
    if (iters) *iters = it;
    return (int)GB_OK;
  });
}

int gb_rattle(int32_t* iters) {
  return guarded([&]() {
    GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
    integ_rattle_launch(false);
    gb_sync_scalars();
    if (iters) *iters = g.ntcons > 0 ? g.hsc->rattle_iters : 0;
    if (g.ntcons > 0 && (g.hsc->status & ST_RATTLE_FAIL)) return (int)GB_ERR_RATTLE;
    return (int)GB_OK;
  });
}

int gb_set_ensemble(int kind, double temp, double tau_t, double chi, const int32_t* seed, double degfre) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    if (kind < GB_NVE || kind > GB_NVT_LANGEVIN) return (int)GB_ERR_ARG;
    if (kind != GB_NVE && !(temp > 0.0)) return (int)GB_ERR_ARG;
    if ((kind == GB_NVT_BERENDSEN || kind == GB_NVT_NOSE_HOOVER) && !(tau_t > 0.0)) return (int)GB_ERR_ARG;
    if (kind == GB_NVT_LANGEVIN && !(chi >= 0.0)) return (int)GB_ERR_ARG;
    thermo_setup(kind, temp, tau_t, chi, seed, degfre);
    return (int)GB_OK;
  });
}

int gb_set_step(int32_t nstep) {
  if (!g.init) return GB_ERR_NOT_INIT;
  g.nstep = nstep;
  return GB_OK;
}

int gb_thermostat_state(double* chi_t, double* cint, double* consv) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    thermo_state(chi_t, cint, consv);
    return (int)GB_OK;
  });
}

int gb_set_thermostat_state(double chi_t, double cint) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    thermo_set_state(chi_t, cint);
    return (int)GB_OK;
  });
}

int gb_rng_eval(int mode, int n, const int64_t* a, const int64_t* b, const int64_t* c, double* out) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    if ((mode != 0 && mode != 1) || n < 0 || (n > 0 && (!a || !b || !c || !out))) return (int)GB_ERR_ARG;
    GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
    rng_eval(mode, n, a, b, c, out);
    gb_sync_scalars();
    return (g.hsc->status & ST_RNG) ? (int)GB_ERR_RNG : (int)GB_OK;
  });
}

int gb_set_metal_eam(int ntab, const int32_t* kind, const int32_t* t1, const int32_t* t2, const int32_t* ngrid,
                     const double* start, const double* finish, const double* values, const int32_t* listed) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    if (ntab < 0 || (ntab > 0 && (!kind || !t1 || !t2 || !ngrid || !start || !finish || !values)))
      return (int)GB_ERR_ARG;
    if (g.precision == GB_MIXED) return (int)GB_ERR_ARG;
    if (ntab == 0) { metal_free(); return (int)GB_OK; }
    return metal_setup(ntab, kind, t1, t2, ngrid, start, finish, values, listed);
  });
}

int gb_metal_energies(double* out4) {
  if (!g.init) return GB_ERR_NOT_INIT;
  if (!out4) return GB_ERR_ARG;
  for (int k = 0; k < 4; ++k) out4[k] = g.metal_e4[k];
  return GB_OK;
}

int gb_metal_rho(double* out) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    if (!out || !g.has_metal) return (int)GB_ERR_ARG;
    metal_rho(out, g.natms);
    return (int)GB_OK;
  });
}

// the DL_POLY or library code of the status bits that a step's kernels set (0: none)
static int md_status(int status) {
  if (status & ST_SHAKE_FAIL) return GB_ERR_SHAKE;
  if (status & ST_METAL_DENSITY) return GB_ERR_METAL_DENSITY;
  if (status & ST_METAL_TABLE) return GB_ERR_METAL_TABLE;
  if (status & ST_RATTLE_FAIL) return GB_ERR_RATTLE;
  if (status & ST_RNG) return GB_ERR_RNG;
  return GB_OK;
}

static void md_step_stats(const DevScalars* h, int32_t rebuilt, gb_step_stats& S) {
  std::memset(&S, 0, sizeof(S));
  double st[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, e6[6] = {0, 0, 0, 0, 0, 0}, m4[4] = {0, 0, 0, 0};
  if (g.has_coul) spme_scalars(h, &S.engcpe_rc, &S.vircpe_rc, st);
  if (g.has_coul || g.has_vdw) pair_scalars(h, e6, st);
  if (g.has_metal) metal_scalars(h, m4, st);
  S.engcpe_rl = e6[0]; S.vircpe_rl = e6[1]; S.engcpe_ex = e6[2]; S.vircpe_ex = e6[3];
  S.engvdw = e6[4]; S.virvdw = e6[5];
  S.engmet = m4[0] + m4[2];
  S.virmet = m4[1] + m4[3];
  for (int k = 0; k < 9; ++k) S.stress[k] = st[k];
  kin_scalars(h, S.strkin, &S.engke);
  if (g.ens == GB_NVT_NOSE_HOOVER) {
    S.engke = h->th[6];
    S.consv = h->th[7];
  }
  if (g.ntcons > 0) {
    con_scalars(h, &S.vircon, S.strcon);
    S.shake_iters = h->shake_iters;
    S.rattle_iters = h->rattle_iters;
  }
  S.list_rebuilt = rebuilt;
  S.mts_full = 1;
}

// The loop without learned MTS: the host waits only for the Verlet-list decision of each
// step (vnl_check), where it also sees the status bits set since the last one.  A RATTLE or
// metal failure of a step thus ends the call at the next step's decision; the work behind it
// has left the state alone (StopIf), and the step counter goes back to the failing step.  Each
// step's energy, virial and stress sums are
// copied to a pinned ring with the step's other work and turned into gb_step_stats after
// the last step (of RING_STEPS at most, 4 MB: a longer run is taken in parts).  With 3 or more steps the steps run as two CUDA graphs: stage 1 with the
// displacement check (its sums copied to the pinned scalars), then, after the host's
// decision and the halo refresh or the list rebuild that it calls for, the forces (SPME
// forked to the side stream) and stage 2; the second is captured again when a rebuild
// changes the kernels that walk the list.  Langevin's stage 1 is launched (its noise is keyed
// on the step).  In plain NVE the total is the only timing; the other systems' kernels at the
// ends of the regions store the device's clock beside the sums.
constexpr int RING_STEPS = 4096;
static int md_run_deferred(int nsteps, gb_step_stats* stats) {
  if (g.ring_cap < nsteps) {
    if (g.ring) cudaFreeHost(g.ring);
    g.ring = nullptr;
    g.ring_cap = 0;
    GB_CUDA(cudaMallocHost(&g.ring, sizeof(DevScalars) * (size_t)std::max(nsteps, 64)));
    g.ring_cap = std::max(nsteps, 64);
  }
  std::vector<int32_t> rebuilt(nsteps, 0);
  GB_CUDA(cudaEventRecord(g.ev[5], g.stream));
  gb_blkacc(9 * nblocks(g.natms, 256) + 4096);  // (no allocation inside a capture)
  GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
  g.defer_scalars = true;
  const bool plain = g.ntcons == 0 && g.ens == GB_NVE;
  g.time_regions = !plain || g.has_metal;
  auto stage1 = [&]() {
    if (plain) {
      integ_stage1_check();
    } else {
      int it = 0;
      integ_vv(1, nullptr, nullptr, &it, nullptr, nullptr);
      integ_vnl_launch();
    }
    GB_CUDA(cudaMemcpyAsync(g.hsc, g.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, g.stream));
  };
  auto step_rest = [&]() {
    compute_forces(nullptr, nullptr, true, true, true, nullptr);
    int it = 0;
    integ_vv(2, nullptr, nullptr, &it, nullptr, nullptr);
  };
  bool graphs = g.use_graphs && !g.prof_on && nsteps >= 3;
  const bool graph1 = graphs && g.ens != GB_NVT_LANGEVIN && capture_graph(&g.gx_vv1, &g.gl_vv1, stage1);
  if (graphs && g.ens != GB_NVT_LANGEVIN && !graph1) graphs = false;
  bool step_ok = false, step_spos = false;  // gx_step holds the step's rest for this kind of list
  int code = GB_OK, done = 0, last = -1;  // steps to report; last step with sums in the ring
  for (int s = 0; s < nsteps && code == GB_OK; ++s) {
    ++g.nstep;
    if (graph1) launch_graph(g.gx_vv1, g.gl_vv1);
    else stage1();
    GB_CUDA(cudaStreamSynchronize(g.stream));
    if (g.prof_on) gb_sync_scalars();  // resolves the pending profile events
    code = md_status(g.hsc->status & ~ST_RNG);
    if (code != GB_OK) {
      done = s;
      if (!(g.hsc->status & ST_SHAKE_FAIL)) {  // of the step before
        done = std::max(0, s - 1);
        --g.nstep;
      }
      break;
    }
    done = s;
    const int32_t upd = integ_vnl_result();
    rebuilt[s] = upd;
    if (upd) {
      code = list_relocate_and_halo(false);
      if (!code) code = list_build();
      if (code) break;
    } else {
      list_refresh_halo();
    }
    if (graphs && !(step_ok && step_spos == g.spos_valid)) {
      step_ok = capture_graph(&g.gx_step, &g.gl_step, step_rest);
      step_spos = g.spos_valid;
    }
    if (graphs && step_ok) launch_graph(g.gx_step, g.gl_step);
    else step_rest();
    GB_CUDA(cudaMemcpyAsync(&g.ring[s], g.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, g.stream));
    last = s;
    done = s + 1;
    if (g.hsc->status & ST_RNG) break;  // Langevin's noise (stage 1) ends the call after the step
  }
  g.defer_scalars = false;
  const bool regions = g.time_regions;
  g.time_regions = false;
  GB_CUDA(cudaEventRecord(g.ev[6], g.stream));
  GB_CUDA(cudaEventSynchronize(g.ev[6]));
  if (code == GB_OK && last >= 0) {
    code = md_status(g.ring[last].status);
    if (code != GB_OK) done = last;
  }
  float span = 0.f;
  cudaEventElapsedTime(&span, g.ev[5], g.ev[6]);
  if (code == GB_OK) {
    double list = 0.0, forces = 0.0;
    for (int s = 0; regions && s < nsteps; ++s) {
      const unsigned long long* t = g.ring[s].t_ns;
      list += 1e-6 * (double)(t[1] - t[0]);
      forces += 1e-6 * (double)(t[2] - t[1]);
    }
    g.last_ms[0] = list;
    g.last_ms[1] = forces;
    g.last_ms[2] = 0.0;
    g.last_ms[3] = regions ? span - list - forces : 0.0;
    g.last_ms[4] = g.last_ms[5] = span;
  }
  if (stats)
    for (int s = 0; s < done; ++s) md_step_stats(&g.ring[s], rebuilt[s], stats[s]);
  if (last >= 0) {  // the sums of the last evaluation (none of a failed one)
    double st[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int k = 0; k < 4; ++k) g.metal_e4[k] = 0.0;
    if (g.has_metal && !(g.ring[last].status & ST_STOP2)) metal_scalars(&g.ring[last], g.metal_e4, st);
  }
  return code;
}

int gb_md_run(int nsteps, gb_step_stats* stats) {
  return guarded([&]() {
    if (nsteps < 0) return (int)GB_ERR_ARG;
    if (nsteps > 0 && g.use_deferred && !mts_active()) {
      try {
        double ms[6] = {0, 0, 0, 0, 0, 0};
        for (int s = 0; s < nsteps; s += RING_STEPS) {
          const int code = md_run_deferred(std::min(RING_STEPS, nsteps - s), stats ? stats + s : nullptr);
          if (code != GB_OK) return code;
          for (int k = 0; k < 6; ++k) ms[k] += g.last_ms[k];
        }
        for (int k = 0; k < 6; ++k) g.last_ms[k] = ms[k];
        return (int)GB_OK;
      } catch (int e) {
        g.defer_scalars = g.time_regions = false;
        throw;
      }
    }
    double tl[5] = {0, 0, 0, 0, 0};
    GB_CUDA(cudaEventRecord(g.ev[5], g.stream));
    for (int s = 0; s < nsteps; ++s) {
      gb_step_stats S;
      std::memset(&S, 0, sizeof(S));
      GB_CUDA(cudaMemsetAsync(&g.sc->status, 0, sizeof(int), g.stream));
      GB_CUDA(cudaEventRecord(g.ev[0], g.stream));
      ++g.nstep;  // flow%step of this step (drivers.F90 advances it before stage 1)
      int it = 0;
      integ_vv(1, nullptr, nullptr, &it, &S.vircon, S.strcon);
      S.shake_iters = it;
      GB_CUDA(cudaEventRecord(g.ev[1], g.stream));
      int32_t upd = 0;
      int st = do_refresh(&upd, true);
      if (st) return st;
      S.list_rebuilt = upd;
      if (upd) {
        st = list_build();
        if (st) return st;
      }
      GB_CUDA(cudaEventRecord(g.ev[2], g.stream));
      double e8[8], s9[9];
      bool full = true;
      compute_forces(e8, s9, true, true, true, &full);
      GB_CUDA(cudaEventRecord(g.ev[3], g.stream));
      S.engcpe_rc = e8[0]; S.vircpe_rc = e8[1]; S.engcpe_rl = e8[2]; S.vircpe_rl = e8[3];
      S.engcpe_ex = e8[4]; S.vircpe_ex = e8[5]; S.engvdw = e8[6]; S.virvdw = e8[7];
      for (int k = 0; k < 9; ++k) S.stress[k] = s9[k];
      integ_vv(2, S.strkin, &S.engke, &it, nullptr, nullptr);
      S.rattle_iters = it;
      S.mts_full = full ? 1 : 0;
      S.consv = g.ens == GB_NVT_NOSE_HOOVER ? g.hsc->th[7] : 0.0;
      S.engmet = g.metal_e4[0] + g.metal_e4[2];
      S.virmet = g.metal_e4[1] + g.metal_e4[3];
      GB_CUDA(cudaEventRecord(g.ev[4], g.stream));
      GB_CUDA(cudaEventSynchronize(g.ev[4]));
      float ms;
      cudaEventElapsedTime(&ms, g.ev[1], g.ev[2]); tl[0] += ms;
      cudaEventElapsedTime(&ms, g.ev[2], g.ev[3]); tl[1] += ms;
      cudaEventElapsedTime(&ms, g.ev[0], g.ev[1]); tl[3] += ms;
      cudaEventElapsedTime(&ms, g.ev[3], g.ev[4]); tl[3] += ms;
      cudaEventElapsedTime(&ms, g.ev[0], g.ev[4]); tl[4] += ms;
      if (stats) stats[s] = S;
    }
    GB_CUDA(cudaEventRecord(g.ev[6], g.stream));
    GB_CUDA(cudaEventSynchronize(g.ev[6]));
    float span = 0.f;
    cudaEventElapsedTime(&span, g.ev[5], g.ev[6]);
    for (int k = 0; k < 5; ++k) g.last_ms[k] = tl[k];
    g.last_ms[5] = span;  // device-timeline span of the whole call (includes host gaps)
    return (int)GB_OK;
  });
}

int gb_mts_config(int k, double tol, int train_steps) {
  return guarded([&]() {
    if (!g.init) return (int)GB_ERR_NOT_INIT;
    if (k < 1 || !(tol > 0.0) || train_steps < 0) return (int)GB_ERR_ARG;
    if (k > 1 && g.precision != GB_MIXED) return (int)GB_ERR_ARG;  // the surrogate feeds the fixed-point forces
    if (k > 1 && !g.has_coul) return (int)GB_ERR_ARG;  // it replaces SPME: needs charges
    // the network's neighbour sums reach 6 A: the half list and the halo must hold those pairs
    if (k > 1 && g.p.rcut < MTS_RCUT_DESC) return (int)GB_ERR_ARG;
    g.mts_k = k;
    g.mts_tol = tol;
    g.mts_train = train_steps;
    if (k > 1) mts_setup();
    else mts_free();
    return (int)GB_OK;
  });
}

int gb_set_precision(int precision) {
  return guarded([&]() {
    if (precision < GB_FP64 || precision > GB_FP64_NATIVE) return (int)GB_ERR_ARG;
    if (precision == GB_MIXED && g.has_metal) return (int)GB_ERR_ARG;  // metals run in the FP64 form
    if (precision != GB_MIXED && mts_active()) {  // the learned form runs on the mixed path only
      mts_free();
      g.mts_k = 1;
    }
    g.precision = precision == GB_MIXED ? GB_MIXED : GB_FP64;
    g.fp64_native = precision == GB_FP64_NATIVE;
    return (int)GB_OK;
  });
}

int gb_last_timings(double* ms, int n) {
  if (!ms) return GB_ERR_ARG;
  for (int k = 0; k < n && k < 8; ++k) ms[k] = g.last_ms[k];
  return GB_OK;
}

int64_t gb_kernel_launches(void) { return g.launches; }

int gb_mts_stats(double* out, int n) {
  if (!out || n < 0) return GB_ERR_ARG;
  return guarded([&]() {
    mts_stats(out, n);
    return (int)GB_OK;
  });
}

int gb_mts_features(float* x, int n, float* scales) {
  if (!g.init) return GB_ERR_NOT_INIT;
  return guarded([&]() { return mts_features(x, n, scales); });
}

int gb_mlp_param_count(void) { return mlp_param_count(); }

int gb_mts_ablation(int no_network) {
  if (no_network != 0 && no_network != 1) return GB_ERR_ARG;
  mts_set_no_network(no_network == 1);
  return GB_OK;
}

int gb_mlp_train_eval(int nb, const float* x, const float* target, const float* params, float* loss, float* grad,
                      float* y) {
  if (!g.init) return GB_ERR_NOT_INIT;
  return guarded([&]() { return mlp_train_eval(nb, x, target, params, loss, grad, y); });
}

int gb_mlp_infer_eval(int nb, const float* x, const float* params, float* y) {
  if (!g.init) return GB_ERR_NOT_INIT;
  return guarded([&]() { return mlp_infer_eval(nb, x, params, y); });
}

int gb_profile(int enable) {
  return guarded([&]() {
    GB_CUDA(cudaStreamSynchronize(g.stream));
    g.pend.clear();
    g.ev_used = 0;
    for (int k = 0; k < P_NPROF; ++k) { g.prof_ms[k] = 0.0; g.prof_n[k] = 0; }
    g.prof_on = enable != 0;
    return (int)GB_OK;
  });
}

int gb_set_overlap(int enable) {
  return guarded([&]() {
    g.use_overlap = enable != 0;
    return (int)GB_OK;
  });
}

int gb_profile_read(char* names, double* ms, int64_t* launches, int max) {
  return guarded([&]() {
    GB_CUDA(cudaStreamSynchronize(g.stream));
    if (!g.pend.empty()) prof_resolve();
    int n = 0;
    for (int k = 0; k < P_NPROF && n < max; ++k, ++n) {
      if (names) { std::memset(names + 32 * n, 0, 32); std::strncpy(names + 32 * n, kProfNames[k], 31); }
      if (ms) ms[n] = g.prof_ms[k];
      if (launches) launches[n] = g.prof_n[k];
    }
    return n;
  });
}

int gb_pair_counts(int64_t* out, int n) {
  return guarded([&]() {
    gb_sync_scalars();
    int64_t v[8] = {(int64_t)g.hsc->npairs_list, (int64_t)g.hsc->npairs_rc, (int64_t)g.hsc->ncand_fp64,
                    (int64_t)g.hsc->halo_fwd, (int64_t)g.hsc->halo_bwd,
                    (int64_t)(g.spos_valid && g.use_sorted), (int64_t)g.n_tile_over, (int64_t)g.tp.m};
    for (int k = 0; k < n && k < 8; ++k) out[k] = v[k];
    return (int)GB_OK;
  });
}

double gb_fp64_peak_tflops(void) {
  try {
    int dev = g.init ? g.p.device : 0;
    GB_CUDA(cudaSetDevice(dev));
    cudaDeviceProp prop;
    GB_CUDA(cudaGetDeviceProperties(&prop, dev));
    double* out = nullptr;
    GB_CUDA(cudaMalloc(&out, sizeof(double)));
    cudaEvent_t a, b;
    GB_CUDA(cudaEventCreate(&a));
    GB_CUDA(cudaEventCreate(&b));
    const int blocks = prop.multiProcessorCount * 8, threads = 256, iters = 4096;
    k_dfma_peak<<<blocks, threads>>>(iters, 0.999999, 1e-7, out);  // warm-up
    GB_CUDA(cudaGetLastError());
    GB_CUDA(cudaEventRecord(a));
    for (int r = 0; r < 5; ++r) k_dfma_peak<<<blocks, threads>>>(iters, 0.999999, 1e-7, out);
    GB_CUDA(cudaEventRecord(b));
    GB_CUDA(cudaEventSynchronize(b));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    double flops = 5.0 * 2.0 * 8.0 * (double)iters * blocks * threads;
    return flops / (ms * 1e-3) / 1e12;
  } catch (int) {
    return -1.0;
  }
}

void gb_finalize(void) {
  if (g.init || g.stream) free_all();
}

const char* gb_strerror(int status) {
  switch (status) {
    case GB_OK: return "success";
    case GB_ERR_CUTOFF_CELL: return "cutoff_extended >= half of the minimum cell width (error 95)";
    case GB_ERR_SHAKE: return "SHAKE did not converge (error 105)";
    case GB_ERR_LIST_OVERFLOW: return "Verlet list overflow, max_list too small (error 106)";
    case GB_ERR_LINK_CELLS: return "link cells per domain < 1 (error 307)";
    case GB_ERR_UNSAFE: return "unsafe state (error 505)";
    case GB_ERR_RATTLE: return "RATTLE did not converge (error 515)";
    case GB_ERR_HALO: return "halo exceeds mxatms (error 56)";
    case GB_ERR_NOT_INIT: return "library not initialised (gb_init)";
    case GB_ERR_CUDA: return "CUDA runtime error";
    case GB_ERR_ARG: return "invalid argument";
    case GB_ERR_NO_DEVICE: return "no CUDA device";
    case GB_ERR_NONFINITE: return "non-finite positions";
    case GB_ERR_METAL_TABLE: return "metal table read below its first point (error 506)";
    case GB_ERR_METAL_DENSITY: return "local density outside its embedding table (error 507)";
    case GB_ERR_RNG: return "a Gaussian deviate's rejection loop hit its iteration cap";
    case GB_ERR_DEVICE_WAIT: return "a tensor-core completion wait hit its iteration limit";
    case GB_ERR_MULTI_RANK: return "more than one MPI rank (comm%mxnode > 1): the device path runs one rank on one GPU";
    case GB_ERR_TOO_LARGE: return "more atoms than gb_kinstress_noalloc takes (1,048,576)";
    default: return "unknown status";
  }
}

}  // extern "C"
