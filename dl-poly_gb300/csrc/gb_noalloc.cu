// gb_noalloc.cu - kinetic stress (kinstress, source/kinetics.F90:218-262) for
// callers that cannot allocate device memory.
//
// Some host programs cannot call cudaMalloc at the point where they need the
// kinetic stress: a driver that has handed its whole device-memory budget to
// a pool owned by another framework, or code that runs where allocation is not
// permitted (for example a step that must not change the device memory
// footprint once a long run has started).  gb_kinstress_noalloc serves them:
// it takes device pointers for its inputs and its output and allocates
// nothing.  Its per-block partial sums live in the file-scope array below,
// which every GPU that loads this library holds until the process exits.
#include "gb_common.cuh"

namespace {

constexpr int KIN_THREADS = 256;
constexpr int KIN_MAX_ATOMS = 1048576;  // the entry point's documented limit
constexpr int KIN_BLOCKS = 304;         // most blocks of a call (two for each of 152 SMs)
constexpr int KIN_MAX_DEVICES = 64;

// 6 partial sums per block, then the 6 sums, then the number of blocks that are done.
static __device__ __align__(256) double g_kin_scratch[(KIN_BLOCKS + 1) * 6 + 1];

// Host side: the device address of g_kin_scratch on each device, looked up
// once per device.  (In host code the symbol name itself is only a host-side
// stand-in, never a device address.)
double* g_kin_scratch_addr[KIN_MAX_DEVICES] = {nullptr};

// A grid-stride loop whose last block adds up the blocks' sums: one launch instead of two,
// and one reduction per thread instead of one per atom.  98,304 atoms: 22.5 -> 17 us a call,
// the latency of the launch, of the loads and of the two stages of the sum.  1.5 us of it clear
// the count of the blocks that are done, on the stream before each launch, so that calls which
// overlapped against the rule leave nothing behind for the next.
__global__ void __launch_bounds__(KIN_THREADS) k_kin_sum(int n, const double* __restrict__ w,
                                                         const int* __restrict__ lfrzn, const double* __restrict__ vx,
                                                         const double* __restrict__ vy, const double* __restrict__ vz,
                                                         double* part, double* __restrict__ out) {
  double a[6] = {0, 0, 0, 0, 0, 0};
  const int stride = gridDim.x * blockDim.x;
#pragma unroll 4
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const bool free_atom = lfrzn == nullptr || lfrzn[i] == 0;
    const double m = w[i], u = vx[i], v = vy[i], t = vz[i];
    if (!free_atom) continue;
    const double mu = m * u, mv = m * v;
    a[0] = fma(mu, u, a[0]); a[1] = fma(mu, v, a[1]); a[2] = fma(mu, t, a[2]);
    a[3] = fma(mv, v, a[3]); a[4] = fma(mv, t, a[4]); a[5] = fma(m * t, t, a[5]);
  }
  block_reduce_store<6>(a, part);
  double* sum = part + KIN_BLOCKS * 6;
  const GridSum gs = {reinterpret_cast<unsigned*>(sum + 6), sum};
  if (grid_finish<6>(part, gs) && threadIdx.x < 6) {
    const int at[6] = {0, 1, 2, 4, 5, 8}, mirror[6] = {0, 3, 6, 4, 7, 8};
    out[at[threadIdx.x]] = sum[threadIdx.x];
    out[mirror[threadIdx.x]] = sum[threadIdx.x];
  }
}

}  // namespace

extern "C" int gb_kinstress_noalloc(const double* vx, const double* vy, const double* vz, const double* weight,
                                    const int32_t* lfrzn, int n, double* strkin_out, void* stream) {
  if (n < 0 || !strkin_out || (n > 0 && (!vx || !vy || !vz || !weight))) return GB_ERR_ARG;
  if (n > KIN_MAX_ATOMS) return GB_ERR_TOO_LARGE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= KIN_MAX_DEVICES) return GB_ERR_CUDA;
  if (!g_kin_scratch_addr[dev]) {
    // first call on this device: look up the device address of the scratch array
    double* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_kin_scratch) != cudaSuccess || !p) return GB_ERR_CUDA;
    g_kin_scratch_addr[dev] = p;
  }
  const int nb = n > 0 ? (n + KIN_THREADS - 1) / KIN_THREADS : 1;
  double* part = g_kin_scratch_addr[dev];
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(part + (KIN_BLOCKS + 1) * 6, 0, sizeof(unsigned), st) != cudaSuccess) return GB_ERR_CUDA;
  k_kin_sum<<<nb < KIN_BLOCKS ? nb : KIN_BLOCKS, KIN_THREADS, 0, st>>>(n, weight, lfrzn, vx, vy, vz, part, strkin_out);
  if (cudaGetLastError() != cudaSuccess) return GB_ERR_CUDA;
  return GB_OK;
}
