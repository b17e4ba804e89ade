// Electronic-grid solve that allocates nothing (eph_fdm_solve_noalloc in
// include/eph_gb.h).
//
// Who needs it: callers that own every byte of device memory themselves and
// may not call cudaMalloc/cudaFree during a run -- an MD engine that sizes one
// device pool at start-up and hands out slices of it, or a time-step loop
// that must not synchronise the device (cudaMalloc and cudaFree can).  The
// caller passes every input and output as device pointers; the only other
// memory used is the file-scope array below, reserved when the library is
// loaded and held on every GPU that loads it until the process exits.
//
// Shared scratch: every call uses the same array and leaves the last call's
// contents in it.  Calls whose work overlaps on the GPU (two streams, or two
// threads issuing on different streams) race on it; order them on one stream
// or serialise them.  Nothing in the array has to start at zero: the
// reduction slots and the ping-pong grid are fully written before they are
// read.
#include <atomic>
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "eph_device.cuh"
#include "eph_gb.h"
#include "eph_softfp.cuh"

using namespace ephgb;

namespace {

constexpr int kMaxDevices = 64;

// [0, MAX_CELLS): second temperature buffer (before the substeps: the blocks'
// bounds); [MAX_CELLS, +3): c_min, rho_min, kappa_max of the stability rule.
static __device__ __align__(256) double g_fdm_scratch[EPH_NOALLOC_MAX_CELLS + 8];

// Device address of g_fdm_scratch per device, filled on the first call on
// that device (host code cannot use the symbol itself as an address).  Two
// host threads making their first call on one device at once both look the
// address up and store the same value.
std::atomic<double *> g_scratch_addr[kMaxDevices];

// Blocks of the bounds reduction; each leaves its three bounds in the scratch
// grid (free until the first substep writes it), and the last kernel of the
// two combines them.  One block over all cells took 657 us at 64^3 cells (GB300);
// 128 blocks and a second small launch take ~8 us.
constexpr int kBoundsBlocks = 128;

__device__ __forceinline__ void block_bounds(double c_min, double r_min, double k_max, double *__restrict__ out) {
  __shared__ double s[3][256];
  s[0][threadIdx.x] = c_min;
  s[1][threadIdx.x] = r_min;
  s[2][threadIdx.x] = k_max;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      s[0][threadIdx.x] = fmin(s[0][threadIdx.x], s[0][threadIdx.x + h]);
      s[1][threadIdx.x] = fmin(s[1][threadIdx.x], s[1][threadIdx.x + h]);
      s[2][threadIdx.x] = fmax(s[2][threadIdx.x], s[2][threadIdx.x + h]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = s[0][0];
    out[1] = s[1][0];
    out[2] = s[2][0];
  }
}

__global__ void k_noalloc_bounds(int ntotal, const double *__restrict__ C, const double *__restrict__ rho,
                                 const double *__restrict__ kappa, const signed char *__restrict__ flag,
                                 double *__restrict__ parts) {
  // eph_fdm.h:290-300: start from cell 0 whatever its flag, then every cell
  // that is not CONSTANT_VALUE
  double c_min = C[0], r_min = rho[0], k_max = kappa[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntotal; i += gridDim.x * blockDim.x)
    if (i > 0 && flag[i] != 0) {
      c_min = fmin(c_min, C[i]);
      r_min = fmin(r_min, rho[i]);
      k_max = fmax(k_max, kappa[i]);
    }
  block_bounds(c_min, r_min, k_max, parts + 3 * blockIdx.x);
}

__global__ void k_noalloc_bounds_of(const double *__restrict__ parts, double *__restrict__ out) {
  const double *p = parts + 3 * threadIdx.x;  // one thread per block of k_noalloc_bounds
  block_bounds(p[0], p[1], p[2], out);
}

// x / 4 by the exponent
__device__ __forceinline__ double quarter(double x) {
  const unsigned e = soft::exponent(soft::bits(x));
  return e - 3u < 0x7ffu - 3u ? soft::from_bits(soft::bits(x) - (2ull << 52)) : 0.25 * x;
}

// One substep of EPH_FDM::solve (eph_fdm.h:315-396) in the reference's
// expression order, rounded as it rounds: T_out from T_in.
// The hardware's thirteen quotients per cell made FP64 issue the bound (two
// lanes per SM and clock).  Quotients and products run on the integer units
// instead (the same bits), what the three spacings' quotients share comes from
// the host, and the quarter is an exponent: 22 operations per cell are left to
// the FP64 pipe.  64^3 cells on GB300, us per substep: 71 with the hardware's
// operations, 18 with products by rounded reciprocals (other bits), 19 with the
// quotients on the integer units, 16 with the products too.
__global__ void __launch_bounds__(128)
    k_noalloc_substep(int nx, int ny, int nz, soft::Divisor hx, soft::Divisor hy, soft::Divisor hz, double inner_dt,
                      const double *__restrict__ T, double *__restrict__ Tout, const double *__restrict__ kappa,
                      const double *__restrict__ rho, const double *__restrict__ C, const double *__restrict__ S,
                      const double *__restrict__ dT, const signed char *__restrict__ flag) {
  griddep_launch();
  griddep_wait();
  const int r = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int nxy = nx * ny;
  if (r >= nxy * nz) return;
  const int row = r / nx, i = r - row * nx, k = row / ny, j = row - k * ny;
  const double Tr = T[r];
  double t = Tr;
  if (flag[r] == 1) {
    const int p3[3] = {i > 0 ? r - 1 : r + (nx - 1), j > 0 ? r - nx : r + (nxy - nx),
                       k > 0 ? r - nxy : r + (nz - 1) * nxy};
    const int q3[3] = {i < nx - 1 ? r + 1 : r - (nx - 1), j < ny - 1 ? r + nx : r - (nxy - nx),
                       k < nz - 1 ? r + nxy : r - (nz - 1) * nxy};
    // every load at once; the wall rule then selects values
    double Tq[3], Tp[3], kq[3], kp[3];
    bool wq[3], wp[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      wq[a] = flag[q3[a]] == 2;
      wp[a] = flag[p3[a]] == 2;
      Tq[a] = T[q3[a]];
      Tp[a] = T[p3[a]];
      kq[a] = kappa[q3[a]];
      kp[a] = kappa[p3[a]];
    }
    const double kr = kappa[r], add = dT[r], src = S[r], cap = soft::mul(rho[r], C[r]);
    double ddT = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const soft::Divisor &h = a == 0 ? hx : (a == 1 ? hy : hz);
      const bool sp = wp[a] && !wq[a];
      const double uq = wq[a] ? Tr : Tq[a], up = sp ? Tr : Tp[a];
      const double dk = (wq[a] ? kr : kq[a]) - (sp ? kr : kp[a]);
      ddT += quarter(soft::div(soft::div(soft::mul(dk, uq - up), h), h));
      ddT += soft::mul(kr, soft::div(soft::div(fma(-2.0, Tr, uq + up), h), h));
    }
    t = Tr + soft::mul(soft::div(ddT + add + src, soft::divisor(cap)), inner_dt);
  }
  if (neg_double(t)) t = 0.0;
  Tout[r] = t;
}

}  // namespace

extern "C" int eph_fdm_solve_noalloc(long nx, long ny, long nz, const double *lo, const double *hi, double dt,
                                     long steps, double *T, const double *dT, const double *S, const double *rho_e,
                                     const double *C_e, const double *kappa, const signed char *flag, void *stream,
                                     unsigned *nsub_out) {
  if (nx < 1 || ny < 1 || nz < 1 || !lo || !hi || !(dt > 0) || steps < 1 || !T || !dT || !S || !rho_e || !C_e ||
      !kappa || !flag)
    return EPH_ERR_ARG;
  const long ntotal = nx * ny * nz;
  if (ntotal > EPH_NOALLOC_MAX_CELLS) return EPH_ERR_CAPACITY;  // larger than the static scratch
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return EPH_ERR_CUDA;
  double *scratch = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (!scratch) {
    // set-up, once per device, with that device current
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_fdm_scratch) != cudaSuccess || !p) return EPH_ERR_CUDA;
    scratch = static_cast<double *>(p);
    g_scratch_addr[dev].store(scratch, std::memory_order_release);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // grid spacing as eph_fdm.h:127-146 computes it
  const double dx = (hi[0] - lo[0]) / (double)(size_t)nx;
  const double dy = (hi[1] - lo[1]) / (double)(size_t)ny;
  const double dz = (hi[2] - lo[2]) / (double)(size_t)nz;
  // stability substeps, eph_fdm.h:275-313
  k_noalloc_bounds<<<kBoundsBlocks, 256, 0, st>>>((int)ntotal, C_e, rho_e, kappa, flag, scratch);
  k_noalloc_bounds_of<<<1, kBoundsBlocks, 0, st>>>(scratch, scratch + EPH_NOALLOC_MAX_CELLS);
  double b[3];
  if (cudaMemcpyAsync(b, scratch + EPH_NOALLOC_MAX_CELLS, sizeof b, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return EPH_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return EPH_ERR_CUDA;
  // the reference only asserts positive bounds; here a zero or negative C_e
  // or rho_e (cell 0 enters the minimum whatever its flag) is an argument
  // error, and so is a substep count above EPH_NOALLOC_MAX_SUBSTEPS, before
  // anything is launched
  if (!(b[0] > 0.0) || !(b[1] > 0.0) || !(b[2] >= 0.0)) return EPH_ERR_ARG;
  if (steps > EPH_NOALLOC_MAX_SUBSTEPS) return EPH_ERR_ARG;
  double inner_dt = dt / (double)(size_t)steps;
  const double dtdxdydz = inner_dt * (1.0 / dx / dx + 1.0 / dy / dy + 1.0 / dz / dz);
  const double r = dtdxdydz / b[0] / b[1] * b[2];
  unsigned nsub = (unsigned)steps;
  if (r > 0.4) {
    inner_dt = 0.4 * inner_dt / r;
    const double want = dt / inner_dt;
    if (!(want < (double)EPH_NOALLOC_MAX_SUBSTEPS + 1.0)) return EPH_ERR_ARG;
    const unsigned s = (unsigned)want;
    nsub = s > 1u ? s : 1u;
    inner_dt = dt / nsub;
  }
  const int threads = 128;
  const soft::Divisor hx = soft::divisor(dx), hy = soft::divisor(dy), hz = soft::divisor(dz);
  double *src = T, *dst = scratch;
  for (unsigned s = 0; s < nsub; ++s) {
    // each substep a programmatic dependent of the one before: its launch
    // overlaps that one's tail, and it waits before it touches memory
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((ntotal + threads - 1) / threads));
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = s > 0 ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_noalloc_substep, (int)nx, (int)ny, (int)nz, hx, hy, hz, inner_dt,
                           (const double *)src, dst, kappa, rho_e, C_e, S, dT, flag) != cudaSuccess)
      return EPH_ERR_CUDA;
    double *t = src;
    src = dst;
    dst = t;
  }
  if (src != T && cudaMemcpyAsync(T, src, sizeof(double) * (size_t)ntotal, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return EPH_ERR_CUDA;
  if (cudaGetLastError() != cudaSuccess) return EPH_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return EPH_ERR_CUDA;
  if (nsub_out) *nsub_out = nsub;
  return EPH_OK;
}
