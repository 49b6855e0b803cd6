// gpe_norm_noalloc: the norm reduction of get_norm for callers that own all
// device memory themselves and must not have a library allocate any.
//
// Typical callers: a host whose device memory belongs to another allocator
// (a framework's caching pool, a Fortran runtime that maps its own buffers)
// and may not see foreign cudaMalloc/cudaFree calls; code running between
// steps of a captured or real-time loop where an allocation would stall or
// be illegal; and embedders that budget device memory up front.
//
// The reduction needs scratch space for at least one partial sum per z-plane.  That
// scratch is the file-scope array below, sized for GPE_NOALLOC_MAX_NZ planes
// (64 KiB).  It is part of this library's device image, so every GPU that
// loads the library holds it until the process exits.
//
// Host code must not use the array's name as a device address: on the host
// it is only a stand-in symbol.  The first call on each device, with that
// device current, looks up the real device address with
// cudaGetSymbolAddress and caches it per device; kernels get that pointer.
// The same first call loads all instances of the reduction kernel on
// that device (cudaFuncGetAttributes), so with lazy module loading no later
// call loads code; make it before any stream capture.  The cached address is
// not refreshed after cudaDeviceReset or a primary-context reset, which this
// entry point does not support.
//
// Pointers are checked for the alignment the kernels read and write with
// (16 bytes for complex128 input, 8 for complex64 input and the output
// double) before anything is launched: a misaligned pointer is rejected
// with GPE_ERR_BADARG rather than faulting the caller's context.
//
// All calls share the one array.  Every call overwrites each partial it
// reads before reading it, so nothing has to be cleared between calls, but
// calls whose work overlaps on the GPU (different streams, or different
// host threads on one device) race on the array and must be serialised by
// the caller.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "../../include/gpe_cuda.h"

namespace {

static __device__ __align__(256) double g_norm_scratch[GPE_NOALLOC_MAX_NZ];

constexpr int kMaxDevices = 64;
// device address of g_norm_scratch, per device; written once under g_setup
std::atomic<double*> g_scratch_addr[kMaxDevices];
std::mutex g_setup;

// Extended closed (Numerical Recipes 4.1.14) weights of integrate_x/y/z
// (src/variables.f90:49-51, 730-840): 3/8, 7/6, 23/24 at both ends, 1 inside.
__device__ __forceinline__ double quad_weight(int q, int n) {
  double w = 1.0;
  if (q == 0) w = 3.0 / 8.0;
  if (q == 1) w = 7.0 / 6.0;
  if (q == 2) w = 23.0 / 24.0;
  if (q == n - 3) w = 23.0 / 24.0;
  if (q == n - 2) w = 7.0 / 6.0;
  if (q == n - 1) w = 3.0 / 8.0;
  return w;
}

// Blocks of the plane sums that give every SM several, and the parts a plane
// is cut into for that: never more partials than the scratch holds, and at
// least a row per warp.
constexpr int kThreads = 256;
constexpr int kBlocks = 148 * 8;
int plane_parts(int ny, int nz) {
  int parts = (kBlocks + nz - 1) / nz;
  if (parts > GPE_NOALLOC_MAX_NZ / nz) parts = GPE_NOALLOC_MAX_NZ / nz;
  if (parts > (ny + kThreads / 32 - 1) / (kThreads / 32)) parts = (ny + kThreads / 32 - 1) / (kThreads / 32);
  return parts < 1 ? 1 : parts;
}

// scratch[k * parts + b] = sum over the b-th share of plane k's rows of
// w_i w_j |psi(i,j,k)|^2, summed in a fixed order (rows to warps round robin,
// lanes along x, then a tree), so results are deterministic.  A warp walks
// whole rows, two at a time: no index division, and a plane is spread over as many blocks as the chip wants.  192 x 192 x 384
// complex128 (216 MiB): 97 us with one 256-thread block per plane and a
// 64-bit division per site, 46 us so (35 at the copy rate).  SITES: rows shorter
// than a warp, whose sites go to threads one by one (6 x 1000 x 1000 complex128
// 98 us by rows, 41 so).
template <class T2, bool SITES>
__global__ void __launch_bounds__(kThreads) k_plane_sums(const T2* __restrict__ psi, int nx, int ny, int parts,
                                                         double* scratch) {
  __shared__ double red[kThreads / 32];
  const int k = blockIdx.x / parts, b = blockIdx.x - k * parts;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j0 = (int)((long long)ny * b / parts), j1 = (int)((long long)ny * (b + 1) / parts);
  double s = 0.0;
  constexpr int kW = kThreads / 32;
  if constexpr (SITES) {
    // a 32-bit division each: a part holds a 1184th of what fits on the device,
    // or a few rows
    const T2* p = psi + ((long long)k * ny + j0) * nx;
    const int n = (j1 - j0) * nx;
#pragma unroll 4
    for (int t = threadIdx.x; t < n; t += kThreads) {
      const int j = t / nx;
      const T2 v = p[t];
      const double re = (double)v.x, im = (double)v.y;
      s += (quad_weight(t - j * nx, nx) * quad_weight(j0 + j, ny)) * (re * re + im * im);
    }
  }
  for (int j = j0 + w; !SITES && j < j1; j += 2 * kW) {
    // two rows at a time: eight loads in flight per lane
    const bool two = j + kW < j1;
    const T2* p = psi + ((long long)k * ny + j) * nx;
    const T2* p2 = two ? p + (long long)kW * nx : p;
    double r = 0.0, r2 = 0.0;
#pragma unroll 4
    for (int i = lane; i < nx; i += 32) {
      const T2 v = p[i], v2 = p2[i];
      const double wx = quad_weight(i, nx);
      const double re = (double)v.x, im = (double)v.y, re2 = (double)v2.x, im2 = (double)v2.y;
      r += wx * (re * re + im * im);
      r2 += wx * (re2 * re2 + im2 * im2);
    }
    s += quad_weight(j, ny) * r;
    if (two) s += quad_weight(j + kW, ny) * r2;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) red[w] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kThreads / 32; ++q) t += red[q];
    scratch[blockIdx.x] = t;
  }
}

// norm = (sum_k w_k sum_b scratch[k parts + b]) * dx * dy * dz into the
// caller's device word.
__global__ void __launch_bounds__(kThreads) k_plane_total(const double* __restrict__ scratch, int nz, int parts,
                                                          double dx, double dy, double dz, double* out) {
  __shared__ double red[kThreads];
  double s = 0.0;
#pragma unroll 4
  for (int q = threadIdx.x; q < nz * parts; q += kThreads) s += quad_weight(q / parts, nz) * scratch[q];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = kThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = ((red[0] * dx) * dy) * dz;
}

int reject(const char* why) {
  fprintf(stderr, "gpe_norm_noalloc: %s\n", why);
  return GPE_ERR_BADARG;
}

// Set-up of the current device (once): the scratch array's device address,
// and the reduction kernels loaded.  Returns nullptr on a CUDA error.
double* scratch_of(int dev) {
  double* p = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (p) return p;
  std::lock_guard<std::mutex> lk(g_setup);
  p = g_scratch_addr[dev].load(std::memory_order_relaxed);
  if (p) return p;
  void* addr = nullptr;
  if (cudaGetSymbolAddress(&addr, g_norm_scratch) != cudaSuccess || !addr) return nullptr;
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, k_plane_sums<double2, false>) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k_plane_sums<double2, true>) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k_plane_sums<float2, false>) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k_plane_sums<float2, true>) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k_plane_total) != cudaSuccess)
    return nullptr;
  p = (double*)addr;
  g_scratch_addr[dev].store(p, std::memory_order_release);
  return p;
}

}  // namespace

extern "C" int gpe_norm_noalloc(const void* psi_dev, int32_t dtype, int32_t nx, int32_t ny, int32_t nz, double dx,
                                double dy, double dz, double* norm_dev, void* stream) {
  if (!psi_dev || !norm_dev) return reject("null device pointer");
  if (dtype != GPE_C128 && dtype != GPE_C64) return reject("dtype must be GPE_C128 or GPE_C64");
  if (nx < 6 || ny < 6 || nz < 6) return reject("nx, ny and nz must be >= 6");
  if (nz > GPE_NOALLOC_MAX_NZ) return reject("nz exceeds GPE_NOALLOC_MAX_NZ (8192 planes of scratch)");
  const uintptr_t in_align = dtype == GPE_C128 ? 16 : 8;
  if ((uintptr_t)psi_dev % in_align != 0)
    return reject(dtype == GPE_C128 ? "psi_dev is not 16-byte aligned (complex128)"
                                    : "psi_dev is not 8-byte aligned (complex64)");
  if ((uintptr_t)norm_dev % 8 != 0) return reject("norm_dev is not 8-byte aligned");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return GPE_ERR_CUDA;
  double* scratch = scratch_of(dev);
  if (!scratch) return GPE_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  const int parts = plane_parts(ny, nz);
  const bool sites = nx < 32;
  if (dtype == GPE_C128)
    (sites ? k_plane_sums<double2, true> : k_plane_sums<double2, false>)<<<nz * parts, kThreads, 0, st>>>(
        (const double2*)psi_dev, nx, ny, parts, scratch);
  else
    (sites ? k_plane_sums<float2, true> : k_plane_sums<float2, false>)<<<nz * parts, kThreads, 0, st>>>(
        (const float2*)psi_dev, nx, ny, parts, scratch);
  k_plane_total<<<1, kThreads, 0, st>>>(scratch, nz, parts, dx, dy, dz, norm_dev);
  return cudaGetLastError() == cudaSuccess ? GPE_OK : GPE_ERR_CUDA;
}
