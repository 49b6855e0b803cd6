// FFT diagnostics (condensed_particles, spectrum, filtered_surface) on the
// device.  Every reduction is deterministic: static assignment of work to
// warps, per-warp shared-memory histograms, fixed-order sums over warps and
// blocks; no floating-point atomics.
#include <cufft.h>
#include <math.h>

#include "gpe_aux.cuh"
#include "gpe_fft.h"
#include "gpe_ic.h"

namespace gpe {

namespace {

constexpr int NS = GPE_SPECTRUM_SHELLS;
constexpr int FFT_BLOCKS = 148 * 2;  // of the spectral sums (two fit on an SM)
constexpr int ROW_BLOCKS = 148 * 8;  // of the row kernels
constexpr int FFT_THREADS = 256;
constexpr double PI_D = 3.1415926535897932384626433832795;

// partial layout per block: [H (nbins)] [eta (NS)] [nharm (NS)] [tot] [n0]
__host__ __device__ inline int part_width(int nbins) { return nbins + 2 * NS + 2; }

// squared index distance of spectral index i on an n-point axis
// (io.f90:547-565, 684-699): i^2 for i <= (n-1)/2 + 1, else (n-i)^2
__device__ __forceinline__ int k2_axis(int i, int n) {
  const int n1 = n - 1;
  return i <= n1 / 2 + 1 ? i * i : (n1 - i + 1) * (n1 - i + 1);
}

// The indices of an axis fold onto 0 .. fold_max(n): i and n - i have the same
// squared distance where n - i lies beyond it.
__host__ __device__ __forceinline__ int fold_max(int n) { return (n - 1) / 2 + 1; }
__device__ __forceinline__ bool has_twin(int i, int n) { return i > 0 && n - i > fold_max(n); }

// Deterministic sum over the block of one value per thread; valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += scratch[q];
  return s;
}

// The psi field as the contiguous complex128 array of the transform, and the
// sum of |psi|^2 (one partial per block).  A warp takes a row at a time: no
// index division per site, and one read of psi instead of the two of a
// separate conversion and mass kernel (256^3 complex128: 87 + 121 us for
// those, 83 for this; bound by HBM, 512 MiB).
template <class S, bool SITES>
__global__ void __launch_bounds__(FFT_THREADS) k_unpack_mass(const S* __restrict__ f, Geom g, double2* __restrict__ a,
                                                             double* part) {
  __shared__ double scratch[32];
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)g.ny * g.nz;
  const int tw = gridDim.x * (FFT_THREADS / 32);
  double acc = 0.0;
  if constexpr (SITES)
    for_each_site(g, [&](int k, int j, int i, long long t) {
      const S v = f[(long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff + i];
      const double x = (double)v.x, y = (double)v.y;
      a[t] = make_double2(x, y);
      acc += x * x + y * y;
    });
  for (long long r = blockIdx.x * (FFT_THREADS / 32) + (threadIdx.x >> 5); !SITES && r < rows; r += tw) {
    const int k = (int)(r / g.ny), j = (int)(r - (long long)k * g.ny);
    const S* src = f + (long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff;
    double2* dst = a + r * g.nx;
#pragma unroll 4
    for (int i = lane; i < g.nx; i += 32) {
      const S v = src[i];
      const double x = (double)v.x, y = (double)v.y;
      dst[i] = make_double2(x, y);
      acc += x * x + y * y;
    }
  }
  const double s = block_sum(acc, scratch);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// Squared distances at which a shell begins: shells m-1 <= |log2(sqrt(k2) /
// (2 pi))| < m, m = 1..7 (io.f90:706-713).  k2 >= up[s] is past shell s
// (0-based) above 2 pi, k2 <= down[s] past it below.
struct Shells {
  int up[NS], down[2];
};

Shells shells() {
  Shells t;
  double b = 4.0 * PI_D * PI_D;
  t.down[0] = (int)(b / 4.0);
  t.down[1] = (int)(b / 16.0);  // |log2| of the smallest k2, 1, is 2.65
  for (int q = 0; q < NS; ++q) {
    b *= 4.0;
    t.up[q] = (int)ceil(b);
  }
  return t;
}

// Spectral sums over a = raw / sqrt(N).  The spectra depend on the squared
// index distance alone, so a warp takes 32 folded x indices of a folded
// (j, k) row and adds the up to eight modes that share a distance before it
// bins them once.  Along the lanes the distance grows, so lanes of one bin are
// neighbours: a segmented scan sums them and the last lane of each segment
// adds to the warp's histogram.  Shell sums and counts stay in registers.
// tot uses the reference's real-space-indexed k grid (kq tables), one term
// per mode.  256^3: 1004 us with a 32-step lane loop per mode and bin, 112 us
// so (one read of 256 MiB takes 41; the FP64 divisions of tot bound it).
template <bool SITES>
__global__ void __launch_bounds__(FFT_THREADS) k_spectrum(const double2* __restrict__ raw, int nx, int ny, int nz,
                                                          const double* __restrict__ kq, int nbins,
                                                          int want_spectrum, Shells th, double* part) {
  extern __shared__ double sh[];
  __shared__ double scratch[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* wh = sh + (size_t)w * nbins;
  for (int b = lane; b < nbins; b += 32) wh[b] = 0.0;
  __syncwarp();

  const double n = (double)nx * (double)ny * (double)nz;
  const double n0 = (raw[0].x * raw[0].x + raw[0].y * raw[0].y) / n;
  const double rho0 = n0 / n;
  const double c12 = -(1.0 / 12.0);
  const double* kx = kq;
  const double* ky = kq + nx;
  const double* kz = kq + nx + ny;

  const int hx = fold_max(nx), hy = fold_max(ny), hz = fold_max(nz);
  const int nch = (hx + 32) / 32;  // 32-lane chunks of 0 .. hx
  const long long units = (long long)(hz + 1) * (hy + 1) * nch;
  const int tw = gridDim.x * nw;
  double tot = 0.0, es[NS];
  int cnt[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    es[q] = 0.0;
    cnt[q] = 0;
  }
  if constexpr (SITES) {  // tot mode by mode where folded rows would leave most lanes idle
    Geom g = {};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    for_each_site(g, [&](int k, int j, int i, long long) {
      const double q = c12 * ((kx[i] + ky[j]) + kz[k]);
      if (q != 0.0) tot += (q + rho0) / (q * q + 2.0 * rho0 * q);
    });
  }
  for (long long u = blockIdx.x * nw + w; (want_spectrum || !SITES) && u < units; u += tw) {
    const long long row = u / nch;
    const int i = (int)(u - row * nch) * 32 + lane;
    const int kk = (int)(row / (hy + 1)), jj = (int)(row - (long long)kk * (hy + 1));
    const bool in = i <= hx && i < nx, tx = in && has_twin(i, nx);
    const int nj = has_twin(jj, ny) ? 2 : 1, nk = has_twin(kk, nz) ? 2 : 1;
    double v = 0.0;
    // (a short axis folds onto indices past its end)
    if (jj < ny && kk < nz && in) {
      // all loads of the group first
      double2 m[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        m[c] = make_double2(0.0, 0.0);
        if (want_spectrum && (c & 1) < nj && ((c >> 1) & 1) < nk && (c < 4 || tx)) {
          const int j = (c & 1) ? ny - jj : jj, k = (c & 2) ? nz - kk : kk;
          m[c] = raw[((long long)k * ny + j) * nx + (c < 4 ? i : nx - i)];
        }
      }
      const double kx0 = kx[i], kx1 = tx ? kx[nx - i] : 0.0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (SITES || (c & 1) >= nj || (c >> 1) >= nk) continue;
        const int j = (c & 1) ? ny - jj : jj, k = (c >> 1) ? nz - kk : kk;
        // io.f90:343-360
        const double q0 = c12 * ((kx0 + ky[j]) + kz[k]);
        if (q0 != 0.0) tot += (q0 + rho0) / (q0 * q0 + 2.0 * rho0 * q0);
        if (tx) {
          const double q1 = c12 * ((kx1 + ky[j]) + kz[k]);
          if (q1 != 0.0) tot += (q1 + rho0) / (q1 * q1 + 2.0 * rho0 * q1);
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) v += m[c].x * m[c].x + m[c].y * m[c].y;
    }
    if (!want_spectrum) continue;
    v /= n;
    const int k2 = i * i + jj * jj + kk * kk;
    const bool mode = in && jj < ny && kk < nz && k2 != 0;
    // F(kk) collects sqrt(k2) <= kk (io.f90:701-705): bin ceil(sqrt(k2))
    int b = (int)sqrtf((float)k2);
    while (b * b < k2) ++b;
    while (b > 1 && (b - 1) * (b - 1) >= k2) --b;
    if (!mode || b >= nbins) b = in ? nbins : nbins + 1;
    if (mode) {
      int s = 0;
#pragma unroll
      for (int q = 0; q < NS; ++q) s += k2 >= th.up[q];
      s += (k2 <= th.down[0]) + (k2 <= th.down[1]);
      const int m = nj * nk * (tx ? 2 : 1);
#pragma unroll
      for (int q = 0; q < NS; ++q)
        if (s == q) {
          es[q] += v;
          cnt[q] += m;
        }
    }
    double run = mode ? v : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, run, o);
      const int ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o && ub == b) run += up;
    }
    const int nb = __shfl_down_sync(0xffffffffu, b, 1);
    if (b < nbins && (lane == 31 || nb != b)) wh[b] += run;
    __syncwarp();
  }

  double* out = part + (size_t)blockIdx.x * part_width(nbins);
  const double bt = block_sum(tot, scratch);  // (its barriers publish the histograms)
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    double acc = 0.0;
    for (int q = 0; q < nw; ++q) acc += sh[(size_t)q * nbins + b];
    out[b] = acc;
  }
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const double e = block_sum(es[q], scratch), c = block_sum((double)cnt[q], scratch);
    if (threadIdx.x == 0) {
      out[nbins + q] = e;
      out[nbins + NS + q] = c;
    }
  }
  if (threadIdx.x == 0) {
    out[nbins + 2 * NS] = bt;
    out[nbins + 2 * NS + 1] = n0;
  }
}

// Column c of the per-block partials summed in a fixed order (one block per
// column); the last column (n0) is the same in every row and is copied.  Block
// `width` sums the mass partials.
constexpr int COL_THREADS = 128;
__global__ void __launch_bounds__(COL_THREADS) k_sum_columns(const double* part, int nblocks, int width,
                                                             const double* mpart, int nmass, double* out) {
  __shared__ double scratch[32];
  const int c = blockIdx.x;
  double acc = 0.0;
  for (int b = threadIdx.x; b < (c == width ? nmass : nblocks); b += COL_THREADS)
    acc += c == width ? mpart[b] : part[(size_t)b * width + c];
  const double s = block_sum(acc, scratch);
  if (threadIdx.x == 0) out[c] = c == width - 1 ? part[c] : s;
}

// raw -> raw (filter max(1 - m k2 / kc^2, 0)) / N (io.f90:567): the factor
// 1/sqrt(N) of the forward transform and that of the inverse that follows
template <bool SITES>
__global__ void __launch_bounds__(FFT_THREADS) k_filter(double2* raw, int nx, int ny, int nz, double mscale, double kc2) {
  const double n = (double)nx * (double)ny * (double)nz;
  auto apply = [&](double2* a, int i, int kjk) {
    const double f = fmax(1.0 - (mscale * (double)(k2_axis(i, nx) + kjk)) / kc2, 0.0) / n;
    const double2 v = *a;
    *a = make_double2(v.x * f, v.y * f);
  };
  Geom g = {};
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  if constexpr (SITES)
    for_each_site(g, [&](int k, int j, int i, long long t) { apply(raw + t, i, k2_axis(j, ny) + k2_axis(k, nz)); });
  else
    for_each_row(g, [&](int k, int j, int lane, long long r) {
      const int kjk = k2_axis(j, ny) + k2_axis(k, nz);
#pragma unroll 4
      for (int i = lane; i < nx; i += 32) apply(raw + r * nx + i, i, kjk);
    });
}

cudaError_t to_contiguous(const Geom& g, int esz, const void* psi_field, double2* buf, double* mpart,
                          cudaStream_t st) {
  const bool sites = short_rows(g);
  if (esz == 16)
    (sites ? k_unpack_mass<double2, true> : k_unpack_mass<double2, false>)<<<ROW_BLOCKS, FFT_THREADS, 0, st>>>(
        (const double2*)psi_field, g, buf, mpart);
  else
    (sites ? k_unpack_mass<float2, true> : k_unpack_mass<float2, false>)<<<ROW_BLOCKS, FFT_THREADS, 0, st>>>(
        (const float2*)psi_field, g, buf, mpart);
  return cudaGetLastError();
}

size_t round256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

size_t fft_work_bytes(const gpe_params& p) {
  const size_t n = (size_t)p.nx * p.ny * p.nz;
  const int nbins = p.nx / 2 + 1;
  return round256(n * sizeof(double2)) +
         round256(((size_t)(FFT_BLOCKS + 1) * part_width(nbins) + 1) * sizeof(double)) +
         round256((size_t)ROW_BLOCKS * sizeof(double)) + 256;
}

void fft_kq_axis(int n, int nx, double d, double* out) {
  // kc = pi, dk = 2 kc / (nx - 1) on every axis (io.f90:323-324, 345-351)
  const double kc = PI_D;
  const double dk = 2.0 * kc / (double)(nx - 1);
  const double d2 = d * d;
  for (int i = 0; i < n; ++i) {
    const double k = -kc + (double)i * dk;
    out[i] = ((-2.0 * cos(2.0 * k * d) + 32.0 * cos(k * d)) - 30.0) / d2;
  }
}

cudaError_t fft_condensed(const gpe_params& p, const Geom& g, int esz, const void* psi_field, const double* kq,
                          bool want_spectrum, void* work, size_t work_bytes, cudaStream_t st, FftDiag& out) {
  if (!work || work_bytes < fft_work_bytes(p)) return cudaErrorInvalidValue;
  const size_t n = (size_t)p.nx * p.ny * p.nz;
  const int nbins = p.nx / 2 + 1;
  const int width = part_width(nbins);
  double2* buf = (double2*)work;
  double* part = (double*)((char*)work + round256(n * sizeof(double2)));
  double* sums = part + (size_t)FFT_BLOCKS * width;  // width column sums, then the mass
  double* mpart = (double*)((char*)part + round256(((size_t)(FFT_BLOCKS + 1) * width + 1) * sizeof(double)));

  cudaError_t e = to_contiguous(g, esz, psi_field, buf, mpart, st);
  if (e != cudaSuccess) return e;
  cufftHandle plan;
  if (!plan_for(p.nx, p.ny, p.nz, &plan)) return cudaErrorUnknown;
  if (cufftSetStream(plan, st) != CUFFT_SUCCESS) return cudaErrorUnknown;
  if (cufftExecZ2Z(plan, (cufftDoubleComplex*)buf, (cufftDoubleComplex*)buf, CUFFT_FORWARD) != CUFFT_SUCCESS)
    return cudaErrorUnknown;
  // (folded, a row of 16 still keeps the other lanes' cost below an extra pass:
  // 26 x 37 x 85 with spectra 117 us folded, 125 with the pass; without spectra
  // 6 x 1000 x 1000 465 folded, 303 by sites, 16 x 700 x 700 519 folded)
  const auto spectrum = g.nx < 16 ? k_spectrum<true> : k_spectrum<false>;
  const size_t shm = (size_t)(FFT_THREADS / 32) * nbins * sizeof(double);
  if (shm > 48 * 1024) {
    e = cudaFuncSetAttribute(spectrum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
    if (e != cudaSuccess) return e;
  }
  spectrum<<<FFT_BLOCKS, FFT_THREADS, shm, st>>>(buf, p.nx, p.ny, p.nz, kq, nbins, want_spectrum ? 1 : 0, shells(), part);
  k_sum_columns<<<width + 1, COL_THREADS, 0, st>>>(part, FFT_BLOCKS, width, mpart, ROW_BLOCKS, sums);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;

  std::vector<double> hs(width + 1);
  e = cudaMemcpyAsync(hs.data(), sums, hs.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  out.mass_sum = hs[width];
  out.H.assign(hs.begin(), hs.begin() + nbins);
  for (int q = 0; q < NS; ++q) {
    out.eta[q] = hs[nbins + q];
    out.nharm[q] = hs[nbins + NS + q];
  }
  out.tot = hs[width - 2];
  out.n0 = hs[width - 1];
  return cudaSuccess;
}

cudaError_t fft_filtered(const gpe_params& p, const Geom& g, int esz, const void* psi_field, double mscale,
                         double filter_kc, void* work, size_t work_bytes, cudaStream_t st) {
  if (!work || work_bytes < fft_work_bytes(p)) return cudaErrorInvalidValue;
  double2* buf = (double2*)work;
  // (the mass is a by-product nobody asked for here)
  double* mpart = (double*)((char*)work + round256((size_t)p.nx * p.ny * p.nz * sizeof(double2)));
  cudaError_t e = to_contiguous(g, esz, psi_field, buf, mpart, st);
  if (e != cudaSuccess) return e;
  cufftHandle plan;
  if (!plan_for(p.nx, p.ny, p.nz, &plan)) return cudaErrorUnknown;
  if (cufftSetStream(plan, st) != CUFFT_SUCCESS) return cudaErrorUnknown;
  if (cufftExecZ2Z(plan, (cufftDoubleComplex*)buf, (cufftDoubleComplex*)buf, CUFFT_FORWARD) != CUFFT_SUCCESS)
    return cudaErrorUnknown;
  (short_rows(g) ? k_filter<true> : k_filter<false>)<<<ROW_BLOCKS, FFT_THREADS, 0, st>>>(buf, p.nx, p.ny, p.nz, mscale,
                                                                                         filter_kc * filter_kc);
  if (cufftExecZ2Z(plan, (cufftDoubleComplex*)buf, (cufftDoubleComplex*)buf, CUFFT_INVERSE) != CUFFT_SUCCESS)
    return cudaErrorUnknown;
  return cudaGetLastError();
}

}  // namespace gpe
