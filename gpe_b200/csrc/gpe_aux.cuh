// Auxiliary kernels: layout conversion between the caller's contiguous
// interior array and the ghost-padded device fields, stand-alone norm,
// deterministic finalisation of block partials, and renormalisation.
#pragma once
#include "gpe_device.cuh"

namespace gpe {

// Launch shape of the row kernels below: a warp takes a row at a time, lanes
// along x.  Index arithmetic is per row, not a 64-bit division per site, and a
// lane has several independent loads in flight.
constexpr int ROW_THREADS = 256;
constexpr int ROW_GRID = 148 * 8;

// Rows shorter than a warp leave lanes idle: their sites go to threads one by
// one instead, at the price of two divisions a site (in 32 bits where the grid
// allows it).  set_state of 6 x 1000 x 1000 complex128 240 us by rows, 77 so;
// 24 x 600 x 600 114, 90.  A second pass over a row with few sites left costs
// k_pack more than its divisions do (33 x 450 x 450 complex64 74 us by rows, 67
// by sites; 40 x 500 x 500 91 either way); the other kernels with this rule are
// faster by rows there already.  Each has an instantiation for either (SITES):
// one with both loops holds fewer threads.
constexpr int SHORT_ROW = 32, SHORT_PACK = 40;
// is a row shorter than a warp, or a little longer (less than `most` sites)?
inline bool leaves_lanes(const Geom& g, int most) { return g.nx < most && g.nx != 32; }
inline bool short_rows(const Geom& g) { return g.nx < SHORT_ROW; }

// f(k, j, i, t): every interior site once, t its index in the contiguous array
template <class F>
__device__ __forceinline__ void for_each_site(const Geom& g, F f) {
  const long long n = (long long)g.nx * g.ny * g.nz;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const long long r = n <= 0x7fffffff ? (int)t / g.nx : t / g.nx;
    const int k = (int)(n <= 0x7fffffff ? (int)r / g.ny : r / g.ny);
    f(k, (int)(r - (long long)k * g.ny), (int)(t - r * g.nx), t);
  }
}

// f(k, j, lane, row): every interior row once, a warp each
template <class F>
__device__ __forceinline__ void for_each_row(const Geom& g, F f) {
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)g.ny * g.nz;
  const int tw = gridDim.x * (ROW_THREADS / 32);
  for (long long r = blockIdx.x * (ROW_THREADS / 32) + (threadIdx.x >> 5); r < rows; r += tw) {
    const int k = (int)(r / g.ny), j = (int)(r - (long long)k * g.ny);
    f(k, j, lane, r);
  }
}

// Store a site's value with its face ghosts.
template <class S>
__device__ __forceinline__ void put_site(S* __restrict__ f, const Geom& g, int R, int bcs, int zmask, int k, int j,
                                         int i, S v) {
  store_with_ghosts(f, g, (long long)(j + 2) * g.px + g.xoff + i, i, j, k, ghost_pos(i, g.nx, R, bcs),
                    ghost_pos(j, g.ny, R, bcs), zghost_pos(k, g.nz, R, bcs, zmask), v);
}

// Store a row's values (val(i) for lanes of x) with their face ghosts: whole
// images of the row in y and z, the first and last sites in x.
template <class S, class F>
__device__ __forceinline__ void put_row(S* __restrict__ f, const Geom& g, int R, int bcs, int zmask, int k, int j,
                                        int lane, F val) {
  S* row = f + (long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff;
  const int gy = ghost_pos(j, g.ny, R, bcs), gz = zghost_pos(k, g.nz, R, bcs, zmask);
  S* yrow = gy == NOGHOST ? nullptr : row + (long long)(gy - j) * g.px;
  S* zrow = gz == NOGHOST ? nullptr : row + (long long)(gz - k) * g.pz;
  for (int i0 = lane; i0 < g.nx; i0 += 4 * 32) {
    S s[4];  // the loads of four chunks before any store
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (i0 + 32 * c < g.nx) s[c] = val(i0 + 32 * c);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + 32 * c;
      if (i >= g.nx) break;
      row[i] = s[c];
      if (yrow) yrow[i] = s[c];
      if (zrow) zrow[i] = s[c];
      const int gx = ghost_pos(i, g.nx, R, bcs);
      if (gx != NOGHOST) row[gx] = s[c];
    }
  }
}

// contiguous interior (complex T2, [k][j][i]) -> ghost-padded field S with
// its face ghosts (the halo exchange of gpe.f90:173-176, done once).  256^3
// complex128: 124 us with an index division per site, 84 us so (82 at the copy
// rate).
template <bool SITES, class S, class T2>
__global__ void __launch_bounds__(ROW_THREADS) k_pack(const T2* __restrict__ src, S* __restrict__ dst, Geom g, int R,
                                                      int bcs, int zmask) {
  auto conv = [](T2 v) {
    S s;
    s.x = (typename Stor<S>::R)v.x;
    s.y = (typename Stor<S>::R)v.y;
    return s;
  };
  if constexpr (SITES)
    for_each_site(g, [&](int k, int j, int i, long long t) { put_site(dst, g, R, bcs, zmask, k, j, i, conv(src[t])); });
  else
    for_each_row(g, [&](int k, int j, int lane, long long r) {
      const T2* p = src + r * g.nx;
      put_row(dst, g, R, bcs, zmask, k, j, lane, [&](int i) { return conv(p[i]); });
    });
}

template <class S, class T2>
void pack(const T2* src, S* dst, const Geom& g, int R, int bcs, int zmask, cudaStream_t st) {
  if (leaves_lanes(g, SHORT_PACK)) k_pack<true><<<ROW_GRID, ROW_THREADS, 0, st>>>(src, dst, g, R, bcs, zmask);
  else k_pack<false><<<ROW_GRID, ROW_THREADS, 0, st>>>(src, dst, g, R, bcs, zmask);
}

// ghost-padded field -> contiguous interior, a warp per row
template <class S, class T2>
__global__ void __launch_bounds__(ROW_THREADS) k_unpack(const S* __restrict__ src, T2* __restrict__ dst, Geom g) {
  for_each_row(g, [&](int k, int j, int lane, long long r) {
    const S* row = src + (long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff;
    T2* p = dst + r * g.nx;
#pragma unroll 4
    for (int i = lane; i < g.nx; i += 32) {
      const S v = row[i];
      T2 o;
      o.x = v.x;
      o.y = v.y;
      p[i] = o;
    }
  });
}

// the same, a thread per site
template <class S, class T2>
__global__ void __launch_bounds__(ROW_THREADS) k_unpack_sites(const S* __restrict__ src, T2* __restrict__ dst, Geom g) {
  for_each_site(g, [&](int k, int j, int i, long long t) {
    const S v = src[(long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff + i];
    T2 o;
    o.x = v.x;
    o.y = v.y;
    dst[t] = o;
  });
}

// Rows that are short, or long but too few to give every second warp one, are
// unpacked site by site, six blocks on an SM (40 x 500 x 500 complex128: 79 us
// by rows, 80, 71, 76 by sites with 8, 6 and 5 blocks; 63 x 350 x 350 62 by
// rows, 66 by sites; 5000 x 6 x 300 75 by rows, 68 by sites).
constexpr int SHORT_UNPACK = 48, LONG_UNPACK = 512;
constexpr int UNPACK_SITES_GRID = 148 * 6;

template <class S, class T2>
void unpack(const S* src, T2* dst, const Geom& g, cudaStream_t st) {
  const bool few = g.nx >= LONG_UNPACK && (long long)g.ny * g.nz < ROW_GRID * (ROW_THREADS / 32) / 2;
  if (few || leaves_lanes(g, SHORT_UNPACK))
    k_unpack_sites<S, T2><<<UNPACK_SITES_GRID, ROW_THREADS, 0, st>>>(src, dst, g);
  else
    k_unpack<S, T2><<<ROW_GRID, ROW_THREADS, 0, st>>>(src, dst, g);
}

// get_norm partials (variables.f90:554-576): w_i w_j w_k |psi|^2 per block,
// same tiling as the stage kernel so the sum order is fixed.
template <class S>
__global__ void __launch_bounds__(256) k_norm(const S* __restrict__ f, Geom g, int zc, const double* __restrict__ wx,
                                               const double* __restrict__ wy, const double* __restrict__ wz,
                                               double* partials) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  const int kb = blockIdx.z * zc, ke = min(kb + zc, g.nz);
  double s = 0.0;
  if (i < g.nx && j < g.ny) {
    const double wxy = wx[i] * wy[j];
    const long long col = (long long)(j + 2) * g.px + g.xoff + i;
    for (int k = kb; k < ke; ++k) {
      const S v = __ldg(f + (long long)(k + 2) * g.pz + col);
      const double vr = (double)v.x, vi = (double)v.y;
      s += (wxy * wz[k]) * (vr * vr + vi * vi);
    }
  }
  block_reduce_store<256>(s, 0.0, 0.0, partials);
}

// get_norm of many solves in one launch: block b sums the planes k0 ..
// k0 + NORM_PLANES - 1 of solve items[b].solve, rows to warps in a fixed order.
// The partition depends on the solve's own grid only, so a solve's norm does
// not depend on what else is in the batch or on the stage launches' items.
struct NormSolve {
  Geom g;
  const double *wx, *wy, *wz;
  const void* psi;
};
struct NormItem {
  int solve, k0;
};
constexpr int NORM_PLANES = 1;  // (a warp's rows are a serial chain of loads)

template <class S>
__global__ void __launch_bounds__(ROW_THREADS) k_norm_batch(const NormSolve* __restrict__ sv,
                                                            const NormItem* __restrict__ items, double* partials) {
  const NormItem it = items[blockIdx.x];
  const NormSolve n = sv[it.solve];
  const Geom g = n.g;
  const int lane = threadIdx.x & 31;
  const int rows = min(NORM_PLANES, g.nz - it.k0) * g.ny;
  double s = 0.0;
  for (int r = threadIdx.x >> 5; r < rows; r += ROW_THREADS / 32) {
    const int dk = r / g.ny, j = r - dk * g.ny, k = it.k0 + dk;
    const S* row = (const S*)n.psi + (long long)(k + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff;
    double t = 0.0;
#pragma unroll 4
    for (int i = lane; i < g.nx; i += 32) {
      const S v = row[i];
      const double vr = (double)v.x, vi = (double)v.y;
      t += n.wx[i] * (vr * vr + vi * vi);
    }
    s += (n.wy[j] * n.wz[k]) * t;
  }
  block_reduce_store_at<ROW_THREADS>(s, 0.0, 0.0, partials, blockIdx.x);
}

// Sum (slots 0,1) and max (slot 2) of nb block partials in a fixed order;
// zeroes *top (the running maximum of the stage that made them) for its next
// launch.
static __global__ void __launch_bounds__(256) k_finalize(const double* __restrict__ partials, long long nb, double* out,
                                                         unsigned long long* top) {
  __shared__ double s0[256], s1[256], s2[256];
  const int t = threadIdx.x;
  double a = 0.0, b = 0.0, c = 0.0;
  for (long long q = t; q < nb; q += 256) {
    a += partials[q * RED_SLOTS + 0];
    b += partials[q * RED_SLOTS + 1];
    c = fmax(c, partials[q * RED_SLOTS + 2]);
  }
  s0[t] = a;
  s1[t] = b;
  s2[t] = c;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      s0[t] += s0[t + w];
      s1[t] += s1[t + w];
      s2[t] = fmax(s2[t], s2[t + w]);
    }
    __syncthreads();
  }
  if (t == 0) {
    out[0] = s0[0];
    out[1] = s1[0];
    out[2] = s2[0];
    *top = 0;
  }
}

// Per-solve sums of work-item partials: block s reduces items
// [first[s], first[s+1]) in a fixed order (thread-strided, then a tree), so a
// solve's result depends only on its own items.
static __global__ void __launch_bounds__(256) k_finalize_ranges(const double* __restrict__ partials,
                                                         const int* __restrict__ first, double* out) {
  __shared__ double s0[256], s1[256], s2[256];
  const int sv = blockIdx.x, t = threadIdx.x;
  double a = 0.0, b = 0.0, c = 0.0;
  for (int q = first[sv] + t; q < first[sv + 1]; q += 256) {
    a += partials[(long long)q * RED_SLOTS + 0];
    b += partials[(long long)q * RED_SLOTS + 1];
    c = fmax(c, partials[(long long)q * RED_SLOTS + 2]);
  }
  s0[t] = a;
  s1[t] = b;
  s2[t] = c;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      s0[t] += s0[t + w];
      s1[t] += s1[t + w];
      s2[t] = fmax(s2[t], s2[t + w]);
    }
    __syncthreads();
  }
  if (t == 0) {
    out[sv * RED_SLOTS + 0] = s0[0];
    out[sv * RED_SLOTS + 1] = s1[0];
    out[sv * RED_SLOTS + 2] = s2[0];
  }
}

// renormalise (variables.f90:715-726): var = sqrt(nn)*var/sqrt(norm), over
// the whole padded buffer (ghost copies scale identically)
template <class S>
__global__ void __launch_bounds__(ROW_THREADS) k_scale(S* f, long long n, double a, double b) {
  const long long step = (long long)gridDim.x * ROW_THREADS;
  for (long long t = blockIdx.x * (long long)ROW_THREADS + threadIdx.x; t < n; t += 4 * step) {
    S v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (t + c * step < n) v[c] = f[t + c * step];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (t + c * step < n) {
        v[c].x = (typename Stor<S>::R)(((double)v[c].x * a) / b);
        v[c].y = (typename Stor<S>::R)(((double)v[c].y * a) / b);
        f[t + c * step] = v[c];
      }
  }
}

}  // namespace gpe
