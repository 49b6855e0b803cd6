// Initial conditions generated on the device (gpe_set_ic,
// gpe_pool_submit_ic).  Each site evaluates the reference's closed-form
// initial states (src/ic.f90) in FP64 and the product is written straight
// into the solve's ghost-padded psi field, ghosts included.  The seeded
// random-phase state is a spectrum built in place, one inverse cuFFT and a
// rescale to mean density 1.
#include <cuda_runtime.h>
#include <cufft.h>

#include <map>
#include <mutex>
#include <tuple>

#include "gpe_aux.cuh"
#include "gpe_common.h"
#include "gpe_ic.h"

namespace gpe {

namespace {

constexpr double kPi = 3.1415926535897932384626433832795;

struct IcGrid {
  int nx, ny, nz;
  double xl, yl, zl, dx, dy, dz;
  double mu, g, omx, omy, omz, scal;
};

__device__ __forceinline__ double coord(double lo, double d, int q) { return lo + (double)q * d; }

// get_rr (src/ic.f90:893-906)
__device__ __forceinline__ double rr_of(double r) {
  const double r2 = r * r, r4 = r2 * r2;
  return sqrt((0.3437 + 0.0286 * r2) / ((1.0 + 0.3333 * r2) + 0.0286 * r4));
}

// get_r / get_theta (src/ic.f90:735-889) for a line along dir: the scaled
// distance r from the line and e^{i theta}, theta = sgn atan2(sc b, sc a).  An
// unperturbed line evaluates no sine of its displacement.
__device__ __forceinline__ void line_geom(const gpe_line& vl, double sc, double x, double y, double z, double* r,
                                          double* cth, double* sth) {
  const double eps = 2.220446049250313e-16;
  double s1 = 0.0, s2 = 0.0;
  if (fabs(vl.ll) < eps) {
    s1 = 1.0;
    s2 = 1.0;
  }
  double a, b, along;
  if (vl.dir == 'x') { a = y - vl.y0; b = z - vl.z0; along = x - vl.x0; }
  else if (vl.dir == 'y') { a = z - vl.z0; b = x - vl.x0; along = y - vl.y0; }
  else { a = x - vl.x0; b = y - vl.y0; along = z - vl.z0; }
  if (vl.amp1 != 0.0) a -= vl.amp1 * sin(2.0 * kPi * along / (vl.ll + s1));
  if (vl.amp2 != 0.0) b -= vl.amp2 * cos(2.0 * kPi * along / (vl.ll + s2));
  *r = sqrt(sc * (a * a) + sc * (b * b));
  sincos(vl.sgn * atan2(sc * b, sc * a), sth, cth);
}

// vortex_ring (src/ic.f90:357-514)
__device__ __forceinline__ void ring_val(const gpe_ring& vr, double sc, double x, double y, double z, double* re,
                                         double* im) {
  double u, v, w, u0, v0, w0;
  if (vr.plane[0] == 'x' && vr.plane[1] == 'y') { u = x; v = y; w = z; u0 = vr.x0; v0 = vr.y0; w0 = vr.z0; }
  else if (vr.plane[0] == 'x' && vr.plane[1] == 'z') { u = x; v = z; w = y; u0 = vr.x0; v0 = vr.z0; w0 = vr.y0; }
  else { u = y; v = z; w = x; u0 = vr.y0; v0 = vr.z0; w0 = vr.x0; }
  double s = sqrt((u - u0) * (u - u0) + (v - v0) * (v - v0)), dist = 0.0, pp = w;
  if (vr.r1 != 0.0 || vr.amp != 0.0) {  // a perturbed ring: the angle enters
    const double theta = atan2(v - v0, u - u0);
    s -= vr.r1 * sin((double)vr.kk * theta);
    dist = vr.amp * cos((double)vr.mm * theta);
    pp -= vr.r1 * cos((double)vr.kk * theta);
  }
  const double A = sc * (pp - w0), Bp = sc * ((s + vr.r0) - dist), Bm = sc * ((s - vr.r0) - dist);
  const double q1 = rr_of(sqrt(A * A + Bp * Bp)), q2 = rr_of(sqrt(A * A + Bm * Bm));
  const double z1r = A + vr.dir * 0.0 * Bp, z1i = vr.dir * Bp;
  const double z2r = A - vr.dir * 0.0 * Bm, z2i = -(vr.dir * Bm);
  const double tr = (q1 * z1r) * q2, ti = (q1 * z1i) * q2;
  *re = tr * z2r - ti * z2i;
  *im = tr * z2i + ti * z2r;
}

// pade_pulse_ring (src/ic.f90:518-587): the Pade approximations of the
// rarefaction pulse (pulse = true) and of the axisymmetric vortex ring that
// move along x (N. G. Berloff, J. Phys. A 37, 1617 (2004)), centred at x0
// with the axis through (y0, z0) and radius r0.  a(1..9), U and m are the
// published coefficients the reference's get_consts lists for the two cases
// (src/ic.f90:572-581); the same numbers give the same state.
__device__ __forceinline__ void pade_val(bool pulse, const gpe_pulse& pp, double x, double y, double z, double* re,
                                         double* im) {
  const double a1 = pulse ? -0.79792 : -1.1, a2 = pulse ? 0.00388059 : 0.0170524;
  const double a3 = pulse ? 0.00882276 : 0.0289452, a4 = pulse ? -0.7981 : -0.953;
  const double a5 = pulse ? -0.012783 : -0.0049767, a6 = pulse ? -0.0574092 : -0.0594346;
  const double a7 = pulse ? 0.0399 : 0.04, a8 = pulse ? 0.199 : 0.21, a9 = pulse ? 0.0058 : 0.00612;
  const double U = pulse ? 0.63 : 0.6, m = pulse ? 8.37 : 8.97;
  const double p74 = 7.0 / 4.0;
  const double one_2u = 1.0 - 2.0 * (U * U);
  const double ma9 = m * pow(a9, p74);
  const double s = sqrt((y - pp.y0) * (y - pp.y0) + (z - pp.z0) * (z - pp.z0));  // get_s, ic.f90:804-820
  const double xs = x - pp.x0;
  const double x2 = xs * xs, s2 = (s - pp.r0) * (s - pp.r0);
  const double t = x2 + one_2u * s2;
  const double denom = pow(((1.0 + a8 * x2) + a7 * s2) + a9 * (t * t), p74);
  *re = 1.0 + ((((a1 + a3 * x2) + a2 * s2) + (ma9 * U) * (2.0 * x2 - one_2u * s2)) * t) / denom;
  *im = (xs * (((a4 + a6 * x2) + a5 * s2) - ma9 * (t * t))) / denom;
}

// vortex_pair (src/ic.f90:591-636): the Pade approximation of a vortex pair
// in the x-y plane, the same in every z plane; coefficients as listed there.
__device__ __forceinline__ void pair_val(double x, double y, double* re, double* im) {
  const double a0 = -1.14026, a1 = -0.150112, a2 = -0.0294564;
  const double b0 = -0.830953, b1 = -0.108296, b2 = -0.073641;
  const double c0 = 0.35022, c1 = 0.03032, c2 = 0.15905, c3 = 0.04123, c4 = 0.01402;
  const double x2 = x * x, y2 = y * y, x4 = x2 * x2, y4 = y2 * y2;
  const double denom = ((((1.0 + c0 * x2) + c1 * x4) + c2 * y2) + (c3 * x2) * y2) + c4 * y4;
  *re = 1.0 + ((a0 + a1 * x2) + a2 * y2) / denom;
  *im = (x * ((b0 + b1 * x2) + b2 * y2)) / denom;
}

// fermi (src/ic.f90:278): sqrt(max(mu - V, 0)/g) with vxy = omx^2 x^2 + omy^2 y^2
__device__ __forceinline__ double fermi_val(const IcGrid& G, double vxy, double z) {
  const double v = 0.5 * (vxy + (G.omz * G.omz) * (z * z));
  const double a = (G.mu - v) / G.g;
  return a >= 0.0 ? sqrt(a) : 0.0;
}

// Closed-form factor q of ic at (x, y, z).
__device__ __forceinline__ void ic_factor(const gpe_ic& ic, int q, const IcGrid& G, double x, double y, double z,
                                          double* out_r, double* out_i) {
  double fr = 1.0, fi = 0.0;
  switch (ic.factor[q]) {
    case GPE_IC_FERMI:
      fr = fermi_val(G, (G.omx * G.omx) * (x * x) + (G.omy * G.omy) * (y * y), z);
      break;
    case GPE_IC_LINE: {
      double r, c, s;
      line_geom(ic.line, G.scal, x, y, z, &r, &c, &s);
      const double a = ic.line.imprint_phase ? 1.0 : 1.0 - exp(-0.7 * pow(r, 1.15));
      fr = a * c;
      fi = a * s;
      break;
    }
    case GPE_IC_LINE_PADE: {
      double r, c, s;
      line_geom(ic.line, G.scal, x, y, z, &r, &c, &s);
      const double a = r * rr_of(r);
      fr = a * c;
      fi = a * s;
      break;
    }
    case GPE_IC_RING:
      ring_val(ic.ring, G.scal, x, y, z, &fr, &fi);
      break;
    case GPE_IC_PADE_PULSE:
    case GPE_IC_PADE_RING:
      pade_val(ic.factor[q] == GPE_IC_PADE_PULSE, ic.pulse, x, y, z, &fr, &fi);
      break;
    case GPE_IC_VORTEX_PAIR:
      pair_val(x, y, &fr, &fi);
      break;
    case GPE_IC_SPHERE:  // ic.f90:640-662 (rad = 10, eps1 = 2)
      fr = 0.5 * (1.0 + tanh((sqrt((x * x + y * y) + z * z) - 10.0) - 2.0));
      break;
    case GPE_IC_SPHERE2:  // ic.f90:666-684 (amp = 100, width = 10)
      fr = 100.0 * exp(-((x * x + y * y) + z * z) / 10.0);
      break;
    case GPE_IC_WALL:  // ic.f90:688-709 (pos = -30)
      fr = z <= -30.0 ? 0.0 : 1.0;
      break;
    default:
      break;
  }
  *out_r = fr;
  *out_i = fi;
}

// Is factor q the same on every plane of a column?
__device__ __forceinline__ bool ic_columnar(const gpe_ic& ic, int q) {
  const int f = ic.factor[q];
  if (f == GPE_IC_UNIFORM || f == GPE_IC_VORTEX_PAIR) return true;
  return (f == GPE_IC_LINE || f == GPE_IC_LINE_PADE) && ic.line.dir == 'z' && ic.line.amp1 == 0.0 && ic.line.amp2 == 0.0;
}

constexpr int IC_THREADS = 256;  // columns of a block
constexpr int IC_CTAS = 3;     // blocks per SM the registers are fitted to
constexpr int IC_PLANES = 16;  // most planes a thread takes of its column
constexpr int IC_MAX = 4;      // factors of a product

// A block is 32 columns along x, or 16 or 8 where x is no longer than that, as
// many rows of them as it has threads for, or as few as y has, and the rest of
// its threads are further chunks of planes.  (A y too long for a launch's blocks
// of few rows gets blocks of many.)
dim3 ic_block(const Geom& g) {
  auto fit = [](int n, int most) { return n <= 8 ? 8 : (n <= 16 && most > 16 ? 16 : most); };
  const bool long_y = g.ny > GRID_YZ_MAX * (IC_THREADS / 32);
  const int w = long_y ? 8 : fit(g.nx, 32), h = fit(g.ny, IC_THREADS / w < 32 ? IC_THREADS / w : 32);
  return dim3(w, h, IC_THREADS / (w * h));
}

// the shape of all but the narrow grids
bool ic_full(const dim3& b) { return b.x == 32 && b.z == 1; }

// Planes per thread: as many as leave the device IC_CTAS blocks per SM, at
// most IC_PLANES (beyond that the column's factors cost little anyway) or what
// one launch needs to reach the end of z.
int ic_planes(const Geom& g) {
  const dim3 b = ic_block(g);
  const long long tiles = (long long)((g.nx + b.x - 1) / b.x) * ((g.ny + b.y - 1) / b.y);
  const long long chunks = (148LL * IC_CTAS + tiles - 1) / tiles * b.z;
  const int z = (int)(g.nz / chunks), least = (int)((g.nz - 1) / (GRID_YZ_MAX * (long long)b.z)) + 1;
  return z > IC_PLANES ? (least > IC_PLANES ? least : IC_PLANES) : (z < least ? least : z);
}

dim3 ic_blocks(const Geom& g) {
  const dim3 b = ic_block(g);
  const int z = ic_planes(g) * b.z;
  return dim3((g.nx + b.x - 1) / b.x, (g.ny + b.y - 1) / b.y, (g.nz + z - 1) / z);
}

// The product of the closed-form factors, taken left to right as the
// reference's init_cond expression multiplies them, over `planes` planes of
// one column (MULT: times the state there, or its modulus).  A thread keeps
// the factors that do not depend on z, so a vortex line along z costs its core
// and phase once per column; products of those and fermi run in a loop of
// their own without the other factors' code, and there is no index division.
// Instruction issue bounds it.  set_ic on 192 x 192 x 384 complex128, us, with
// every factor (and an arc tangent, a sine and a cosine) per site / so:
// fermi x line_pade 958 / 72, fermi x line 1104 / 79, ring 1027 / 298.
// FULL: blocks of the shape ordinary grids have.
template <class S, bool MULT, bool FULL>
__device__ __forceinline__ void ic_column(S* f, const Geom& g, int R, int bcs, const IcGrid& G, const gpe_ic& ic,
                                          int planes, int modulus) {
  const int i = blockIdx.x * (FULL ? 32 : blockDim.x) + threadIdx.x;
  const int j = blockIdx.y * (FULL ? IC_THREADS / 32 : blockDim.y) + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const int k0 = (FULL ? blockIdx.z : blockIdx.z * blockDim.z + threadIdx.z) * planes, k1 = min(k0 + planes, g.nz);
  const double x = coord(G.xl, G.dx, i), y = coord(G.yl, G.dy, j);
  const double vxy = (G.omx * G.omx) * (x * x) + (G.omy * G.omy) * (y * y);
  double fr[IC_MAX], fi[IC_MAX];
  bool other = false;  // a factor that changes along the column and is not fermi
#pragma unroll
  for (int q = 0; q < IC_MAX; ++q) {
    fr[q] = 1.0;
    fi[q] = 0.0;
    if (q >= ic.nfactors) continue;
    if (ic_columnar(ic, q)) ic_factor(ic, q, G, x, y, 0.0, &fr[q], &fi[q]);
    else other |= ic.factor[q] != GPE_IC_FERMI;
  }

  const int gx = ghost_pos(i, g.nx, R, bcs), gy = ghost_pos(j, g.ny, R, bcs);
  S* p = f + (long long)(k0 + 2) * g.pz + (long long)(j + 2) * g.px + g.xoff + i;
  const long long ox = gx - i, oy = (long long)(gy - j) * g.px;
  auto put = [&](int k, double pr, double pi) {
    if constexpr (MULT) {
      double ar = (double)p->x, ai = (double)p->y;
      if (modulus) {
        ar = hypot(ar, ai);
        ai = 0.0;
      }
      const double nr = ar * pr - ai * pi, ni = ar * pi + ai * pr;
      pr = nr;
      pi = ni;
    }
    S s;
    s.x = (typename Stor<S>::R)pr;
    s.y = (typename Stor<S>::R)pi;
    *p = s;
    if (gx != NOGHOST) p[ox] = s;
    if (gy != NOGHOST) p[oy] = s;
    if (k <= R || k >= g.nz - 1 - R) {
      const int gz = ghost_pos(k, g.nz, R, bcs);
      if (gz != NOGHOST) p[(long long)(gz - k) * g.pz] = s;
    }
    p += g.pz;
  };
  if (!other) {
#pragma unroll 2
    for (int k = k0; k < k1; ++k) {
      const double fv = fermi_val(G, vxy, coord(G.zl, G.dz, k));
      double pr = 1.0, pi = 0.0;
#pragma unroll
      for (int q = 0; q < IC_MAX; ++q) {
        if (q >= ic.nfactors) break;
        const double ar = ic.factor[q] == GPE_IC_FERMI ? fv : fr[q], ai = fi[q];
        const double nr = pr * ar - pi * ai, ni = pr * ai + pi * ar;
        pr = nr;
        pi = ni;
      }
      put(k, pr, pi);
    }
  } else {
    for (int k = k0; k < k1; ++k) {
      const double z = coord(G.zl, G.dz, k);
      double pr = 1.0, pi = 0.0;
#pragma unroll
      for (int q = 0; q < IC_MAX; ++q) {
        if (q >= ic.nfactors) break;
        double ar = fr[q], ai = fi[q];
        if (!ic_columnar(ic, q)) ic_factor(ic, q, G, x, y, z, &ar, &ai);
        const double nr = pr * ar - pi * ai, ni = pr * ai + pi * ar;
        pr = nr;
        pi = ni;
      }
      put(k, pr, pi);
    }
  }
}

template <class S, bool FULL>
__global__ void __launch_bounds__(IC_THREADS, IC_CTAS) k_ic_closed_form(S* f, Geom g, int R, int bcs, IcGrid G,
                                                                        const __grid_constant__ gpe_ic ic,
                                                                        int planes) {
  ic_column<S, false, FULL>(f, g, R, bcs, G, ic, planes, 0);
}

// psi <- psi * IC (modulus = 0: the state_restart product with init_cond,
// src/ic.f90:160-162) or psi <- |psi| * IC (modulus = 1:
// imprint_vortex_line, src/variables.f90:1166-1180), in FP64 per site, the
// new value stored with its ghosts.
template <class S, bool FULL>
__global__ void __launch_bounds__(IC_THREADS, IC_CTAS) k_ic_multiply(S* f, Geom g, int R, int bcs, IcGrid G,
                                                                     const __grid_constant__ gpe_ic ic, int planes,
                                                                     int modulus) {
  ic_column<S, true, FULL>(f, g, R, bcs, G, ic, planes, modulus);
}

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long seed, unsigned long long idx) {
  unsigned long long z = seed + (idx + 1ULL) * 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

// psi_hat(m) = exp(i 2 pi u_m) for |k_m| < kc, else 0; modes in numpy's
// fftfreq order, u_m from SplitMix64 over the linear mode index
template <bool SITES>
__global__ void __launch_bounds__(ROW_THREADS) k_random_spectrum(double2* buf, Geom g, double dx, double dy, double dz,
                                                                 unsigned long long seed, double kc) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  auto row2 = [&](int k, int j) {  // ky^2 + kz^2
    const int mj = j < (ny + 1) / 2 ? j : j - ny, mk = k < (nz + 1) / 2 ? k : k - nz;
    const double ky = 2.0 * kPi * mj / (ny * dy), kz = 2.0 * kPi * mk / (nz * dz);
    return kz * kz + ky * ky;
  };
  auto mode = [&](double kyz, int i, long long t) {
    const int mi = i < (nx + 1) / 2 ? i : i - nx;
    const double kx = 2.0 * kPi * mi / (nx * dx);
    double2 v = make_double2(0.0, 0.0);
    if (kyz + kx * kx < kc * kc) {
      const double u = (double)(splitmix64(seed, (unsigned long long)t) >> 11) * (1.0 / 9007199254740992.0);
      const double th = 2.0 * kPi * u;
      v = make_double2(cos(th), sin(th));
    }
    buf[t] = v;
  };
  if constexpr (SITES)
    for_each_site(g, [&](int k, int j, int i, long long t) { mode(row2(k, j), i, t); });
  else
    for_each_row(g, [&](int k, int j, int lane, long long r) {
      const double kyz = row2(k, j);
      for (int i = lane; i < nx; i += 32) mode(kyz, i, r * nx + i);
    });
}

// sum |psi|^2 over the buffer (fixed-order block partials, then one block)
__global__ void __launch_bounds__(256) k_sumsq(const double2* __restrict__ buf, long long n, double* part) {
  __shared__ double red[256];
  double s = 0.0;
  for (long long t = blockIdx.x * 256LL + threadIdx.x; t < n; t += 256LL * gridDim.x)
    s += buf[t].x * buf[t].x + buf[t].y * buf[t].y;
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(256) k_sum_parts(double* part, int nb) {
  __shared__ double red[256];
  double s = 0.0;
  for (int q = threadIdx.x; q < nb; q += 256) s += part[q];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[nb] = red[0];
}

// psi = buf * sqrt(n / sum|buf|^2) into the padded field with ghosts
template <bool SITES, class S>
__global__ void __launch_bounds__(ROW_THREADS) k_pack_scaled(const double2* __restrict__ buf,
                                                             const double* __restrict__ total, S* f, Geom g, int R,
                                                             int bcs) {
  const double n = (double)g.nx * (double)g.ny * (double)g.nz;
  const double sc = 1.0 / sqrt(*total / n);
  auto scaled = [&](double2 v) {
    S s;
    s.x = (typename Stor<S>::R)(v.x * sc);
    s.y = (typename Stor<S>::R)(v.y * sc);
    return s;
  };
  if constexpr (SITES)
    for_each_site(g, [&](int k, int j, int i, long long t) { put_site(f, g, R, bcs, 3, k, j, i, scaled(buf[t])); });
  else
    for_each_row(g, [&](int k, int j, int lane, long long r) {
      const double2* p = buf + r * g.nx;
      put_row(f, g, R, bcs, 3, k, j, lane, [&](int i) { return scaled(p[i]); });
    });
}

template <class S>
void pack_scaled(const double2* buf, const double* total, S* f, const Geom& g, int R, int bcs, cudaStream_t st) {
  if (short_rows(g)) k_pack_scaled<true><<<ROW_GRID, ROW_THREADS, 0, st>>>(buf, total, f, g, R, bcs);
  else k_pack_scaled<false><<<ROW_GRID, ROW_THREADS, 0, st>>>(buf, total, f, g, R, bcs);
}

// 3-D Z2Z plans, one per (device, grid), created on first use
std::mutex g_plan_mu;
std::map<std::tuple<int, int, int, int>, cufftHandle> g_plans;

}  // namespace

bool plan_for(int nx, int ny, int nz, cufftHandle* out) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_plan_mu);
  auto key = std::make_tuple(dev, nx, ny, nz);
  auto it = g_plans.find(key);
  if (it != g_plans.end()) {
    *out = it->second;
    return true;
  }
  cufftHandle p;
  if (cufftPlan3d(&p, nz, ny, nx, CUFFT_Z2Z) != CUFFT_SUCCESS) return false;
  g_plans[key] = p;
  *out = p;
  return true;
}

int ic_validate(const gpe_ic* ic, std::string& why) {
  if (!ic || ic->nfactors < 1 || ic->nfactors > 4) {
    why = "gpe_ic: nfactors must be 1..4";
    return GPE_ERR_BADARG;
  }
  for (int q = 0; q < ic->nfactors; ++q) {
    const int f = ic->factor[q];
    if (f < GPE_IC_UNIFORM || f > GPE_IC_WALL) {
      why = "gpe_ic: unknown factor";
      return GPE_ERR_BADARG;
    }
    if (f == GPE_IC_RANDOM_PHASE && ic->nfactors != 1) {
      why = "gpe_ic: the random-phase state must be the only factor";
      return GPE_ERR_BADARG;
    }
    if (f == GPE_IC_RING) {
      const char* p = ic->ring.plane;
      const bool ok = (p[0] == 'x' && p[1] == 'y') || (p[0] == 'x' && p[1] == 'z') || (p[0] == 'y' && p[1] == 'z');
      if (!ok) {
        why = "ERROR: Unrecognised vortex ring plane.";  // src/ic.f90:510
        return GPE_ERR_BADARG;
      }
    }
    if (f == GPE_IC_LINE || f == GPE_IC_LINE_PADE) {
      const double eps = 2.220446049250313e-16;
      if (fabs(ic->line.ll) < eps && (fabs(ic->line.amp1) >= eps || fabs(ic->line.amp2) >= eps)) {
        why = "ERROR: vortex line disturbance wavelength is zero, but amplitude is non-zero.";  // ic.f90:755
        return GPE_ERR_BADARG;
      }
      if (ic->line.dir != 'x' && ic->line.dir != 'y' && ic->line.dir != 'z') {
        why = "gpe_ic: line direction must be x, y or z";
        return GPE_ERR_BADARG;
      }
    }
  }
  return GPE_OK;
}

bool ic_needs_fft(const gpe_ic* ic) { return ic->nfactors == 1 && ic->factor[0] == GPE_IC_RANDOM_PHASE; }

IcGrid ic_grid(const gpe_params& p) {
  IcGrid G;
  G.nx = p.nx;
  G.ny = p.ny;
  G.nz = p.nz;
  G.xl = -p.xr;
  G.yl = -p.yr;
  G.zl = -p.zr;
  G.dx = (p.xr - G.xl) / (p.nx - 1);
  G.dy = (p.yr - G.yl) / (p.ny - 1);
  G.dz = (p.zr - G.zl) / (p.nz - 1);
  G.mu = p.mu;
  G.g = p.g;
  G.omx = p.omx;
  G.omy = p.omy;
  G.omz = p.omz;
  G.scal = p.scal;
  return G;
}

cudaError_t ic_multiply(const gpe_params& p, const Geom& g, int esz, int R, const gpe_ic& ic, void* psi_field,
                        int modulus, cudaStream_t st) {
  if (ic_needs_fft(&ic)) return cudaErrorInvalidValue;
  const IcGrid G = ic_grid(p);
  const dim3 nb = ic_blocks(g), nt = ic_block(g);
  const bool full = ic_full(nt);
  if (esz == 16)
    (full ? k_ic_multiply<double2, true> : k_ic_multiply<double2, false>)<<<nb, nt, 0, st>>>(
        (double2*)psi_field, g, R, p.bcs, G, ic, ic_planes(g), modulus);
  else
    (full ? k_ic_multiply<float2, true> : k_ic_multiply<float2, false>)<<<nb, nt, 0, st>>>(
        (float2*)psi_field, g, R, p.bcs, G, ic, ic_planes(g), modulus);
  return cudaGetLastError();
}

cudaError_t ic_generate(const gpe_params& p, const Geom& g, int esz, int R, const gpe_ic& ic, void* psi_field,
                        void* work, size_t work_bytes, cudaStream_t st) {
  const IcGrid G = ic_grid(p);
  if (!ic_needs_fft(&ic)) {
    const dim3 nb = ic_blocks(g), nt = ic_block(g);
    const bool full = ic_full(nt);
    if (esz == 16)
      (full ? k_ic_closed_form<double2, true> : k_ic_closed_form<double2, false>)<<<nb, nt, 0, st>>>(
          (double2*)psi_field, g, R, p.bcs, G, ic, ic_planes(g));
    else
      (full ? k_ic_closed_form<float2, true> : k_ic_closed_form<float2, false>)<<<nb, nt, 0, st>>>(
          (float2*)psi_field, g, R, p.bcs, G, ic, ic_planes(g));
    return cudaGetLastError();
  }
  const long long n = (long long)p.nx * p.ny * p.nz;
  const size_t need = (size_t)n * sizeof(double2) + 1024 * sizeof(double) + 256;
  if (!work || work_bytes < need) return cudaErrorInvalidValue;
  double2* buf = (double2*)work;
  double* part = (double*)((char*)work + (((size_t)n * sizeof(double2) + 255) & ~size_t(255)));
  (short_rows(g) ? k_random_spectrum<true> : k_random_spectrum<false>)<<<ROW_GRID, ROW_THREADS, 0, st>>>(
      buf, g, G.dx, G.dy, G.dz, (unsigned long long)ic.seed, ic.kc);
  cufftHandle plan;
  if (!plan_for(p.nx, p.ny, p.nz, &plan)) return cudaErrorUnknown;
  if (cufftSetStream(plan, st) != CUFFT_SUCCESS) return cudaErrorUnknown;
  if (cufftExecZ2Z(plan, (cufftDoubleComplex*)buf, (cufftDoubleComplex*)buf, CUFFT_INVERSE) != CUFFT_SUCCESS)
    return cudaErrorUnknown;
  const int nbs = 1000;
  k_sumsq<<<nbs, 256, 0, st>>>(buf, n, part);
  k_sum_parts<<<1, 256, 0, st>>>(part, nbs);
  if (esz == 16) pack_scaled(buf, part + nbs, (double2*)psi_field, g, R, p.bcs, st);
  else pack_scaled(buf, part + nbs, (float2*)psi_field, g, R, p.bcs, st);
  return cudaGetLastError();
}

size_t ic_work_bytes(const gpe_params& p, const gpe_ic& ic) {
  if (!ic_needs_fft(&ic)) return 0;
  const size_t n = (size_t)p.nx * p.ny * p.nz;
  return ((n * sizeof(double2) + 255) & ~size_t(255)) + 1024 * sizeof(double) + 256;
}

}  // namespace gpe
