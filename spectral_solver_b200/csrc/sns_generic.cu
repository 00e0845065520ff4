// Generic-shape transforms and the legacy solver's right-hand side on the device:
// sns_fft3d_* (the FFT-backend contract of FftwFft3D for any nx, ny, nz > 1 and any box
// lengths, src/fftw_fft.cpp:8-85 of ovankerm/Spectral_solver) and the host-vector
// SpectralNavierStokes numerics for those domains (src/spectral_solver.cpp:94-486:
// project, truncate, product_dealiased, nonlinear_rhs with or without the phase-shift pair,
// rhs, step_rk3, the diagnostics and the vorticity slice of write_vorticity_ppm).
//
// The fused pass kernels (sns_kernels.cu, sns_small.cu) serve the reference's benchmark
// domain: cubic, L = 2 pi, N in a fixed list, half spectrum.  This file serves everything
// else, in the reference's own storage: full complex fields [nz][ny][nx] of double2, x
// fastest.  One kernel transforms along any axis with a mixed-radix Stockham FFT whose radices
// are a runtime plan (register butterflies of 2 .. 8, 12 and 16; any other prime as a direct
// DFT of that length): a CTA takes TW sequences (TW consecutive x columns for the y and z
// axes, so every global access is a coalesced row segment; TW whole rows for x); the first
// stage reads global memory, the last one writes it, the stages between meet in shared memory.
//
// The dealiased solver's transforms carry two real fields in a complex one.  The reference keeps
// the real part of every inverse transform, and Re(IDFT(c)) = IDFT(H(c)) with H(c)_m =
// (c_m + conj(c_-m)) / 2, for any c.  So the first inverse pass reads Z = H(U) + i H(V) from
// the spectrum (U, V: the plain and the shifted grid of one component), the x passes work on
// u + i v, the forward passes read products formed on the fly, and the finishing kernel takes
// both spectra apart through the mirror mode.  Two components never share a transform: the
// round-off of the larger one would reach the smaller (a perturbation of a planar flow, or a
// component that is exactly zero), so without the shifted grid the imaginary part stays empty.
// A stage is 3 inverse and 5 forward complex transforms in seven launches; one transform per
// real field, with a table lookup per DFT term, took 18 and 75 launches.  Six steps at
// 96 x 80 x 60, host copies included, take 10.8 ms instead of 56.2.
#include "sns_fft.cuh"
#include "sns_kernels.cuh"
#include "../../include/sns_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <exception>
#include <new>
#include <string>
#include <vector>

namespace {

constexpr int kMaxFactors = 24;
constexpr int kNT = 256;                    // most threads per CTA of the axis kernel
constexpr size_t kSmemBudget = 200 * 1024;  // two tile buffers of L x TW complex doubles

struct AxisPlan {
  int L;                 // transform length
  int nfac;              // number of radices
  int fac[kMaxFactors];  // radices in application order (product L)
  int tw;                // sequences per tile
};

struct Dims {
  int nx, ny, nz;
};

// ------------------------------------------------------------------------------------
// Modes of the legacy solver (src/spectral_solver.cpp).  Mode numbers follow
// FftwFft3D::signed_mode (index n/2 -> +n/2), k = (2 pi m) / L per axis.
struct Modes {
  Dims d;
  double lx, ly, lz;  // box lengths
  double hx, hy, hz;  // half-cell shift L / (2 n) per axis (the phase-shift pair)
};

__device__ __forceinline__ int smode(int i, int n) { return i <= n / 2 ? i : i - n; }

struct Mode {
  double kx, ky, kz, k2;
  int mx, my, mz;
};

__device__ __forceinline__ Mode mode_of(long long id, const Modes& md) {
  constexpr double kTwoPi = 6.283185307179586476925286766559005768;
  Mode m;
  const int ix = (int)(id % md.d.nx);
  const int iy = (int)((id / md.d.nx) % md.d.ny);
  const int iz = (int)(id / ((long long)md.d.nx * md.d.ny));
  m.mx = smode(ix, md.d.nx);
  m.my = smode(iy, md.d.ny);
  m.mz = smode(iz, md.d.nz);
  m.kx = kTwoPi * m.mx / md.lx;
  m.ky = kTwoPi * m.my / md.ly;
  m.kz = kTwoPi * m.mz / md.lz;
  m.k2 = m.kx * m.kx + m.ky * m.ky + m.kz * m.kz;
  return m;
}

// keep_mode (src/spectral_solver.cpp:392-398): the ellipsoid sum (m / (n/2))^2 <= 1
__device__ __forceinline__ bool keep_of(const Mode& m, const Dims& d) {
  const double hx = d.nx / 2.0, hy = d.ny / 2.0, hz = d.nz / 2.0;
  return (m.mx * m.mx) / (hx * hx) + (m.my * m.my) / (hy * hy) + (m.mz * m.mz) / (hz * hz) <= 1.0;
}

// phase_shift_ (src/spectral_solver.cpp:48-54): exp(i (kx dx + ky dy + kz dz))
__device__ __forceinline__ double2 phase_of(const Mode& m, const Modes& md) {
  double s, c;
  sincos(m.kx * md.hx + m.ky * md.hy + m.kz * md.hz, &s, &c);
  return make_double2(c, s);
}

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ------------------------------------------------------------------------------------
// Axis transforms.
// Where a transform's elements come from: a complex field, a real field (imaginary part 0;
// FftwFft3D::forward), the packed Hermitian parts of two spectra (kPack, z axis only), or a
// product of packed physical fields (kProduct).
enum { kComplex = 0, kReal = 1, kPack = 2, kProduct = 3 };

struct AxisArgs {
  const double2* in;    // field 0; blockIdx.y steps by n3
  const double* in_real;
  double2* out;
  double* out_real;     // non-null: the real part is written there (FftwFft3D::backward)
  double scale;         // of the output
  int axis;
  Dims d;
  long long n3;
  AxisPlan plan;
  const double2* twl;   // W_L^t = exp(-2 pi i t / L)
  Modes md;             // kPack
  int shifted;          // kProduct: the input holds both grids, else the plain one (its real part)
  int nprod;            // kProduct: 5 (squares less u_2^2) or 6 products; -1: u_0 u_1 alone
};

__device__ __forceinline__ double2 mirror_of(const double2* __restrict__ f, int ix, int iy, int iz, Dims d) {
  const int jx = ix ? d.nx - ix : 0, jy = iy ? d.ny - iy : 0, jz = iz ? d.nz - iz : 0;
  return f[((long long)jz * d.ny + jy) * d.nx + jx];
}
__device__ __forceinline__ Mode mode_at(int ix, int iy, int iz, const Modes& md) {
  return mode_of(((long long)iz * md.d.ny + iy) * md.d.nx + ix, md);
}
__device__ __forceinline__ double2 herm(double2 a, double2 m) {
  return make_double2(0.5 * (a.x + m.x), 0.5 * (a.y - m.y));
}

// H(U) + i H(V) at one mode: U, V = u_f on both grids.
__device__ double2 packed_pair(const AxisArgs& a, int f, int ix, int iy, int iz) {
  const long long id = ((long long)iz * a.d.ny + iy) * a.d.nx + ix;
  const double2* u = a.in + f * a.n3;
  const double2 c = u[id], m = mirror_of(u, ix, iy, iz, a.d);
  const Mode mo = mode_at(ix, iy, iz, a.md);
  const double2 ph = phase_of(mo, a.md);
  // the mirror mode's phase: its wavenumber is -k, except +n/2 on an axis of index n/2
  const int nx = a.d.nx, ny = a.d.ny, nz = a.d.nz;
  double2 pm = make_double2(ph.x, -ph.y);
  if (2 * ix == nx || 2 * iy == ny || 2 * iz == nz)
    pm = phase_of(mode_at(ix ? nx - ix : 0, iy ? ny - iy : 0, iz ? nz - iz : 0, a.md), a.md);
  const double2 U = herm(c, m), V = herm(cm(c, ph), cm(m, pm));
  return make_double2(U.x - V.y, U.y + V.x);
}

// Product f of the physical fields at point id, on both grids or (not shifted) on the plain one:
// 00, 01, 02, 11, 12, 22, the squares less u_2^2 when only 5 are asked for (the difference is a
// gradient's, which the projection removes).
__device__ __forceinline__ double one_product(double a, double b, bool diff) {
  return diff ? (a - b) * (a + b) : a * b;
}
__device__ double2 packed_product(const AxisArgs& a, int f, long long id) {
  const int p = a.nprod < 0 ? 1 : f;
  const int x = (p >= 3) + (p >= 5);
  int y = p < 3 ? p : (p < 5 ? p - 2 : 2);
  const bool diff = a.nprod == 5 && x == y;
  if (diff) y = 2;
  const double2 u = a.in[x * a.n3 + id], v = a.in[y * a.n3 + id];
  return make_double2(one_product(u.x, v.x, diff), a.shifted ? one_product(u.y, v.y, diff) : 0.0);
}

// One Stockham stage: butterfly j of a sequence reads elements j + p L/R, multiplies by
// W_{Ns R}^(p (j mod Ns)), and writes (j / Ns) Ns R + j mod Ns + q Ns.  Lanes run over the
// sequences (axes y, z) or along the row (x), whichever is contiguous in global memory.
template <int R, int DIR, class Ld, class St>
__device__ __forceinline__ void axis_stage(const Ld& ld, const St& st, int L, int tw, bool row, int Ns,
                                           const double2* __restrict__ twl) {
  const int m = L / R, stride = m / Ns, total = tw * m;
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    int s, j;
    if (row) {
      s = b / m;
      j = b - s * m;
    } else {
      s = b & (tw - 1);  // tw is a power of two
      j = b / tw;
    }
    double2 v[R];
#pragma unroll
    for (int p = 0; p < R; ++p) v[p] = ld(s, j + p * m);
    int base = 0, k = 0;
    if (Ns > 1) {
      const int q = j / Ns;
      k = j - q * Ns;
      base = q * Ns * R + k;
#pragma unroll
      for (int p = 1; p < R; ++p) {
        double2 w = __ldg(&twl[p * k * stride]);
        if (DIR > 0) w.y = -w.y;
        v[p] = cm(v[p], w);
      }
    } else {
      base = j * R;
    }
    sns::dftR<R, DIR>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) st(s, base + q * Ns, v[q]);
  }
}

// The same for any other radix (a prime above 7), O(r) per output from shared memory: the stage
// twiddle and the DFT are one table lookup per term.
template <int DIR, class St>
__device__ void axis_stage_any(const double2* src, int es, int ss, const St& st, int L, int tw, bool row, int r,
                               int Ns, const double2* __restrict__ twl) {
  const int m = L / r, stride = m / Ns, total = tw * m;
  for (int b = threadIdx.x; b < total * r; b += blockDim.x) {
    const int q = b / total, c = b - q * total;
    int s, j;
    if (row) {
      s = c / m;
      j = c - s * m;
    } else {
      s = c & (tw - 1);
      j = c / tw;
    }
    const int k = j % Ns, a = k * stride + q * m;  // exponent step of this output (< L)
    double re = 0.0, im = 0.0;
    int e = 0;
    for (int p = 0; p < r; ++p) {
      const double2 v = src[(j + p * m) * es + s * ss];
      double2 w = __ldg(&twl[e]);
      if (DIR > 0) w.y = -w.y;
      re += v.x * w.x - v.y * w.y;
      im += v.x * w.y + v.y * w.x;
      e += a;
      if (e >= L) e -= L;
    }
    st(s, (j / Ns) * Ns * r + k + q * Ns, make_double2(re, im));
  }
}

template <int DIR, class Ld, class St>
__device__ __forceinline__ void axis_stage_switch(int r, const Ld& ld, const St& st, int L, int tw, bool row, int Ns,
                                                  const double2* __restrict__ twl) {
  switch (r) {
    case 2: axis_stage<2, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 3: axis_stage<3, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 4: axis_stage<4, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 5: axis_stage<5, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 6: axis_stage<6, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 7: axis_stage<7, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 8: axis_stage<8, DIR>(ld, st, L, tw, row, Ns, twl); break;
    case 12: axis_stage<12, DIR>(ld, st, L, tw, row, Ns, twl); break;
    default: axis_stage<16, DIR>(ld, st, L, tw, row, Ns, twl); break;
  }
}
__host__ __device__ constexpr bool register_radix(int r) { return r <= 8 || r == 12 || r == 16; }

// Transform every sequence along a.axis; grid (tiles, fields).  In place is fine: a tile is
// read whole before it is written (its last stage starts after a barrier, or, when a single
// butterfly spans the sequence, each thread writes only what it read), and tiles are disjoint.
template <int DIR, int LOAD>
__global__ void __launch_bounds__(kNT) k_axis_fft(const AxisArgs a) {
  extern __shared__ double2 sm[];
  const int L = a.plan.L, tw = a.plan.tw, fld = blockIdx.y;
  const bool row = a.axis == 0;
  const long long t = blockIdx.x;
  // element e of sequence s is base + s ss + e es, s < smax; in shared memory s sss + e ses
  long long base, es, ss;
  int smax, ix0 = 0, other = 0;
  if (row) {
    base = t * tw * a.d.nx;
    es = 1;
    ss = a.d.nx;
    const long long left = (long long)a.d.ny * a.d.nz - t * tw;
    smax = left < tw ? (int)left : tw;
  } else {
    const int xt = (a.d.nx + tw - 1) / tw;
    other = (int)(t / xt);  // iz (axis 1) or iy (axis 2)
    ix0 = (int)(t - (long long)other * xt) * tw;
    smax = a.d.nx - ix0 < tw ? a.d.nx - ix0 : tw;
    ss = 1;
    if (a.axis == 1) {
      base = (long long)other * a.d.ny * a.d.nx + ix0;
      es = a.d.nx;
    } else {
      base = (long long)other * a.d.nx + ix0;
      es = (long long)a.d.nx * a.d.ny;
    }
  }
  const int ses = row ? 1 : tw, sss = row ? L : 1;
  const double2* in = a.in + (LOAD == kComplex ? fld * a.n3 : 0);
  auto from_global = [&](int s, int e) -> double2 {
    if (s >= smax) return make_double2(0.0, 0.0);
    const long long id = base + s * ss + e * es;
    if constexpr (LOAD == kComplex) return in[id];
    else if constexpr (LOAD == kReal) return make_double2(a.in_real[id], 0.0);
    else if constexpr (LOAD == kPack) return packed_pair(a, fld, ix0 + s, other, e);
    else return packed_product(a, fld, id);
  };
  auto to_global = [&](int s, int e, double2 v) {
    if (s >= smax) return;
    const long long id = base + s * ss + e * es;
    if (a.out_real) a.out_real[id] = v.x * a.scale;
    else a.out[fld * a.n3 + id] = make_double2(v.x * a.scale, v.y * a.scale);
  };
  double2* src = sm;
  double2* dst = sm + (size_t)L * tw;  // (plans of one or two register stages never touch it)
  const int nfac = a.plan.nfac;
  int f = 0, Ns = 1;
  if (nfac == 1 && register_radix(a.plan.fac[0])) {
    axis_stage_switch<DIR>(a.plan.fac[0], from_global, to_global, L, tw, row, 1, a.twl);
    return;
  }
  auto into = [&](double2* p) { return [=](int s, int e, double2 v) { p[s * sss + e * ses] = v; }; };
  if (register_radix(a.plan.fac[0])) {
    axis_stage_switch<DIR>(a.plan.fac[0], from_global, into(src), L, tw, row, 1, a.twl);
    Ns = a.plan.fac[0];
    f = 1;
  } else {
    for (int i = threadIdx.x; i < L * tw; i += blockDim.x) {
      const int s = row ? i / L : i & (tw - 1), e = row ? i - s * L : i / tw;
      into(src)(s, e, from_global(s, e));
    }
  }
  __syncthreads();
  for (; f < nfac; ++f) {
    const int r = a.plan.fac[f];
    const bool last = f == nfac - 1;
    auto from_src = [&](int s, int e) { return src[s * sss + e * ses]; };
    if (register_radix(r)) {
      if (last) axis_stage_switch<DIR>(r, from_src, to_global, L, tw, row, Ns, a.twl);
      else axis_stage_switch<DIR>(r, from_src, into(dst), L, tw, row, Ns, a.twl);
    } else {
      if (last) axis_stage_any<DIR>(src, ses, sss, to_global, L, tw, row, r, Ns, a.twl);
      else axis_stage_any<DIR>(src, ses, sss, into(dst), L, tw, row, r, Ns, a.twl);
    }
    if (last) return;
    __syncthreads();
    Ns *= r;
    double2* tmp = src;
    src = dst;
    dst = tmp;
  }
}

// ------------------------------------------------------------------------------------
// Point-wise kernels.

// The dealiased (or plain), masked spectrum of product p at mode id from the packed
// transforms Z (nonlinear_rhs, src/spectral_solver.cpp:186-228).
__device__ double2 product_value(const double2* __restrict__ Z, int p, long long id, int ix, int iy, int iz,
                                 long long n3, Dims d, double2 ph, bool keep, int dealias) {
  if (!keep) return make_double2(0.0, 0.0);
  const double2* f = Z + p * n3;
  const double2 z = f[id];
  if (!dealias) return z;
  const double2 m = mirror_of(f, ix, iy, iz, d);
  const double2 re = herm(z, m);                                             // the real part's spectrum
  const double2 im = make_double2(0.5 * (z.y + m.y), -0.5 * (z.x - m.x));    // the imaginary part's
  const double2 sb = cm(im, make_double2(ph.x, -ph.y));
  return make_double2(0.5 * (re.x + sb.x), 0.5 * (re.y + sb.y));
}

__device__ __forceinline__ void project_mode(const Mode& m, bool drop, double2 v[3]) {
  if (m.k2 != 0.0) {
    const double2 dot = make_double2(m.kx * v[0].x + m.ky * v[1].x + m.kz * v[2].x,
                                     m.kx * v[0].y + m.ky * v[1].y + m.kz * v[2].y);
    const double2 f = make_double2(dot.x / m.k2, dot.y / m.k2);
    const double kv[3] = {m.kx, m.ky, m.kz};
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = make_double2(v[i].x - kv[i] * f.x, v[i].y - kv[i] * f.y);
  }
  if (drop) v[0] = v[1] = v[2] = make_double2(0.0, 0.0);  // zero_mean, truncate
}

// rhs_i = -i (kx P_0i + ky P_1i + kz P_2i), truncated (:230-238); for the full RHS (:242-260)
// minus nu k^2 u_hat, the projection with zero mean (:94-109, 400-409) and the truncation
// again; with g, one stage of step_rk3 (:262-309) on it: g = ga g + rhs (first stage: g = rhs),
// u += b g, project with zero mean, truncate.  nprod = 6: all products; 5: the diagonal ones
// less u_2^2 (full RHS only).
struct FinishArgs {
  const double2* Z;
  double2* u;
  double2* r;  // the right-hand side is written here (g null)
  double2* g;
  double nu, ga, b;
  int dealias, nprod, full, first;
};
__global__ void __launch_bounds__(256) k_finish(const FinishArgs a, long long n3, Modes md) {
  const long long id = (long long)blockIdx.x * 256 + threadIdx.x;
  if (id >= n3) return;
  const Mode m = mode_of(id, md);
  const int ix = (int)(id % md.d.nx), iy = (int)((id / md.d.nx) % md.d.ny);
  const int iz = (int)(id / ((long long)md.d.nx * md.d.ny));
  const bool keep = keep_of(m, md.d), drop = id == 0 || !keep;
  double2 ph = make_double2(1.0, 0.0);
  if (a.dealias && keep) ph = phase_of(m, md);
  double2 P[6];
#pragma unroll
  for (int p = 0; p < 6; ++p)
    P[p] = p < a.nprod ? product_value(a.Z, p, id, ix, iy, iz, n3, md.d, ph, keep, a.dealias)
                       : make_double2(0.0, 0.0);
  const int slot[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  double2 out[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double2 p0 = P[slot[0][i]], p1 = P[slot[1][i]], p2 = P[slot[2][i]];
    out[i] = make_double2(m.kx * p0.y + m.ky * p1.y + m.kz * p2.y, -(m.kx * p0.x + m.ky * p1.x + m.kz * p2.x));
  }
  double2 uu[3];
  if (a.full) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      uu[i] = a.u[i * n3 + id];
      out[i] = make_double2(out[i].x - a.nu * m.k2 * uu[i].x, out[i].y - a.nu * m.k2 * uu[i].y);
    }
    project_mode(m, drop, out);
  }
  if (a.g == nullptr) {
#pragma unroll
    for (int i = 0; i < 3; ++i) a.r[i * n3 + id] = out[i];
    return;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double2 gg = out[c];
    if (!a.first) {
      const double2 go = a.g[c * n3 + id];
      gg = make_double2(a.ga * go.x + gg.x, a.ga * go.y + gg.y);
    }
    a.g[c * n3 + id] = gg;
    uu[c] = make_double2(uu[c].x + a.b * gg.x, uu[c].y + a.b * gg.y);
  }
  project_mode(m, drop, uu);
#pragma unroll
  for (int c = 0; c < 3; ++c) a.u[c * n3 + id] = uu[c];
}

// product_dealiased (:122-158): one packed product's value
__global__ void __launch_bounds__(256) k_pair_value(const double2* __restrict__ Z, double2* __restrict__ out,
                                                    long long n3, Modes md) {
  const long long id = (long long)blockIdx.x * 256 + threadIdx.x;
  if (id >= n3) return;
  const Mode m = mode_of(id, md);
  const int ix = (int)(id % md.d.nx), iy = (int)((id / md.d.nx) % md.d.ny);
  const int iz = (int)(id / ((long long)md.d.nx * md.d.ny));
  out[id] = product_value(Z, 0, id, ix, iy, iz, n3, md.d, phase_of(m, md), keep_of(m, md.d), 1);
}

// omega_hat = i k x u_hat (vorticity_hat, src/spectral_solver.cpp:338-351)
__global__ void k_vorticity_hat(const double2* __restrict__ u, double2* __restrict__ w, long long n3, Modes md) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= n3) return;
  const Mode m = mode_of(id, md);
  const double2 ux = u[id], uy = u[n3 + id], uz = u[2 * n3 + id];
  const double2 cx = make_double2(m.ky * uz.x - m.kz * uy.x, m.ky * uz.y - m.kz * uy.y);
  const double2 cy = make_double2(m.kz * ux.x - m.kx * uz.x, m.kz * ux.y - m.kx * uz.y);
  const double2 cz = make_double2(m.kx * uy.x - m.ky * ux.x, m.kx * uy.y - m.ky * ux.y);
  w[id] = make_double2(-cx.y, cx.x);  // i (x + i y) = (-y, x)
  w[n3 + id] = make_double2(-cy.y, cy.x);
  w[2 * n3 + id] = make_double2(-cz.y, cz.x);
}

// Per-block partials of sum(0.5 |v|^2) and max |v|^2 over 3 real fields (fixed order).
__global__ void __launch_bounds__(256) k_sq_partials(const double* __restrict__ f, long long n3,
                                                     double* __restrict__ part) {
  __shared__ double ss[256], sm[256];
  double acc = 0.0, mx = 0.0;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n3; i += (long long)gridDim.x * 256) {
    const double a = f[i], b = f[n3 + i], c = f[2 * n3 + i];
    const double q = a * a + b * b + c * c;
    acc += 0.5 * q;
    mx = fmax(mx, q);
  }
  ss[threadIdx.x] = acc;
  sm[threadIdx.x] = mx;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      ss[threadIdx.x] += ss[threadIdx.x + o];
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = ss[0];
    part[2 * blockIdx.x + 1] = sm[0];
  }
}

// max |k . u_hat| per block (max_spectral_divergence, :367-378)
__global__ void __launch_bounds__(256) k_div_partials(const double2* __restrict__ u, long long n3, Modes md,
                                                      double* __restrict__ part) {
  __shared__ double sm[256];
  double mx = 0.0;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n3; i += (long long)gridDim.x * 256) {
    const Mode m = mode_of(i, md);
    const double2 a = u[i], b = u[n3 + i], c = u[2 * n3 + i];
    const double re = m.kx * a.x + m.ky * b.x + m.kz * c.x, im = m.kx * a.y + m.ky * b.y + m.kz * c.y;
    mx = fmax(mx, sqrt(re * re + im * im));
  }
  sm[threadIdx.x] = mx;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sm[0];
}

// |v| on one z-plane of 3 real fields -> nx * ny doubles
__global__ void k_slice_mag(const double* __restrict__ f, long long n3, long long plane0, int nxy,
                            double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nxy) return;
  const double a = f[plane0 + i], b = f[n3 + plane0 + i], c = f[2 * n3 + plane0 + i];
  out[i] = sqrt(a * a + b * b + c * c);
}

// ------------------------------------------------------------------------------------
// Host side
struct GenericError : std::exception {
  int code;
  std::string msg;
  GenericError(int c, std::string m) : code(c), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};

void gck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw GenericError(SNS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// Radices of L in application order: the primes above 7 (direct DFTs) first, then the fewest
// register butterflies of 2 .. 8, 12, 16 whose product is the rest, the largest first (the
// first stage has no twiddles); of equal counts the smallest largest radix.
bool factor(int L, AxisPlan& p) {
  p.L = L;
  p.nfac = 0;
  int rest = L;
  auto push = [&](int r) {
    if (p.nfac >= kMaxFactors) return false;
    p.fac[p.nfac++] = r;
    return true;
  };
  for (int f = 2; f <= 7; ++f)
    while (rest % f == 0) rest /= f;
  const int smooth = L / rest;
  for (int f = 11; rest > 1; f += 2) {
    if ((long long)f * f > rest) f = rest;
    while (rest % f == 0) {
      if (!push(f)) return false;
      rest /= f;
    }
  }
  static const int radix[] = {2, 3, 4, 5, 6, 7, 8, 12, 16};
  // by depth-first search: few divisors, a handful of stages
  std::vector<int> best, cur;
  auto search = [&](auto&& self, int n, int most) -> void {
    if (n == 1) {
      if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && cur[0] < best[0])) best = cur;
      return;
    }
    if (!best.empty() && cur.size() >= best.size()) return;
    for (int i = 8; i >= 0; --i)
      if (radix[i] <= most && n % radix[i] == 0) {
        cur.push_back(radix[i]);
        self(self, n / radix[i], radix[i]);
        cur.pop_back();
      }
  };
  search(search, smooth, 16);
  for (int r : best)
    if (!push(r)) return false;
  return true;
}

unsigned blocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

struct sns_fft3d {
  Dims d{};
  double len[3] = {0, 0, 0};
  int device = 0;
  cudaStream_t stream = nullptr;
  long long n3 = 0;
  AxisPlan plan[3]{};
  double2* tw[3] = {nullptr, nullptr, nullptr};
  double2* work = nullptr;  // one complex field
  double* real = nullptr;   // one real field
  // the legacy solver's working set, allocated by the first solver call
  double2* sw = nullptr;  // 18 complex fields: u (3), g (3), h (3), products (6), scratch (3)
  double* pr = nullptr;   // 3 real fields (diagnostics, the vorticity slice)
  double* part = nullptr;  // reduction partials
  double* red = nullptr;
  size_t bytes = 0;
  std::string err;
};

namespace {

constexpr int kRedBlocks = 1184;

Modes modes_of(const sns_fft3d* h) {
  Modes m;
  m.d = h->d;
  m.lx = h->len[0];
  m.ly = h->len[1];
  m.lz = h->len[2];
  m.hx = 0.5 * h->len[0] / h->d.nx;
  m.hy = 0.5 * h->len[1] / h->d.ny;
  m.hz = 0.5 * h->len[2] / h->d.nz;
  return m;
}

// One axis pass of nf fields (a.axis and the sources set by the caller).
template <int LOAD>
void launch_axis(sns_fft3d* h, int dir, AxisArgs a, int nf = 1) {
  const AxisPlan& p = h->plan[a.axis];
  const Dims& d = h->d;
  a.d = d;
  a.n3 = h->n3;
  a.plan = p;
  a.twl = h->tw[a.axis];
  long long tiles;
  if (a.axis == 0) tiles = ((long long)d.ny * d.nz + p.tw - 1) / p.tw;
  else tiles = (long long)((d.nx + p.tw - 1) / p.tw) * (a.axis == 1 ? d.nz : d.ny);
  // two register stages meet in one buffer; one needs none; a thread per butterfly of 8 points
  const bool regs = register_radix(p.fac[0]) && register_radix(p.fac[p.nfac - 1]);
  const int nbuf = regs && p.nfac <= 2 ? p.nfac - 1 : 2;
  const size_t smem = nbuf * (size_t)p.L * p.tw * sizeof(double2);
  const int nt = std::min(kNT, std::max(32, (p.L * p.tw / 8 + 31) / 32 * 32));
  const dim3 grid((unsigned)tiles, nf);
  if constexpr (LOAD == kPack) {
    k_axis_fft<+1, LOAD><<<grid, nt, smem, h->stream>>>(a);
  } else if constexpr (LOAD == kComplex) {
    if (dir < 0) k_axis_fft<-1, LOAD><<<grid, nt, smem, h->stream>>>(a);
    else k_axis_fft<+1, LOAD><<<grid, nt, smem, h->stream>>>(a);
  } else {
    k_axis_fft<-1, LOAD><<<grid, nt, smem, h->stream>>>(a);
  }
}
AxisArgs axis_args(int axis, const double2* in, double2* out, double scale = 1.0) {
  AxisArgs a{};
  a.axis = axis;
  a.in = in;
  a.out = out;
  a.scale = scale;
  return a;
}

// Forward transform of one real field into a complex field (x, y, z passes).
void forward_real(sns_fft3d* h, const double* real, double2* spec) {
  AxisArgs a = axis_args(0, nullptr, spec);
  a.in_real = real;
  launch_axis<kReal>(h, -1, a);
  launch_axis<kComplex>(h, -1, axis_args(1, spec, spec));
  launch_axis<kComplex>(h, -1, axis_args(2, spec, spec));
}

// Re(IDFT(spec)) / N into a real field; `scratch` (a complex field) may alias `spec` when the
// spectrum need not survive.
void backward_real(sns_fft3d* h, const double2* spec, double2* scratch, double* real) {
  launch_axis<kComplex>(h, +1, axis_args(2, spec, scratch));
  launch_axis<kComplex>(h, +1, axis_args(1, scratch, scratch));
  AxisArgs a = axis_args(0, scratch, nullptr, 1.0 / (double)h->n3);
  a.out_real = real;
  launch_axis<kComplex>(h, +1, a);
}

void dalloc(sns_fft3d* h, void** p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw GenericError(SNS_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  h->bytes += bytes;
}

void ensure_solver_memory(sns_fft3d* h) {
  if (h->sw) return;
  const size_t cf = (size_t)h->n3 * sizeof(double2), rf = (size_t)h->n3 * sizeof(double);
  size_t free_b = 0, total_b = 0;
  gck(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
  const size_t need = 18 * cf + 3 * rf + (2 * kRedBlocks + 16) * sizeof(double);
  if (need > free_b)
    throw GenericError(SNS_ERR_NOMEM, "the solver working set needs " + std::to_string(need) + " bytes, device has " +
                                          std::to_string(free_b) + " free");
  dalloc(h, (void**)&h->sw, 18 * cf);
  dalloc(h, (void**)&h->pr, 3 * rf);
  dalloc(h, (void**)&h->part, 2 * kRedBlocks * sizeof(double));
  dalloc(h, (void**)&h->red, 16 * sizeof(double));
}

double2* SW(sns_fft3d* h, int f) { return h->sw + (size_t)f * h->n3; }
double* PR(sns_fft3d* h, int f) { return h->pr + (size_t)f * h->n3; }
// slots of the working set
constexpr int kU = 0, kG = 3, kH = 6, kP = 9, kS = 15;

// The products' spectra of u (slots kU) into the slots from kP, packed with those on the shifted
// grid (`shifted`); the physical fields are formed in kS.
void product_spectra(sns_fft3d* h, int shifted, int nprod) {
  AxisArgs a = axis_args(2, SW(h, kU), SW(h, kS), 1.0 / (double)h->n3);
  a.md = modes_of(h);
  if (shifted) launch_axis<kPack>(h, +1, a, 3);
  else launch_axis<kComplex>(h, +1, a, 3);
  launch_axis<kComplex>(h, +1, axis_args(1, SW(h, kS), SW(h, kS)), 3);
  launch_axis<kComplex>(h, +1, axis_args(0, SW(h, kS), SW(h, kS)), 3);
  a = axis_args(0, SW(h, kS), SW(h, kP));
  a.shifted = shifted;
  a.nprod = nprod;
  launch_axis<kProduct>(h, -1, a, nprod);
  launch_axis<kComplex>(h, -1, axis_args(1, SW(h, kP), SW(h, kP)), nprod);
  launch_axis<kComplex>(h, -1, axis_args(2, SW(h, kP), SW(h, kP)), nprod);
}

// The product of the two fields in slots kU, kU + 1, on both grids, into slot kP.
void pair_spectrum(sns_fft3d* h) {
  AxisArgs a = axis_args(2, SW(h, kU), SW(h, kS), 1.0 / (double)h->n3);
  a.md = modes_of(h);
  launch_axis<kPack>(h, +1, a, 2);
  launch_axis<kComplex>(h, +1, axis_args(1, SW(h, kS), SW(h, kS)), 2);
  launch_axis<kComplex>(h, +1, axis_args(0, SW(h, kS), SW(h, kS)), 2);
  a = axis_args(0, SW(h, kS), SW(h, kP));
  a.shifted = 1;
  a.nprod = -1;  // u_0 u_1 alone
  launch_axis<kProduct>(h, -1, a);
  launch_axis<kComplex>(h, -1, axis_args(1, SW(h, kP), SW(h, kP)));
  launch_axis<kComplex>(h, -1, axis_args(2, SW(h, kP), SW(h, kP)));
}

// The right-hand side of u (slots kU; full = 0: nonlinear_rhs), or one RK stage on it.
void stage_device(sns_fft3d* h, FinishArgs f) {
  f.nprod = f.full ? 5 : 6;
  product_spectra(h, f.dealias, f.nprod);
  f.Z = SW(h, kP);
  f.u = SW(h, kU);
  k_finish<<<blocks(h->n3, 256), 256, 0, h->stream>>>(f, h->n3, modes_of(h));
}

void gsync(sns_fft3d* h, const char* what) {
  gck(cudaGetLastError(), what);
  gck(cudaStreamSynchronize(h->stream), what);
}

void upload3(sns_fft3d* h, const double* const f[3], int slot) {
  for (int c = 0; c < 3; ++c)
    gck(cudaMemcpyAsync(SW(h, slot + c), f[c], (size_t)h->n3 * sizeof(double2), cudaMemcpyHostToDevice, h->stream),
        "upload");
}
void download3(sns_fft3d* h, int slot, double* const f[3]) {
  for (int c = 0; c < 3; ++c)
    gck(cudaMemcpyAsync(f[c], SW(h, slot + c), (size_t)h->n3 * sizeof(double2), cudaMemcpyDeviceToHost, h->stream),
        "download");
}

bool null3(const void* const f[3]) { return f == nullptr || !f[0] || !f[1] || !f[2]; }

template <class F>
int guard(sns_fft3d* h, F&& f) {
  if (h == nullptr) return SNS_ERR_INVALID;
  try {
    gck(cudaSetDevice(h->device), "cudaSetDevice");
    f();
    h->err.clear();
    return SNS_OK;
  } catch (const GenericError& e) {
    h->err = e.msg;
    return e.code;
  } catch (const std::bad_alloc&) {
    h->err = "host allocation failed";
    return SNS_ERR_NOMEM;
  } catch (const std::exception& e) {
    h->err = e.what();
    return SNS_ERR_INVALID;
  }
}

void release(sns_fft3d* h) {
  if (!h) return;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto* t : h->tw) cudaFree(t);
  cudaFree(h->work);
  cudaFree(h->real);
  cudaFree(h->sw);
  cudaFree(h->pr);
  cudaFree(h->part);
  cudaFree(h->red);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

}  // namespace

extern "C" {

int sns_fft3d_create(int nx, int ny, int nz, double lx, double ly, double lz, sns_fft3d** out) {
  sns::set_handleless_error("");
  if (out == nullptr) {
    sns::set_handleless_error("null output pointer");
    return SNS_ERR_INVALID;
  }
  *out = nullptr;
  if (nx <= 1 || ny <= 1 || nz <= 1) {
    sns::set_handleless_error("FFT grid dimensions must be greater than one");
    return SNS_ERR_INVALID;
  }
  if (!(lx > 0.0) || !(ly > 0.0) || !(lz > 0.0) || !std::isfinite(lx) || !std::isfinite(ly) || !std::isfinite(lz)) {
    sns::set_handleless_error("FFT box lengths must be positive and finite");
    return SNS_ERR_INVALID;
  }
  const int n[3] = {nx, ny, nz};
  AxisPlan plans[3];
  sns_fft3d* h = nullptr;
  try {
    for (int a = 0; a < 3; ++a) {
      if (!factor(n[a], plans[a])) throw GenericError(SNS_ERR_UNSUPPORTED, "FFT axis length has too many factors");
      int tw = 8;
      while (tw > 1 && 2 * (size_t)n[a] * tw * sizeof(double2) > kSmemBudget) tw /= 2;
      if (2 * (size_t)n[a] * tw * sizeof(double2) > kSmemBudget)
        throw GenericError(SNS_ERR_UNSUPPORTED, "FFT axis length " + std::to_string(n[a]) + " is above the " +
                                                    std::to_string(kSmemBudget / (2 * sizeof(double2))) +
                                                    " points one CTA's shared memory holds");
      plans[a].tw = tw;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
      cudaGetLastError();
      throw GenericError(SNS_ERR_NO_DEVICE, "no CUDA device visible");
    }
    h = new sns_fft3d();
    gck(cudaGetDevice(&h->device), "cudaGetDevice");
    h->d = Dims{nx, ny, nz};
    h->len[0] = lx;
    h->len[1] = ly;
    h->len[2] = lz;
    h->n3 = (long long)nx * ny * nz;
    for (int a = 0; a < 3; ++a) h->plan[a] = plans[a];
    gck(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    size_t free_b = 0, total_b = 0;
    gck(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    const size_t need = (size_t)h->n3 * (sizeof(double2) + sizeof(double));
    if (need > free_b)
      throw GenericError(SNS_ERR_NOMEM, "grid needs " + std::to_string(need) + " bytes, device has " +
                                            std::to_string(free_b) + " free");
    dalloc(h, (void**)&h->work, (size_t)h->n3 * sizeof(double2));
    dalloc(h, (void**)&h->real, (size_t)h->n3 * sizeof(double));
    for (int a = 0; a < 3; ++a) {
      std::vector<double2> t((size_t)n[a]);
      sns::fill_twiddles(n[a], t.data());
      dalloc(h, (void**)&h->tw[a], t.size() * sizeof(double2));
      gck(cudaMemcpyAsync(h->tw[a], t.data(), t.size() * sizeof(double2), cudaMemcpyHostToDevice, h->stream), "tw");
      gck(cudaStreamSynchronize(h->stream), "tw");
    }
    auto allow = [](auto k) {
      gck(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget), "attr");
    };
    allow(k_axis_fft<-1, kComplex>);
    allow(k_axis_fft<-1, kReal>);
    allow(k_axis_fft<-1, kProduct>);
    allow(k_axis_fft<+1, kComplex>);
    allow(k_axis_fft<+1, kPack>);
    gsync(h, "sns_fft3d_create");
  } catch (const GenericError& e) {
    sns::set_handleless_error(e.msg.c_str());
    release(h);
    return e.code;
  } catch (const std::exception&) {  // std::bad_alloc
    sns::set_handleless_error("host allocation failed");
    release(h);
    return SNS_ERR_NOMEM;
  }
  *out = h;
  return SNS_OK;
}

int sns_fft3d_destroy(sns_fft3d* h) {
  if (h == nullptr) return SNS_ERR_INVALID;
  release(h);
  return SNS_OK;
}

const char* sns_fft3d_last_error(const sns_fft3d* h) { return h ? h->err.c_str() : "null handle"; }

size_t sns_fft3d_device_bytes(const sns_fft3d* h) { return h ? h->bytes : 0; }

int sns_fft3d_forward(sns_fft3d* h, const double* host_physical, double* host_spectral) {
  return guard(h, [&] {
    if (!host_physical || !host_spectral) throw GenericError(SNS_ERR_INVALID, "null buffer");
    gck(cudaMemcpyAsync(h->real, host_physical, (size_t)h->n3 * sizeof(double), cudaMemcpyHostToDevice, h->stream),
        "upload");
    forward_real(h, h->real, h->work);
    gck(cudaMemcpyAsync(host_spectral, h->work, (size_t)h->n3 * sizeof(double2), cudaMemcpyDeviceToHost, h->stream),
        "download");
    gsync(h, "sns_fft3d_forward");
  });
}

int sns_fft3d_backward(sns_fft3d* h, const double* host_spectral, double* host_physical) {
  return guard(h, [&] {
    if (!host_physical || !host_spectral) throw GenericError(SNS_ERR_INVALID, "null buffer");
    gck(cudaMemcpyAsync(h->work, host_spectral, (size_t)h->n3 * sizeof(double2), cudaMemcpyHostToDevice, h->stream),
        "upload");
    backward_real(h, h->work, h->work, h->real);
    gck(cudaMemcpyAsync(host_physical, h->real, (size_t)h->n3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
        "download");
    gsync(h, "sns_fft3d_backward");
  });
}

int sns_fft3d_rhs(sns_fft3d* h, double nu, int dealias, int full, const double* const uhat[3], double* const out[3]) {
  return guard(h, [&] {
    if (null3((const void* const*)uhat) || null3((const void* const*)out))
      throw GenericError(SNS_ERR_INVALID, "null buffer");
    if (!(nu >= 0.0) || (dealias != 0 && dealias != 1) || (full != 0 && full != 1))
      throw GenericError(SNS_ERR_INVALID, "nu must be >= 0, dealias and full 0 or 1");
    ensure_solver_memory(h);
    upload3(h, uhat, kU);
    FinishArgs f{};
    f.r = SW(h, kH);
    f.nu = nu;
    f.dealias = dealias;
    f.full = full;
    stage_device(h, f);
    download3(h, kH, out);
    gsync(h, "sns_fft3d_rhs");
  });
}

int sns_fft3d_step(sns_fft3d* h, double nu, int dealias, double dt, int nsteps, double* const uhat[3]) {
  return guard(h, [&] {
    if (null3((const void* const*)uhat)) throw GenericError(SNS_ERR_INVALID, "null buffer");
    if (!(nu >= 0.0) || (dealias != 0 && dealias != 1) || nsteps < 0 || !std::isfinite(dt))
      throw GenericError(SNS_ERR_INVALID, "nu must be >= 0, dealias 0 or 1, nsteps >= 0, dt finite");
    ensure_solver_memory(h);
    upload3(h, uhat, kU);
    // Williamson low-storage RK3 with the reference's coefficient products (:262-309)
    const double ga[3] = {0.0, -(5.0 / 9.0), -(153.0 / 128.0)};
    const double b[3] = {dt / 3.0, (15.0 / 16.0) * dt, (8.0 / 15.0) * dt};
    FinishArgs f{};
    f.g = SW(h, kG);
    f.nu = nu;
    f.dealias = dealias;
    f.full = 1;
    for (int s = 0; s < nsteps; ++s)
      for (int st = 0; st < 3; ++st) {
        f.ga = ga[st];
        f.b = b[st];
        f.first = st == 0;
        stage_device(h, f);
      }
    download3(h, kU, uhat);
    gsync(h, "sns_fft3d_step");
  });
}

int sns_fft3d_diagnostics(sns_fft3d* h, double nu, const double* const uhat[3], double t, sns_diag* out) {
  return guard(h, [&] {
    if (null3((const void* const*)uhat) || !out) throw GenericError(SNS_ERR_INVALID, "null buffer");
    ensure_solver_memory(h);
    upload3(h, uhat, kU);
    const Modes md = modes_of(h);
    const long long n3 = h->n3;
    for (int c = 0; c < 3; ++c) backward_real(h, SW(h, kU + c), SW(h, kS), PR(h, c));
    k_sq_partials<<<kRedBlocks, 256, 0, h->stream>>>(PR(h, 0), n3, h->part);
    sns::launch_reduce(h->part, kRedBlocks, 2, 0, h->red + 0, h->stream);
    sns::launch_reduce(h->part + 1, kRedBlocks, 2, 1, h->red + 1, h->stream);
    k_vorticity_hat<<<blocks(n3, 256), 256, 0, h->stream>>>(SW(h, kU), SW(h, kG), n3, md);
    for (int c = 0; c < 3; ++c) backward_real(h, SW(h, kG + c), SW(h, kS), PR(h, c));
    k_sq_partials<<<kRedBlocks, 256, 0, h->stream>>>(PR(h, 0), n3, h->part);
    sns::launch_reduce(h->part, kRedBlocks, 2, 0, h->red + 2, h->stream);
    k_div_partials<<<kRedBlocks, 256, 0, h->stream>>>(SW(h, kU), n3, md, h->part);
    sns::launch_reduce(h->part, kRedBlocks, 1, 1, h->red + 3, h->stream);
    double r[4];
    gck(cudaMemcpyAsync(r, h->red, sizeof r, cudaMemcpyDeviceToHost, h->stream), "download");
    gsync(h, "sns_fft3d_diagnostics");
    out->t = t;
    out->kinetic_energy = r[0] / (double)n3;
    out->enstrophy = r[2] / (double)n3;
    out->dissipation = 2.0 * nu * out->enstrophy;
    out->max_spectral_divergence = r[3];
    out->max_velocity = std::sqrt(r[1]);
  });
}

int sns_fft3d_product(sns_fft3d* h, const double* a_hat, const double* b_hat, double* out) {
  return guard(h, [&] {
    if (!a_hat || !b_hat || !out) throw GenericError(SNS_ERR_INVALID, "null buffer");
    ensure_solver_memory(h);
    const long long n3 = h->n3;
    const size_t cf = (size_t)n3 * sizeof(double2);
    gck(cudaMemcpyAsync(SW(h, kU), a_hat, cf, cudaMemcpyHostToDevice, h->stream), "upload");
    gck(cudaMemcpyAsync(SW(h, kU + 1), b_hat, cf, cudaMemcpyHostToDevice, h->stream), "upload");
    // product_dealiased (src/spectral_solver.cpp:122-158): both grids, whatever the solver's
    // dealiasing flag
    pair_spectrum(h);
    k_pair_value<<<blocks(n3, 256), 256, 0, h->stream>>>(SW(h, kP), SW(h, kH), n3, modes_of(h));
    gck(cudaMemcpyAsync(out, SW(h, kH), cf, cudaMemcpyDeviceToHost, h->stream), "download");
    gsync(h, "sns_fft3d_product");
  });
}

int sns_fft3d_vorticity_slice(sns_fft3d* h, const double* const uhat[3], int iz, double* host_mag) {
  return guard(h, [&] {
    if (null3((const void* const*)uhat) || !host_mag) throw GenericError(SNS_ERR_INVALID, "null buffer");
    if (iz < 0 || iz >= h->d.nz) throw GenericError(SNS_ERR_INVALID, "plane index out of range");
    ensure_solver_memory(h);
    upload3(h, uhat, kU);
    const long long n3 = h->n3;
    k_vorticity_hat<<<blocks(n3, 256), 256, 0, h->stream>>>(SW(h, kU), SW(h, kG), n3, modes_of(h));
    for (int c = 0; c < 3; ++c) backward_real(h, SW(h, kG + c), SW(h, kS), PR(h, c));
    const int nxy = h->d.nx * h->d.ny;
    k_slice_mag<<<blocks(nxy, 256), 256, 0, h->stream>>>(PR(h, 0), n3, (long long)iz * nxy, nxy,
                                                       reinterpret_cast<double*>(SW(h, kS)));
    gck(cudaMemcpyAsync(host_mag, SW(h, kS), (size_t)nxy * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
        "download");
    gsync(h, "sns_fft3d_vorticity_slice");
  });
}

}  // extern "C"
