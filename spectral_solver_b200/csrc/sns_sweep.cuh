// Device functions of the k-space sweep shared by the pass kernels: the products, the
// dealiased pair value, the compensated state's encoding, and one mode's viscous term,
// projection and RK3 update.
#pragma once

#include "sns_fft.cuh"
#include "sns_kernels.cuh"

namespace sns {

__device__ __forceinline__ int signed_mode(int i, int n) { return i <= n / 2 ? i : i - n; }

// The products of the nonlinear term on one grid (or both: real and imaginary part).  The
// conservative form needs u_a u_b, 6 products.  A field q added to all three diagonal ones
// changes the term -i k_b FFT(u_a u_b) by -i k_a q_hat, a gradient, which the projection
// removes; q = -u_2 u_2 makes the last product zero, so every projected right-hand side
// (stepping, sns_rhs) runs on 5: u_0^2 - u_2^2, u_0 u_1, u_0 u_2, u_1^2 - u_2^2, u_1 u_2 --
// 10 instead of 12 fields through the forward passes.  sns_nonlinear returns the term
// unprojected and takes the 6.  The differences are formed as (a - b)(a + b), whose rounding
// error is relative to the difference.  A stage moves 78 instead of 86 N^3 words (g read in two
// stages of three, nothing pruned): a step at 512^3 29.1 -> 26.7 ms (FP32), at 256^3 7.1 -> 6.5 ms
// (FP64), error against 64 bits unchanged.
template <class C>
__device__ __forceinline__ C diff_squares(C a, C b) {
  return cmk((a.x - b.x) * (a.x + b.x), (a.y - b.y) * (a.y + b.y));
}

// Product ab of NP: u_a u_b, or (NP = 5, true returned) u_a^2 - u_b^2: 00 - 22, 01, 02, 11 - 22, 12.
template <int NP>
__device__ __forceinline__ bool product_pair(int ab, int* a, int* b) {
  if constexpr (NP == 5) {
    const bool sq = ab == 0 || ab == 3;
    *a = ab >= 3 ? 1 : 0;
    *b = (sq || ab == 4) ? 2 : ab;
    return sq;
  } else {
    *a = ab < 3 ? 0 : (ab < 5 ? 1 : 2);
    *b = ab < 3 ? ab : (ab < 5 ? ab - 2 : 2);
    return false;
  }
}

// ------------------------------------------------------------------------------------
// P5 sweep: per mode, the reference's accumulate (:926-936), add_viscous_project
// (:955-974), RK stage update (:994-1033) and project_truncate (:825-844).
template <class C, int NP>
struct ModeIn {
  C p0[NP];
  C ps[NP];
};

template <class C>
__device__ __forceinline__ C minus_i_k(C a, int k) {
  const real_of<C> rk = (real_of<C>)k;
  return cmk(rk * a.y, -rk * a.x);
}

// Dealiased product value of one pair at one mode (accumulate lambda, :928-931).
template <class C>
__device__ __forceinline__ C pair_value(C p0, C ps, C phase, bool keep, int dealias) {
  C value = dealias ? cscale(cadd(p0, cmulc(ps, phase)), 0.5) : p0;
  if (!keep) value = czero<C>();
  return value;
}

// Viscous term, Leray projection and mask (:955-974), then the RK stage update and the
// projection of u (:994-1039) -- or the RHS itself in modes 1 and 2.
template <class C>
__device__ __forceinline__ void finish_mode(C r[3], int ix, int iy, int iz, int n, C uu[3], C gg[3],
                                            bool load_g, C rr[3], const SweepArgs& a, CompWord lo[3]);

// Compensated state of the FP32 precision form.  The RK update u += b*dt*g adds an
// increment some 1e-3 of |u| at dt = 1e-3; rounding u to FP32 after every stage drops the
// increment's low bits, and over thousands of steps that dominates the form's error.  So u
// is carried as its stored FP32 value hi plus a remainder, and the sweep forms the update
// in FP64 from the two.  The remainder U - hi of each real part is kept as an int8 q, the
// remainder in units of ulp(hi)/255 truncated toward zero (so |q| <= 127 and the decoded
// value never reaches the rounding boundary of hi: round-to-nearest(hi + lo) == hi), and a
// decoded pair encodes back to the same pair, so states round-trip exactly through the host.
// The precision kept is about ulp(hi)/255, 2^-32 relative, against 2^-24 for FP32 alone.
// ulp(hi) = 2^(E - 150), E the biased exponent of hi (at least 1): the factors between a
// remainder and its q are 255 and 1/255 with their exponent moved, one multiplication each way.
__device__ __forceinline__ int comp_exp(float hi) {
  const int e = (int)((__float_as_uint(hi) >> 23) & 0xffu);
  return e > 0 ? e : 1;
}
// c * 2^k for a normal c, by its exponent bits
__device__ __forceinline__ double scaled(double c, int k) {
  return __hiloint2double(__double2hiint(c) + (k << 20), __double2loint(c));
}
__device__ __forceinline__ double comp_part(float hi, int q) {
  return (double)q * scaled(1.0 / 255.0, comp_exp(hi) - 150);
}
__device__ __forceinline__ int comp_q(double U, float hi) {
  const double r = (U - (double)hi) * scaled(255.0, 150 - comp_exp(hi));  // U - hi exact; |r| <= 127.5
  // toward zero, after a nudge of 1e-6 away from it: a decoded remainder (an integer up to
  // FP64 round-off) comes back as the same integer, and the bounds 63.75 (hi a power of two,
  // U below it) and 127.5 are never crossed
  return (int)(r + copysign(1.0e-6, r));
}
__device__ __forceinline__ double2 comp_decode(float2 hi, CompWord lo) {
  const int qr = (int)(int8_t)(lo & 0xffu), qi = (int)(int8_t)(lo >> 8);
  return make_double2((double)hi.x + comp_part(hi.x, qr), (double)hi.y + comp_part(hi.y, qi));
}
__device__ __forceinline__ float2 comp_encode(double2 U, CompWord* lo) {
  const float2 hi = make_float2(__double2float_rn(U.x), __double2float_rn(U.y));
  const int qr = comp_q(U.x, hi.x), qi = comp_q(U.y, hi.y);
  *lo = (CompWord)(((unsigned)(qr & 0xff)) | ((unsigned)(qi & 0xff) << 8));
  return hi;
}

// Per-stage scalars with the step taken from a device clock: the same expressions as the
// host's stage arguments (the reference's Real-typed products, :998, 1014, 1030), on the
// clock's current step size.
__device__ __forceinline__ SweepArgs resolve_step(SweepArgs a) {
  if (a.clock == nullptr) return a;
  const double dt = a.clock[kClockDt];
  a.frozen = a.clock[kClockStopped] != 0.0;
  a.nu = a.clock[kClockNu];
  if (a.stage == 0) {
    a.ub = dt / 3.0;
    a.if_tau = dt / 3.0;
  } else if (a.stage == 1) {
    a.ub = 15.0 * dt / 16.0;
    a.if_tau = 5.0 * dt / 12.0;
  } else {
    a.ub = 8.0 * dt / 15.0;
    a.if_tau = dt / 4.0;
  }
  return a;
}

template <class C, int NP>
__device__ __forceinline__ void sweep_mode(const ModeIn<C, NP>& in, int ix, int iy, int iz, int n, C phase,
                                           C uu[3], C gg[3], bool load_g, C rr[3],
                                           const SweepArgs& a, CompWord lo[3]) {
  const int m2 = ix * ix + iy * iy + iz * iz;
  const bool keep = 4LL * m2 <= (long long)n * n;
  const int kv[3] = {ix, iy, iz};
  C r[3] = {czero<C>(), czero<C>(), czero<C>()};
  const int pa[6] = {0, 0, 0, 1, 1, 2};
  const int pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const C value = pair_value(in.p0[p], in.ps[p], phase, keep, a.dealias);
    r[pa[p]] = cadd(r[pa[p]], minus_i_k(value, kv[pb[p]]));
    if (pa[p] != pb[p]) r[pb[p]] = cadd(r[pb[p]], minus_i_k(value, kv[pa[p]]));
  }
  finish_mode(r, ix, iy, iz, n, uu, gg, load_g, rr, a, lo);
}

template <class C>
__device__ __forceinline__ void finish_mode(C r[3], int ix, int iy, int iz, int n, C uu[3], C gg[3],
                                            bool load_g, C rr[3], const SweepArgs& a, CompWord lo[3]) {
  const int m2 = ix * ix + iy * iy + iz * iz;
  const bool keep = 4LL * m2 <= (long long)n * n;
  const double k2 = (double)m2;
  // the wavenumber in the form's precision (exact), and 1/k^2 formed once, in FP64
  using RT = real_of<C>;
  const RT kx = (RT)ix, ky = (RT)iy, kz = (RT)iz;
  const double inv = 1.0 / k2;
  const RT rinv = (RT)inv;
  if (a.mode == 2) {  // nonlinear term only: masked, neither viscous term nor projection
#pragma unroll
    for (int c = 0; c < 3; ++c) rr[c] = keep ? r[c] : czero<C>();
    return;
  }
  if (!a.visc_if) {
#pragma unroll
    for (int c = 0; c < 3; ++c) r[c] = csub(r[c], cscale(uu[c], (RT)(a.nu * k2)));
  }
  if (k2 > 0.0 && keep) {
    const C dot = cadd(cadd(cscale(r[0], kx), cscale(r[1], ky)), cscale(r[2], kz));
    const C factor = cscale(dot, rinv);
    r[0] = csub(r[0], cscale(factor, kx));
    r[1] = csub(r[1], cscale(factor, ky));
    r[2] = csub(r[2], cscale(factor, kz));
  } else {
    r[0] = r[1] = r[2] = czero<C>();
  }
  if (a.mode == 1) {
    rr[0] = r[0];
    rr[1] = r[1];
    rr[2] = r[2];
    return;
  }
  if (a.frozen) return;  // the solve's clock reached its horizon: u and g stay as they are
  if constexpr (sizeof(C) == 8) {
    if (a.ulo != nullptr) {
      // FP32 form with the compensated state: u = hi + lo updated and projected in FP64
      double2 U[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        gg[c] = load_g ? cadd(cscale(gg[c], (float)a.ga), r[c]) : r[c];
        U[c] = comp_decode(uu[c], lo[c]);
        U[c] = make_double2(U[c].x + a.ub * (double)gg[c].x, U[c].y + a.ub * (double)gg[c].y);
      }
      if (a.visc_if) {
        const double f = exp(-a.nu * k2 * a.if_tau);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          U[c] = make_double2(U[c].x * f, U[c].y * f);
          gg[c] = cscale(gg[c], (float)f);
        }
      }
      if (k2 > 0.0 && keep) {
        const double kv[3] = {(double)ix, (double)iy, (double)iz};
        const double2 dot = make_double2((U[0].x * kv[0] + U[1].x * kv[1]) + U[2].x * kv[2],
                                         (U[0].y * kv[0] + U[1].y * kv[1]) + U[2].y * kv[2]);
        const double2 factor = make_double2(dot.x * inv, dot.y * inv);
#pragma unroll
        for (int c = 0; c < 3; ++c) uu[c] = comp_encode(make_double2(U[c].x - factor.x * kv[c],
                                                                     U[c].y - factor.y * kv[c]), &lo[c]);
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          uu[c] = czero<C>();
          lo[c] = 0;
        }
      }
      return;
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    gg[c] = load_g ? cadd(cscale(gg[c], a.ga), r[c]) : r[c];
    uu[c] = cadd(uu[c], cscale(gg[c], a.ub));
  }
  if (a.visc_if) {
    // integrating factor to the next stage time, exponent in FP64 for either precision
    const double f = exp(-a.nu * k2 * a.if_tau);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      uu[c] = cscale(uu[c], f);
      gg[c] = cscale(gg[c], f);
    }
  }
  if (k2 > 0.0 && keep) {
    const C dot = cadd(cadd(cscale(uu[0], kx), cscale(uu[1], ky)), cscale(uu[2], kz));
    const C factor = cscale(dot, rinv);
    uu[0] = csub(uu[0], cscale(factor, kx));
    uu[1] = csub(uu[1], cscale(factor, ky));
    uu[2] = csub(uu[2], cscale(factor, kz));
  } else {
    uu[0] = uu[1] = uu[2] = czero<C>();
  }
}

}  // namespace sns
