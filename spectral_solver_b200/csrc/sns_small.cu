// The RK3 stage of small grids (N <= 128).  At these sizes the fields sit in L2 and a pass is
// a few microseconds: what counts is how many launches a stage takes, and that each has every
// load in flight at once and enough small CTAs to fill the chip.  So no persistent loops and no
// TMA pipelines here (they serve the large grids, six launches a stage): four launches a stage,
//   k_ysmall : inverse y of the six fields
//   k_xsmall : inverse x, the five products on both grids, forward x
//   k_ysmall : forward y of the ten product fields
//   k_zsweep : forward z of the ten fields, the k-space sweep, and the next stage's inverse z
//              of u on both grids (the first stage's is k_zphase).
// Pencils outside the sphere are neither stored by the forward y pass nor read by the inverse
// one (the state is zero there).
// Transforms of length N = R1 * R2 run as two in-place passes of register butterflies with one
// barrier between them.  Natural input leaves element k = k1 + R1 k2 in slot (k1, k2); the
// reverse order takes that layout back to natural order, so the sweep and the products, which
// do not care about the order, work on it as it lies.  Slot (a, b) sits at a (R2 + 1) + b: the
// spare element per R2 keeps both passes free of bank conflicts.
#include "sns_small.cuh"
#include "sns_sweep.cuh"

namespace sns {

namespace {

template <int A, int B>
struct Split {
  static constexpr int R1 = A, R2 = B;
  static constexpr int SLOTS = A * (B + 1);
  static __device__ __forceinline__ int slot(int a, int b) { return a * (B + 1) + b; }
  static __device__ __forceinline__ int natural(int e) { return slot(e / B, e % B); }   // element e, natural order
};
// x and y transforms: R2 small, since a thread holds three components of R2 positions
template <int N> struct XYSplit;
template <> struct XYSplit<8> : Split<2, 4> {};
template <> struct XYSplit<12> : Split<3, 4> {};
template <> struct XYSplit<16> : Split<4, 4> {};
template <> struct XYSplit<24> : Split<6, 4> {};
template <> struct XYSplit<32> : Split<8, 4> {};
template <> struct XYSplit<48> : Split<12, 4> {};
template <> struct XYSplit<64> : Split<16, 4> {};
template <> struct XYSplit<96> : Split<16, 6> {};
template <> struct XYSplit<128> : Split<16, 8> {};
// z transforms: balanced, for few registers and many resident CTAs
template <int N> struct ZSplit;
template <> struct ZSplit<8> : Split<2, 4> {};
template <> struct ZSplit<12> : Split<3, 4> {};
template <> struct ZSplit<16> : Split<4, 4> {};
template <> struct ZSplit<24> : Split<6, 4> {};
template <> struct ZSplit<32> : Split<4, 8> {};
template <> struct ZSplit<48> : Split<6, 8> {};
template <> struct ZSplit<64> : Split<8, 8> {};
template <> struct ZSplit<96> : Split<12, 8> {};
template <> struct ZSplit<128> : Split<16, 8> {};

// The four passes of a transform on one sequence: `at(slot)` is its element's index, `lim` the
// buffer's size (index checks of the debug build).
// Natural in: pass 1 of column n2 (size R1, then the twiddle), pass 2 of row k1 (size R2).
template <class S, int DIR, class C, class At>
__device__ __forceinline__ void fwd1(C* p, At at, const C* tw, int n2, int lim) {
  C v[S::R1];
#pragma unroll
  for (int r = 0; r < S::R1; ++r) v[r] = p[SNS_IDX(at(S::slot(r, n2)), lim)];
  dftR<S::R1, DIR>(v);
  p[SNS_IDX(at(S::slot(0, n2)), lim)] = v[0];
#pragma unroll
  for (int k1 = 1; k1 < S::R1; ++k1)
    p[SNS_IDX(at(S::slot(k1, n2)), lim)] = cmul(v[k1], stage_twiddle<DIR>(tw, SNS_IDX(n2 * k1, S::R1 * S::R2)));
}
template <class S, int DIR, class C, class At>
__device__ __forceinline__ void fwd2(const C* p, At at, int k1, int lim, C v[S::R2]) {
#pragma unroll
  for (int n2 = 0; n2 < S::R2; ++n2) v[n2] = p[SNS_IDX(at(S::slot(k1, n2)), lim)];
  dftR<S::R2, DIR>(v);
}
// Permuted in: pass 1 of row k1 (size R2, on registers), pass 2 of column m2 (size R1).
template <class S, int DIR, class C, class At>
__device__ __forceinline__ void rev1(C v[S::R2], C* p, At at, const C* tw, int k1, int lim) {
  dftR<S::R2, DIR>(v);
  p[SNS_IDX(at(S::slot(k1, 0)), lim)] = v[0];
#pragma unroll
  for (int m2 = 1; m2 < S::R2; ++m2)
    p[SNS_IDX(at(S::slot(k1, m2)), lim)] = cmul(v[m2], stage_twiddle<DIR>(tw, SNS_IDX(k1 * m2, S::R1 * S::R2)));
}
template <class S, int DIR, class C, class At>
__device__ __forceinline__ void rev2(const C* p, At at, int m2, int lim, C v[S::R1]) {
#pragma unroll
  for (int k1 = 0; k1 < S::R1; ++k1) v[k1] = p[SNS_IDX(at(S::slot(k1, m2)), lim)];
  dftR<S::R1, DIR>(v);
}

// Asynchronous copy of V consecutive values (8 or 16 bytes, aligned to their size).
template <int V, class C>
__device__ __forceinline__ void copy_async(C* dst, const C* src) {
  if constexpr (V * sizeof(C) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
// Programmatic dependent launch between this file's kernels: a kernel may be scheduled while
// the one before it on the stream finishes.  It waits for that one's end (and with it every
// earlier one's) before it touches anything but constants, and lets its own successor be
// scheduled when its last pass begins.  The kernels' data pointers are not __restrict__: a load
// through a restrict pointer may be moved above the wait, whatever the wait clobbers (only the
// tables, written once at a handle's creation, stay restrict).
__device__ __forceinline__ void predecessor_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Is the pencil (mx, my) wholly outside the sphere |k| <= N/2?
template <int N>
__device__ __forceinline__ bool dead_pencil(int mx, int my) {
  return 4 * (mx * mx + my * my) > N * N;
}

// ------------------------------------------------------------------------------------
// z kernels: tile of TW columns (64 bytes a row) x all mz at one my
template <int N, class C>
struct ZT {
  using S = ZSplit<N>;
  static constexpr int NH = N / 2;
  static constexpr int TW = (int)(64 / sizeof(C));
  static constexpr int NCB = (NH + TW - 1) / TW;
  static constexpr int NT = N <= 32 ? 160 : (N <= 64 ? 320 : 256);
  static constexpr int MINB = NT == 256 ? 2 : (NT == 320 ? 2 : 1);
  static constexpr int FP = S::SLOTS * TW;  // one field's tile
  static constexpr size_t smem(int fields) { return (size_t)(N + fields * FP) * sizeof(C); }
  static constexpr int MODES = (N * TW + NT - 1) / NT;  // per thread in the sweep
};

// u_hat at one mode on both grids: (scaled, scaled and shifted); modes with 0 < mx < N/2 and
// index N/2 in exactly one of y, z drop out of the shifted grid (anti-Hermitian there).
template <int N, class C>
__device__ __forceinline__ void both_grids(C u, int mx, int iy, int iz, const C* __restrict__ phase, real_of<C> sc,
                                           C* U, C* V) {
  *U = cscale(u, sc);
  const bool anti = mx > 0 && ((iy == N / 2) != (iz == N / 2));
  *V = anti ? czero<C>()
            : cmul(*U, __ldg(&phase[SNS_IDX(mx + signed_mode(iy, N) + signed_mode(iz, N) + 3 * N / 2, 3 * N + 1)]));
}

// Vorticity i k x u_hat at one mode (index N/2 -> wavenumber +N/2).
template <class C>
__device__ __forceinline__ void vorticity(const C u[3], int ix, int iy, int iz, C w[3]) {
  using RT = real_of<C>;
  const RT kx = (RT)ix, ky = (RT)iy, kz = (RT)iz;
  const C a = cmk(ky * u[2].x - kz * u[1].x, ky * u[2].y - kz * u[1].y);
  const C b = cmk(kz * u[0].x - kx * u[2].x, kz * u[0].y - kx * u[2].y);
  const C c = cmk(kx * u[1].x - ky * u[0].x, kx * u[1].y - ky * u[0].y);
  w[0] = cmk(-a.y, a.x);
  w[1] = cmk(-b.y, b.x);
  w[2] = cmk(-c.y, c.x);
}

// Inverse z of u on both grids: work fields 2c, 2c + 1; ROT (the rotational form): of the
// vorticity too, fields 6 + 2c, 7 + 2c.  grid (NCB, N).
template <int N, class C, bool ROT>
__global__ void __launch_bounds__(ZT<N, C>::NT)
k_zphase(const C* u, C* work, const C* __restrict__ phase, const C* __restrict__ tw,
         double scale, int clean, Geom g) {
  using Z = ZT<N, C>;
  using S = typename Z::S;
  constexpr int NQ = ROT ? 12 : 6;  // sequences per column
  constexpr int TW = Z::TW, NT = Z::NT, FP = Z::FP, LIM = NQ * FP, NH = Z::NH;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* const s_tw = reinterpret_cast<C*>(smraw);
  C* const buf = s_tw + N;
  const int tid = threadIdx.x, mx0 = blockIdx.x * TW, my = blockIdx.y;
  if (clean && dead_pencil<N>(mx0, signed_mode(my, N))) return;  // never read (k_ysmall)
  const real_of<C> sc = (real_of<C>)scale;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  predecessor_wait();
  if constexpr (ROT) {
    for (int e = tid; e < N * TW; e += NT) {
      const int s = e % TW, row = e / TW, mx = mx0 + s, at = S::natural(row) * TW + s;
      C f[6] = {};
      if (mx < NH) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          f[c] = u[SNS_IDX(c * g.field + ((long long)row * N + my) * g.pitch + mx, 3 * g.field)];
        vorticity(f, mx, signed_mode(my, N), signed_mode(row, N), f + 3);
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        C U = czero<C>(), V = czero<C>();
        if (mx < NH) both_grids<N>(f[q], mx, my, row, phase, sc, &U, &V);
        buf[SNS_IDX(2 * q * FP + at, LIM)] = U;
        buf[SNS_IDX((2 * q + 1) * FP + at, LIM)] = V;
      }
    }
  } else {
    for (int e = tid; e < 3 * N * TW; e += NT) {
      const int s = e % TW, row = (e / TW) % N, c = e / (TW * N);
      const int mx = mx0 + s;
      C U = czero<C>(), V = czero<C>();
      if (mx < NH)
        both_grids<N>(u[SNS_IDX(c * g.field + ((long long)row * N + my) * g.pitch + mx, 3 * g.field)], mx, my, row,
                      phase, sc, &U, &V);
      const int at = S::natural(row) * TW + s;
      buf[SNS_IDX(2 * c * FP + at, LIM)] = U;
      buf[SNS_IDX((2 * c + 1) * FP + at, LIM)] = V;
    }
  }
  __syncthreads();
  for (int b = tid; b < NQ * TW * S::R2; b += NT) {
    const int s = b % TW, n2 = (b / TW) % S::R2, f = b / (TW * S::R2);
    fwd1<S, +1>(buf, [&](int q) { return f * FP + q * TW + s; }, s_tw, n2, LIM);
  }
  __syncthreads();
  successor_start();
  for (int b = tid; b < NQ * TW * S::R1; b += NT) {
    const int s = b % TW, k1 = (b / TW) % S::R1, f = b / (TW * S::R1);
    C v[S::R2];
    fwd2<S, +1>(buf, [&](int q) { return f * FP + q * TW + s; }, k1, LIM, v);
    if (mx0 + s < NH) {
#pragma unroll
      for (int k2 = 0; k2 < S::R2; ++k2)
        work[SNS_IDX(f * g.field + ((long long)(k1 + S::R1 * k2) * N + my) * g.pitch + mx0 + s, 12 * g.field)] = v[k2];
    }
  }
}

// Forward z of the 10 product fields (ROT: the 6 of u x omega on both grids), the sweep, and
// (emit) the next stage's k_zphase on the updated u.  The state's loads are in flight while the
// fields are transformed.  grid (NCB, N).
template <int N, class C, bool ROT>
__global__ void __launch_bounds__(ZT<N, C>::NT, ZT<N, C>::MINB)
k_zsweep(C* work, C* u, C* gbuf, C* rhs,
         const double* nyq_part, int nparts, const C* __restrict__ phase, const C* __restrict__ tw,
         SweepArgs a0, int prune, int emit, double scale, Geom g) {
  using Z = ZT<N, C>;
  using S = typename Z::S;
  constexpr int NI = ROT ? 6 : 10, NQ = ROT ? 12 : 6;  // fields in, sequences out
  constexpr int TW = Z::TW, NT = Z::NT, FP = Z::FP, LIM = (ROT ? 12 : 10) * FP, NH = Z::NH, MODES = Z::MODES;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* const s_tw = reinterpret_cast<C*>(smraw);
  C* const buf = s_tw + N;
  const int tid = threadIdx.x, mx0 = blockIdx.x * TW, my = blockIdx.y;
  const int iy = signed_mode(my, N);
  // u is zero in such a tile before the stage and stays zero; its products are never needed
  if (prune && dead_pencil<N>(mx0, iy)) return;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  predecessor_wait();
  const SweepArgs a = resolve_step(a0);
  const bool load_g = a.stage > 0;

  constexpr int VL = 16 / (int)sizeof(C);  // (a row's padding past N/2 is 128-byte aligned: inside the field)
  for (int e = tid; e < NI * N * (TW / VL); e += NT) {
    const int s = e % (TW / VL) * VL, row = (e / (TW / VL)) % N, f = e / (TW / VL * N);
    copy_async<VL>(buf + SNS_IDX(f * FP + S::natural(row) * TW + s, LIM - VL + 1),
                   work + SNS_IDX(f * g.field + ((long long)row * N + my) * g.pitch + mx0 + s, 12 * g.field));
  }
  // mode i of this thread: column s, slot (k1, k2), iz index k1 + R1 k2
  auto mode = [&](int i, int* s, int* sl, int* ez) {
    const int m = tid + i * NT, q = m / TW;
    *s = m % TW;
    *sl = S::slot(q / S::R2, q % S::R2);
    *ez = q / S::R2 + S::R1 * (q % S::R2);
    return m < N * TW && mx0 + *s < NH;
  };
  C uu[MODES][3], gg[MODES][3];
  CompWord lo[MODES][3];
#pragma unroll
  for (int i = 0; i < MODES; ++i) {
    int s, sl, ez;
    const bool on = mode(i, &s, &sl, &ez);
    const long long idx = ((long long)ez * N + my) * g.pitch + mx0 + s;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      uu[i][c] = on ? u[SNS_IDX(c * g.field + idx, 3 * g.field)] : czero<C>();
      gg[i][c] = on && load_g ? gbuf[SNS_IDX(c * g.field + idx, 3 * g.field)] : czero<C>();
      lo[i][c] = on && a.ulo ? a.ulo[SNS_IDX(c * g.field + idx, 3 * g.field)] : 0;
    }
  }
  // r from the products' (or u x omega's) spectra on both grids, then the mode's update
  auto one_mode = [&](const auto& in, int ix, int iy_, int iz, C ph, C* un, C* gn, C* rr, CompWord* ln) {
    if constexpr (ROT) {
      const bool keep = 4LL * (ix * ix + iy_ * iy_ + iz * iz) <= (long long)N * N;
      C r[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) r[c] = pair_value(in.p0[c], in.ps[c], ph, keep, a.dealias);
      finish_mode(r, ix, iy_, iz, N, un, gn, load_g, rr, a, ln);
    } else {
      sweep_mode(in, ix, iy_, iz, N, ph, un, gn, load_g, rr, a, ln);
    }
  };
  copies_wait();
  __syncthreads();
  for (int b = tid; b < NI * TW * S::R2; b += NT) {
    const int s = b % TW, n2 = (b / TW) % S::R2, f = b / (TW * S::R2);
    fwd1<S, -1>(buf, [&](int q) { return f * FP + q * TW + s; }, s_tw, n2, LIM);
  }
  __syncthreads();
  for (int b = tid; b < NI * TW * S::R1; b += NT) {
    const int s = b % TW, k1 = (b / TW) % S::R1, f = b / (TW * S::R1);
    auto at = [&](int q) { return f * FP + q * TW + s; };
    C v[S::R2];
    fwd2<S, -1>(buf, at, k1, LIM, v);
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) buf[SNS_IDX(at(S::slot(k1, k2)), LIM)] = v[k2];
  }
  __syncthreads();

#pragma unroll
  for (int i = 0; i < MODES; ++i) {
    int s, sl, ez;
    const bool on = mode(i, &s, &sl, &ez);
    if (tid + i * NT >= N * TW) continue;
    const int at = sl * TW + s, ix = mx0 + s, iz = signed_mode(ez, N);
    if (on) {
      constexpr int NV = NI / 2;
      ModeIn<C, NV> in;
#pragma unroll
      for (int p = 0; p < NV; ++p) {
        in.p0[p] = buf[SNS_IDX(2 * p * FP + at, LIM)];
        in.ps[p] = buf[SNS_IDX((2 * p + 1) * FP + at, LIM)];
      }
      C rr[3];
      one_mode(in, ix, iy, iz, __ldg(&phase[SNS_IDX(ix + iy + iz + 3 * N / 2, 3 * N + 1)]), uu[i], gg[i], rr, lo[i]);
      const long long row = (long long)ez * N + my, idx = row * g.pitch + ix, inq = row * g.pitch + NH;
      const bool nyq_zero = ix == 0 && row != 0 && !a.frozen;  // the plane mx = N/2 is zero off (N/2,0,0)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (a.mode != 0) {
          rhs[SNS_IDX(c * g.field + idx, 3 * g.field)] = rr[c];
          if (nyq_zero) rhs[SNS_IDX(c * g.field + inq, 3 * g.field)] = czero<C>();
        } else {
          u[c * g.field + idx] = uu[i][c];
          gbuf[c * g.field + idx] = gg[i][c];
          if (a.ulo) a.ulo[c * g.field + idx] = lo[i][c];
          if (nyq_zero) {
            u[SNS_IDX(c * g.field + inq, 3 * g.field)] = czero<C>();
            gbuf[c * g.field + inq] = czero<C>();
            if (a.ulo) a.ulo[c * g.field + inq] = 0;
          }
        }
      }
    }
    if (emit) {  // this thread's slots: nobody else reads them any more
      C f[NQ / 2] = {};
      if (on) {
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = uu[i][c];
        if constexpr (ROT) vorticity(f, ix, iy, iz, f + 3);
      }
#pragma unroll
      for (int q = 0; q < NQ / 2; ++q) {
        C U = czero<C>(), V = czero<C>();
        if (on) both_grids<N>(f[q], ix, my, ez, phase, (real_of<C>)scale, &U, &V);
        buf[SNS_IDX(2 * q * FP + at, LIM)] = U;
        buf[SNS_IDX((2 * q + 1) * FP + at, LIM)] = V;
      }
    }
  }

  if (mx0 == 0 && my == 0) {
    // the self-conjugate mode (N/2, 0, 0): a warp per field sums the x pass's per-CTA plane
    // sums (lane-strided, then a fixed shuffle tree)
    __shared__ double s_part[NI];
    for (int f = tid / 32; f < NI; f += NT / 32) {
      double acc = 0.0;
#pragma unroll 8
      for (int i = tid % 32; i < nparts; i += 32) acc += nyq_part[f * nparts + i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (tid % 32 == 0) s_part[f] = acc;
    }
    __syncthreads();
    if (tid == 0) {
      ModeIn<C, NI / 2> in;
#pragma unroll
      for (int p = 0; p < NI / 2; ++p) {
        in.p0[p] = cmk((real_of<C>)s_part[2 * p], real_of<C>(0));
        in.ps[p] = cmk((real_of<C>)s_part[2 * p + 1], real_of<C>(0));
      }
      C un[3], gn[3], rr[3];
      CompWord ln[3] = {0, 0, 0};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        un[c] = u[c * g.field + NH];
        gn[c] = load_g ? gbuf[c * g.field + NH] : czero<C>();
        if (a.ulo) ln[c] = a.ulo[c * g.field + NH];
      }
      one_mode(in, NH, 0, 0, phase[NH + 3 * N / 2], un, gn, rr, ln);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (a.mode != 0) {
          rhs[c * g.field + NH] = rr[c];
        } else {
          u[c * g.field + NH] = un[c];
          gbuf[c * g.field + NH] = gn[c];
          if (a.ulo) a.ulo[c * g.field + NH] = ln[c];
        }
      }
    }
  }
  successor_start();
  if (!emit) return;

  __syncthreads();
  for (int b = tid; b < NQ * TW * S::R1; b += NT) {
    const int s = b % TW, k1 = (b / TW) % S::R1, f = b / (TW * S::R1);
    auto at = [&](int q) { return f * FP + q * TW + s; };
    C v[S::R2];
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) v[k2] = buf[SNS_IDX(at(S::slot(k1, k2)), LIM)];
    rev1<S, +1>(v, buf, at, s_tw, k1, LIM);
  }
  __syncthreads();
  for (int b = tid; b < NQ * TW * S::R2; b += NT) {
    const int s = b % TW, m2 = (b / TW) % S::R2, f = b / (TW * S::R2);
    C v[S::R1];
    rev2<S, +1>(buf, [&](int q) { return f * FP + q * TW + s; }, m2, LIM, v);
    if (mx0 + s < NH) {
#pragma unroll
      for (int m1 = 0; m1 < S::R1; ++m1)
        work[SNS_IDX(f * g.field + ((long long)(m1 * S::R2 + m2) * N + my) * g.pitch + mx0 + s, 12 * g.field)] = v[m1];
    }
  }
}

// ------------------------------------------------------------------------------------
// y pass, in place: F fields per CTA (first + 2 i: the fields of one grid), tiles as the z
// kernels'.  Inverse: pencils outside the sphere are zero when `clean`; forward: they are not
// stored (the sweep drops them whatever they hold).  grid (NCB, N [z], groups).
template <int N, class C, int DIR, int NF>
struct YT {
  using S = ZSplit<N>;
  static constexpr int NH = N / 2;
  static constexpr int TW = (int)(64 / sizeof(C));
  static constexpr int NCB = (NH + TW - 1) / TW;
  static constexpr int F = NF;
  static constexpr int NT = N <= 32 ? 64 : 160;
  static constexpr int FP = S::SLOTS * TW;
  static constexpr size_t smem = (size_t)(N + F * FP) * sizeof(C);
};

template <int N, class C, int DIR, int NF>
__global__ void __launch_bounds__(YT<N, C, DIR, NF>::NT)
k_ysmall(C* work, const C* __restrict__ tw, int clean, Geom g) {
  using Y = YT<N, C, DIR, NF>;
  using S = typename Y::S;
  constexpr int TW = Y::TW, NT = Y::NT, FP = Y::FP, F = Y::F, LIM = F * FP, NH = Y::NH, VL = 16 / (int)sizeof(C);
  extern __shared__ __align__(16) unsigned char smraw[];
  C* const s_tw = reinterpret_cast<C*>(smraw);
  C* const buf = s_tw + N;
  const int tid = threadIdx.x, mx0 = blockIdx.x * TW;
  const long long plane = (long long)blockIdx.y * N;
  // groups 0, 1: fields 0, 2, .. and 1, 3, ..; groups 2, 3 (12 fields): 6, 8, 10 and 7, 9, 11
  C* const fld = work + (long long)(blockIdx.z < 2 ? blockIdx.z : blockIdx.z + 4) * g.field;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  predecessor_wait();
  for (int e = tid; e < F * N * (TW / VL); e += NT) {
    const int s = e % (TW / VL) * VL, row = (e / (TW / VL)) % N, f = e / (TW / VL * N);
    C* dst = buf + SNS_IDX(f * FP + S::natural(row) * TW + s, LIM - VL + 1);
    if (DIR > 0 && clean && dead_pencil<N>(mx0 + s, signed_mode(row, N))) {
      for (int i = 0; i < VL; ++i) dst[i] = czero<C>();
    } else {
      copy_async<VL>(dst, fld + SNS_IDX(2 * f * g.field + (plane + row) * g.pitch + mx0 + s, 11 * g.field));
    }
  }
  copies_wait();
  __syncthreads();
  for (int b = tid; b < F * TW * S::R2; b += NT) {
    const int s = b % TW, n2 = (b / TW) % S::R2, f = b / (TW * S::R2);
    fwd1<S, DIR>(buf, [&](int q) { return f * FP + q * TW + s; }, s_tw, n2, LIM);
  }
  __syncthreads();
  successor_start();
  for (int b = tid; b < F * TW * S::R1; b += NT) {
    const int s = b % TW, k1 = (b / TW) % S::R1, f = b / (TW * S::R1);
    C v[S::R2];
    fwd2<S, DIR>(buf, [&](int q) { return f * FP + q * TW + s; }, k1, LIM, v);
    const int mx = mx0 + s;
    if (mx < NH) {
#pragma unroll
      for (int k2 = 0; k2 < S::R2; ++k2) {
        const int y = k1 + S::R1 * k2;
        if (DIR > 0 || !dead_pencil<N>(mx, signed_mode(y, N)))
          fld[SNS_IDX(2 * f * g.field + (plane + y) * g.pitch + mx, 11 * g.field)] = v[k2];
      }
    }
  }
}

// ------------------------------------------------------------------------------------
// x pass, in place: RB rows per CTA.  Z_c = U_c + i V_c packed on the way in, inverse x, the
// products formed in registers (a thread holds R2 positions of a row, all components), forward
// x, the two grids' half spectra unpacked on the way out.  `part`: [10][grid] Nyquist-plane sums.
// DIAG: the physical velocity's energy and vmax^2 instead: u_c on the unshifted grid (fields 0,
// 2, 4), packed u_0 + i u_1 and u_2; one (sum |u|^2 / 2, max |u|^2) pair per CTA in `part`.
// Pitch of a row in shared memory: R2 modulo a wavefront's 16 complex floats (8 complex doubles),
// so that lanes that run over R2 columns and then over rows meet no bank twice.  At 96^3 FP64 the
// padding would cost a resident CTA; its rows stay packed.
template <int N, class C, class S>
constexpr int row_stride() {
  return N == 96 && sizeof(C) == 16 ? S::SLOTS : S::SLOTS + (16 + S::R2 % 16 - S::SLOTS % 16) % 16;
}

template <int N, class C>
struct XT {
  using S = XYSplit<N>;
  static constexpr int NH = N / 2;
  static constexpr int NT = N <= 32 ? 64 : 128;
  // rows per CTA: a thread per (row, k1), a power of two that divides N^2
  static constexpr int RB = NT / S::R1 >= 32 ? 32 : (NT / S::R1 >= 16 ? 16 : (NT / S::R1 >= 8 ? 8 : 4));
  static constexpr int RP = row_stride<N, C, S>();
  static constexpr int GRID = N * N / RB;
  static constexpr size_t smem = (size_t)(N + 5 * RB * RP) * sizeof(C);
  static_assert(N * N % RB == 0 && RB * S::R1 <= NT, "whole row groups");
};

template <int N, class C, bool DIAG>
__global__ void __launch_bounds__(XT<N, C>::NT)
k_xsmall(C* work, const C* unyq, const C* __restrict__ phase, const C* __restrict__ tw,
         double scale, double* part, Geom g) {
  using X = XT<N, C>;
  using S = typename X::S;
  using RT = real_of<C>;
  constexpr int NH = X::NH, RB = X::RB, NT = X::NT, RP = X::RP, LIM = 5 * RB * RP, NC = DIAG ? 2 : 3;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* const s_tw = reinterpret_cast<C*>(smraw);
  C* const buf = s_tw + N;
  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * RB;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  predecessor_wait();
  constexpr int ITEMS = NC * RB * NH;
#pragma unroll 4
  for (int e = tid; e < ITEMS; e += NT) {
    const int k = e % NH, q = e / NH, r = q % RB, c = q / RB;
    const bool has_v = !(DIAG && c == 1);
    const long long at = (row0 + r) * g.pitch + k;
    // DIAG: u_c on the unshifted grid is field 2 c'
    const C U = work[SNS_IDX((DIAG ? 4 * c : 2 * c) * g.field + at, 12 * g.field)];
    const C V = has_v ? work[SNS_IDX((DIAG ? 2 : 2 * c + 1) * g.field + at, 12 * g.field)] : czero<C>();
    C zk, zm;
    if (k == 0) {
      // real parts only at mx = 0 and N/2 (the real part of the inverse transform); the
      // plane mx = N/2 of a masked state holds (N/2, 0, 0) alone, a constant here
      C A, B;
      if constexpr (DIAG) {
        A = cscale(unyq[SNS_IDX(2 * c * g.field + NH, 3 * g.field)], (RT)scale);
        B = has_v ? cscale(unyq[SNS_IDX((2 * c + 1) * g.field + NH, 3 * g.field)], (RT)scale) : czero<C>();
      } else {
        A = cscale(unyq[SNS_IDX(c * g.field + NH, 3 * g.field)], (RT)scale);
        B = cmul(A, phase[NH + 3 * N / 2]);
      }
      zk = cmk(U.x, V.x);
      zm = cmk(A.x, B.x);
    } else {
      zk = cmk(U.x - V.y, U.y + V.x);
      zm = cmk(U.x + V.y, V.x - U.y);
    }
    buf[SNS_IDX(q * RP + S::natural(k), LIM)] = zk;
    buf[SNS_IDX(q * RP + S::natural(k == 0 ? NH : N - k), LIM)] = zm;
  }
  __syncthreads();
  for (int b = tid; b < NC * RB * S::R2; b += NT) {
    const int n2 = b % S::R2, q = b / S::R2;
    fwd1<S, +1>(buf, [&](int sl) { return q * RP + sl; }, s_tw, n2, LIM);
  }
  __syncthreads();
  // second pass and what follows on the thread's own (row, k1): positions k1 + R1 k2
  const bool mine = tid < RB * S::R1;
  const int k1 = tid % S::R1, r = tid / S::R1;
  C zc[NC][S::R2];
  if (mine) {
#pragma unroll
    for (int c = 0; c < NC; ++c) fwd2<S, +1>(buf, [&](int sl) { return (c * RB + r) * RP + sl; }, k1, LIM, zc[c]);
  }
  if constexpr (DIAG) {
    __shared__ double red[2 * (NT / 32)];
    double es = 0.0, vm = 0.0;
    if (mine) {
#pragma unroll
      for (int k2 = 0; k2 < S::R2; ++k2) {
        const double ax = zc[0][k2].x, ay = zc[0][k2].y, cx = zc[1][k2].x;
        const double s2 = ax * ax + ay * ay + cx * cx;
        es += 0.5 * s2;
        vm = fmax(vm, s2);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      es += __shfl_xor_sync(0xffffffffu, es, o);
      vm = fmax(vm, __shfl_xor_sync(0xffffffffu, vm, o));
    }
    if (tid % 32 == 0) {
      red[2 * (tid / 32)] = es;
      red[2 * (tid / 32) + 1] = vm;
    }
    __syncthreads();
    if (tid == 0) {
      es = 0.0;
      vm = 0.0;
      for (int w = 0; w < NT / 32; ++w) {
        es += red[2 * w];
        vm = fmax(vm, red[2 * w + 1]);
      }
      part[2 * blockIdx.x] = es;
      part[2 * blockIdx.x + 1] = vm;
    }
    return;
  } else {
    __syncthreads();
    if (mine) {
#pragma unroll
      for (int p = 0; p < 5; ++p) {  // 00 - 22, 01, 02, 11 - 22, 12
        const bool sq = p == 0 || p == 3;
        const int ca = p >= 3 ? 1 : 0, cb = (sq || p == 4) ? 2 : p;
        C v[S::R2];
#pragma unroll
        for (int k2 = 0; k2 < S::R2; ++k2) {
          const C a = zc[ca][k2], b = zc[cb][k2];
          v[k2] = sq ? diff_squares(a, b) : cmk(a.x * b.x, a.y * b.y);
        }
        rev1<S, -1>(v, buf, [&](int sl) { return (p * RB + r) * RP + sl; }, s_tw, k1, LIM);
      }
    }
    __syncthreads();
    for (int b = tid; b < 5 * RB * S::R2; b += NT) {
      const int m2 = b % S::R2, q = b / S::R2;
      auto at = [&](int sl) { return q * RP + sl; };
      C v[S::R1];
      rev2<S, -1>(buf, at, m2, LIM, v);
#pragma unroll
      for (int m1 = 0; m1 < S::R1; ++m1) buf[SNS_IDX(at(S::slot(m1, m2)), LIM)] = v[m1];
    }
    __syncthreads();
    successor_start();
#pragma unroll 4
    for (int e = tid; e < 5 * RB * NH; e += NT) {
      const int k = e % NH, q = e / NH, rr = q % RB, p = q / RB;
      const C Zk = buf[SNS_IDX(q * RP + S::natural(k), LIM)];
      const C Zm = buf[SNS_IDX(q * RP + S::natural(k == 0 ? 0 : N - k), LIM)];
      const long long at = 2 * p * g.field + (row0 + rr) * g.pitch + k;
      work[SNS_IDX(at, 12 * g.field)] = cmk(RT(0.5) * (Zk.x + Zm.x), RT(0.5) * (Zk.y - Zm.y));
      work[SNS_IDX(at + g.field, 12 * g.field)] = cmk(RT(0.5) * (Zk.y + Zm.y), RT(-0.5) * (Zk.x - Zm.x));
    }
    if (tid < 10) {
      // the (N/2, 0, 0) output of the y and z transforms is the plain sum of the plane
      // mx = N/2; its values are X(N/2)'s real part on one grid, imaginary part on the other
      const int p = tid >> 1;
      double s = 0.0;
      for (int rr = 0; rr < RB; ++rr) {
        const C X = buf[SNS_IDX((p * RB + rr) * RP + S::natural(NH), LIM)];
        s += (tid & 1) ? X.y : X.x;
      }
      part[tid * gridDim.x + blockIdx.x] = s;
    }
  }
}

// x pass of the rotational form, in place: u x omega on both grids.  Six packed sequences a row
// are too many for a thread's registers, so the cross product runs point by point in shared
// memory between the two transforms.  Inputs: fields 2c, 2c + 1 (u_c), 6 + 2c, 7 + 2c (omega_c);
// outputs: fields 2c, 2c + 1.  `part`: [6][grid] Nyquist-plane sums.
template <int N, class C>
struct XR {
  using S = ZSplit<N>;
  static constexpr int NH = N / 2;
  static constexpr int NT = N <= 32 ? 64 : 128;
  static constexpr int RB = N <= 32 ? 8 : 4;
  static constexpr int RP = row_stride<N, C, S>();
  static constexpr int GRID = N * N / RB;
  static constexpr size_t smem = (size_t)(N + 6 * RB * RP) * sizeof(C);
  static_assert(N * N % RB == 0, "whole row groups");
};

template <int N, class C>
__global__ void __launch_bounds__(XR<N, C>::NT)
k_xrot(C* work, const C* unyq, const C* __restrict__ phase, const C* __restrict__ tw,
       double scale, double* part, Geom g) {
  using X = XR<N, C>;
  using S = typename X::S;
  using RT = real_of<C>;
  constexpr int NH = X::NH, RB = X::RB, NT = X::NT, RP = X::RP, LIM = 6 * RB * RP;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* const s_tw = reinterpret_cast<C*>(smraw);
  C* const buf = s_tw + N;
  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * RB;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  predecessor_wait();
#pragma unroll 4
  for (int e = tid; e < 6 * RB * NH; e += NT) {
    const int k = e % NH, q = e / NH, r = q % RB, c = q / RB;  // c: u_0 u_1 u_2 omega_0 omega_1 omega_2
    const long long at = (row0 + r) * g.pitch + k;
    const C U = work[SNS_IDX(2 * c * g.field + at, 12 * g.field)];
    const C V = work[SNS_IDX((2 * c + 1) * g.field + at, 12 * g.field)];
    C zk, zm;
    if (k == 0) {  // as k_xsmall; the vorticity of the mode (N/2, 0, 0) from u's
      C un[6];
#pragma unroll
      for (int i = 0; i < 3; ++i) un[i] = unyq[SNS_IDX(i * g.field + NH, 3 * g.field)];
      vorticity(un, NH, 0, 0, un + 3);
      C A = un[0];
#pragma unroll
      for (int i = 1; i < 6; ++i) A = c == i ? un[i] : A;
      A = cscale(A, (RT)scale);
      const C B = cmul(A, phase[NH + 3 * N / 2]);
      zk = cmk(U.x, V.x);
      zm = cmk(A.x, B.x);
    } else {
      zk = cmk(U.x - V.y, U.y + V.x);
      zm = cmk(U.x + V.y, V.x - U.y);
    }
    buf[SNS_IDX(q * RP + S::natural(k), LIM)] = zk;
    buf[SNS_IDX(q * RP + S::natural(k == 0 ? NH : N - k), LIM)] = zm;
  }
  __syncthreads();
  for (int b = tid; b < 6 * RB * S::R2; b += NT) {
    const int n2 = b % S::R2, q = b / S::R2;
    fwd1<S, +1>(buf, [&](int sl) { return q * RP + sl; }, s_tw, n2, LIM);
  }
  __syncthreads();
  for (int b = tid; b < 6 * RB * S::R1; b += NT) {
    const int k1 = b % S::R1, q = b / S::R1;
    auto at = [&](int sl) { return q * RP + sl; };
    C v[S::R2];
    fwd2<S, +1>(buf, at, k1, LIM, v);
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) buf[SNS_IDX(at(S::slot(k1, k2)), LIM)] = v[k2];
  }
  __syncthreads();
  for (int e = tid; e < RB * N; e += NT) {
    const int at = (e / N) * RP + S::natural(e % N);
    C f[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) f[c] = buf[SNS_IDX(c * RB * RP + at, LIM)];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      buf[SNS_IDX(c * RB * RP + at, LIM)] = cmk(f[a].x * f[3 + b].x - f[b].x * f[3 + a].x,
                                                f[a].y * f[3 + b].y - f[b].y * f[3 + a].y);
    }
  }
  __syncthreads();
  for (int b = tid; b < 3 * RB * S::R1; b += NT) {
    const int k1 = b % S::R1, q = b / S::R1;
    auto at = [&](int sl) { return q * RP + sl; };
    C v[S::R2];
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) v[k2] = buf[SNS_IDX(at(S::slot(k1, k2)), LIM)];
    rev1<S, -1>(v, buf, at, s_tw, k1, LIM);
  }
  __syncthreads();
  for (int b = tid; b < 3 * RB * S::R2; b += NT) {
    const int m2 = b % S::R2, q = b / S::R2;
    auto at = [&](int sl) { return q * RP + sl; };
    C v[S::R1];
    rev2<S, -1>(buf, at, m2, LIM, v);
#pragma unroll
    for (int m1 = 0; m1 < S::R1; ++m1) buf[SNS_IDX(at(S::slot(m1, m2)), LIM)] = v[m1];
  }
  __syncthreads();
  successor_start();
#pragma unroll 4
  for (int e = tid; e < 3 * RB * NH; e += NT) {
    const int k = e % NH, q = e / NH, r = q % RB, c = q / RB;
    const C Zk = buf[SNS_IDX(q * RP + S::natural(k), LIM)];
    const C Zm = buf[SNS_IDX(q * RP + S::natural(k == 0 ? 0 : N - k), LIM)];
    const long long at = 2 * c * g.field + (row0 + r) * g.pitch + k;
    work[SNS_IDX(at, 12 * g.field)] = cmk(RT(0.5) * (Zk.x + Zm.x), RT(0.5) * (Zk.y - Zm.y));
    work[SNS_IDX(at + g.field, 12 * g.field)] = cmk(RT(0.5) * (Zk.y + Zm.y), RT(-0.5) * (Zk.x - Zm.x));
  }
  if (tid < 6) {
    double s = 0.0;
    for (int r = 0; r < RB; ++r) {
      const C X_ = buf[SNS_IDX(((tid >> 1) * RB + r) * RP + S::natural(NH), LIM)];
      s += (tid & 1) ? X_.y : X_.x;
    }
    part[tid * gridDim.x + blockIdx.x] = s;
  }
}

// ------------------------------------------------------------------------------------
// Forward transform of one real field to the reference's full layout, two launches (FP64,
// N <= 64): x and y on a whole z plane per CTA, then z with the mirror half written from the
// same registers.
template <int N>
struct FT {
  using S = XYSplit<N>;
  using Z = ZSplit<N>;
  static constexpr int NH = N / 2, NC = NH + 1;
  static constexpr int NT = N <= 16 ? 64 : 256;
  static constexpr int SEQ = NH * S::SLOTS;   // N / 2 packed row pairs
  static constexpr int COL = S::SLOTS * NC;   // the plane's columns 0 .. N/2
  static constexpr size_t smem_plane = (size_t)(N + SEQ + COL) * sizeof(double2);
  static constexpr int TW = 4, NCB = (NC + TW - 1) / TW, NTZ = N <= 16 ? 32 : 64;
  static constexpr size_t smem_z = (size_t)(N + Z::SLOTS * TW) * sizeof(double2);
};

// One z plane: real rows (two per complex sequence), x, the two rows' half spectra taken
// apart, y; work rows (z, ky) of g.pitch values.  grid N.
template <int N>
__global__ void __launch_bounds__(FT<N>::NT)
k_plane_r2c(const double* __restrict__ in, double2* __restrict__ work, const double2* __restrict__ tw, Geom g) {
  using T = FT<N>;
  using S = typename T::S;
  constexpr int NT = T::NT, NH = T::NH, NC = T::NC, RP = S::SLOTS;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const s_tw = reinterpret_cast<double2*>(smraw);
  double2* const seq = s_tw + N;
  double2* const col = seq + T::SEQ;
  const int tid = threadIdx.x, z = blockIdx.x;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  for (int e = tid; e < NH * N; e += NT) {
    const int x = e % N, q = e / N;
    const double* r = in + ((long long)z * N + 2 * q) * N + x;
    seq[SNS_IDX(q * RP + S::natural(x), T::SEQ)] = make_double2(r[0], r[N]);
  }
  __syncthreads();
  for (int b = tid; b < NH * S::R2; b += NT) {
    const int n2 = b % S::R2, q = b / S::R2;
    fwd1<S, -1>(seq, [&](int sl) { return q * RP + sl; }, s_tw, n2, T::SEQ);
  }
  __syncthreads();
  for (int b = tid; b < NH * S::R1; b += NT) {
    const int k1 = b % S::R1, q = b / S::R1;
    auto at = [&](int sl) { return q * RP + sl; };
    double2 v[S::R2];
    fwd2<S, -1>(seq, at, k1, T::SEQ, v);
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) seq[SNS_IDX(at(S::slot(k1, k2)), T::SEQ)] = v[k2];
  }
  __syncthreads();
  for (int e = tid; e < NH * NC; e += NT) {
    const int k = e % NC, q = e / NC, m = k == 0 ? 0 : N - k;
    const double2 Zk = seq[SNS_IDX(q * RP + S::slot(k % S::R1, k / S::R1), T::SEQ)];
    const double2 Zm = seq[SNS_IDX(q * RP + S::slot(m % S::R1, m / S::R1), T::SEQ)];
    col[SNS_IDX(S::natural(2 * q) * NC + k, T::COL)] = make_double2(0.5 * (Zk.x + Zm.x), 0.5 * (Zk.y - Zm.y));
    col[SNS_IDX(S::natural(2 * q + 1) * NC + k, T::COL)] = make_double2(0.5 * (Zk.y + Zm.y), -0.5 * (Zk.x - Zm.x));
  }
  __syncthreads();
  for (int b = tid; b < NC * S::R2; b += NT) {
    const int c = b % NC, n2 = b / NC;
    fwd1<S, -1>(col, [&](int sl) { return sl * NC + c; }, s_tw, n2, T::COL);
  }
  __syncthreads();
  for (int b = tid; b < NC * S::R1; b += NT) {
    const int c = b % NC, k1 = b / NC;
    double2 v[S::R2];
    fwd2<S, -1>(col, [&](int sl) { return sl * NC + c; }, k1, T::COL, v);
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2)
      work[SNS_IDX(((long long)z * N + k1 + S::R1 * k2) * g.pitch + c, g.field)] = v[k2];
  }
}

// z of TW columns at one my, out to the full layout [z][y][x]: mode m and, for 0 < mx < N/2, its
// conjugate mirror.  grid (NCB, N).
template <int N>
__global__ void __launch_bounds__(FT<N>::NTZ)
k_zfull(const double2* __restrict__ work, double2* __restrict__ full, const double2* __restrict__ tw, Geom g) {
  using T = FT<N>;
  using S = typename T::Z;
  constexpr int NT = T::NTZ, TW = T::TW, LIM = S::SLOTS * TW;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const s_tw = reinterpret_cast<double2*>(smraw);
  double2* const buf = s_tw + N;
  const int tid = threadIdx.x, mx0 = blockIdx.x * TW, my = blockIdx.y;
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[t];
  for (int e = tid; e < N * TW; e += NT) {  // (columns past N/2: the row's padding, never stored)
    const int s = e % TW, row = e / TW;
    copy_async<1>(buf + SNS_IDX(S::natural(row) * TW + s, LIM),
                  work + SNS_IDX(((long long)row * N + my) * g.pitch + mx0 + s, g.field));
  }
  copies_wait();
  __syncthreads();
  for (int b = tid; b < TW * S::R2; b += NT) {
    const int s = b % TW, n2 = b / TW;
    fwd1<S, -1>(buf, [&](int q) { return q * TW + s; }, s_tw, n2, LIM);
  }
  __syncthreads();
  for (int b = tid; b < TW * S::R1; b += NT) {
    const int s = b % TW, k1 = b / TW, mx = mx0 + s;
    double2 v[S::R2];
    fwd2<S, -1>(buf, [&](int q) { return q * TW + s; }, k1, LIM, v);
    if (mx > N / 2) continue;
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) {
      const int z = k1 + S::R1 * k2;
      full[SNS_IDX(((long long)z * N + my) * N + mx, (long long)N * N * N)] = v[k2];
      if (mx > 0 && mx < N / 2)
        full[SNS_IDX(((long long)(z ? N - z : 0) * N + (my ? N - my : 0)) * N + N - mx, (long long)N * N * N)] =
            cconj(v[k2]);
    }
  }
}

template <class... P, class... A>
void launch(void (*kernel)(P...), dim3 grid, int nt, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // (the callers check cudaGetLastError)
}

template <class K>
void allow_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  // the largest carveout: several CTAs of these kernels share an SM
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}

template <int N, class C>
struct Small {
  using Z = ZT<N, C>;
  static C* F(void* p) { return static_cast<C*>(p); }
  static const C* F(const void* p) { return static_cast<const C*>(p); }
  static void init() {
    allow_smem(k_ysmall<N, C, +1, 3>, YT<N, C, +1, 3>::smem);
    allow_smem(k_ysmall<N, C, -1, 5>, YT<N, C, -1, 5>::smem);
    allow_smem(k_ysmall<N, C, -1, 3>, YT<N, C, -1, 3>::smem);
    allow_smem(k_xrot<N, C>, XR<N, C>::smem);
    allow_smem(k_xsmall<N, C, false>, XT<N, C>::smem);
    allow_smem(k_xsmall<N, C, true>, XT<N, C>::smem);
    allow_smem(k_zphase<N, C, false>, Z::smem(6));
    allow_smem(k_zphase<N, C, true>, Z::smem(12));
    allow_smem(k_zsweep<N, C, false>, Z::smem(10));
    allow_smem(k_zsweep<N, C, true>, Z::smem(12));
  }
  static void forward_init() {
    if constexpr (N <= 64) {
      allow_smem(k_plane_r2c<N>, FT<N>::smem_plane);
      allow_smem(k_zfull<N>, FT<N>::smem_z);
    }
  }
  static void forward(const double* phys, void* work, void* full, const void* tw, Geom g, cudaStream_t st) {
    if constexpr (N <= 64 && sizeof(C) == 16) {
      using T = FT<N>;
      k_plane_r2c<N><<<N, T::NT, T::smem_plane, st>>>(phys, F(work), F(tw), g);
      k_zfull<N><<<dim3(T::NCB, N), T::NTZ, T::smem_z, st>>>(F(work), F(full), F(tw), g);
    }
  }
  static void zphase(const void* u, void* work, const void* phase, const void* tw, double scale, int clean, int rot,
                     Geom g, cudaStream_t st) {
    auto k = rot ? k_zphase<N, C, true> : k_zphase<N, C, false>;
    launch(k, dim3(Z::NCB, N), Z::NT, Z::smem(rot ? 12 : 6), st, F(u), F(work), F(phase), F(tw), scale, clean, g);
  }
  static void yinv(void* work, const void* tw, int groups, int clean, Geom g, cudaStream_t st) {
    using Y = YT<N, C, +1, 3>;
    launch(k_ysmall<N, C, +1, 3>, dim3(Y::NCB, N, groups), Y::NT, Y::smem, st, F(work), F(tw), clean, g);
  }
  static void yfwd(void* work, const void* tw, int fields, Geom g, cudaStream_t st) {
    using Y5 = YT<N, C, -1, 5>;
    using Y3 = YT<N, C, -1, 3>;
    if (fields == 10) launch(k_ysmall<N, C, -1, 5>, dim3(Y5::NCB, N, 2), Y5::NT, Y5::smem, st, F(work), F(tw), 0, g);
    else launch(k_ysmall<N, C, -1, 3>, dim3(Y3::NCB, N, fields / 3), Y3::NT, Y3::smem, st, F(work), F(tw), 0, g);
  }
  static void xrot(void* work, const void* unyq, const void* phase, const void* tw, double scale, double* part, Geom g,
                   cudaStream_t st) {
    using X = XR<N, C>;
    launch(k_xrot<N, C>, X::GRID, X::NT, X::smem, st, F(work), F(unyq), F(phase), F(tw), scale, part, g);
  }
  static void xpass(void* work, const void* unyq, const void* phase, const void* tw, double scale, double* part,
                    int diag, Geom g, cudaStream_t st) {
    using X = XT<N, C>;
    launch(diag ? k_xsmall<N, C, true> : k_xsmall<N, C, false>, X::GRID, X::NT, X::smem, st, F(work), F(unyq),
           F(phase), F(tw), scale, part, g);
  }
  static void zsweep(void* work, void* u, void* gbuf, void* rhs, const double* part, int nparts, const void* phase,
                     const void* tw, SweepArgs a, int prune, int emit, int rot, double scale, Geom g,
                     cudaStream_t st) {
    auto k = rot ? k_zsweep<N, C, true> : k_zsweep<N, C, false>;
    launch(k, dim3(Z::NCB, N), Z::NT, Z::smem(rot ? 12 : 10), st, F(work), F(u), F(gbuf), F(rhs), part, nparts,
           F(phase), F(tw), a, prune, emit, scale, g);
  }
  static const SmallOps* table() {
    static const SmallOps ops = {XT<N, C>::GRID, XR<N, C>::GRID, init, zphase, yinv, xpass, xrot, yfwd, zsweep,
                                 N <= 64 && sizeof(C) == 16 ? forward_init : nullptr,
                                 N <= 64 && sizeof(C) == 16 ? forward : nullptr};
    return &ops;
  }
};

template <class C>
const SmallOps* small_for_type(int n) {
  switch (n) {
    case 8: return Small<8, C>::table();
    case 12: return Small<12, C>::table();
    case 16: return Small<16, C>::table();
    case 24: return Small<24, C>::table();
    case 32: return Small<32, C>::table();
    case 48: return Small<48, C>::table();
    case 64: return Small<64, C>::table();
    case 96: return Small<96, C>::table();
    case 128: return Small<128, C>::table();
    default: return nullptr;
  }
}

}  // namespace

const SmallOps* small_for(int n, int precision) {
  return precision == 0 ? small_for_type<double2>(n) : small_for_type<float2>(n);
}

int bounds_record_small(long long* out3) {
#ifdef SNS_BOUNDS_CHECK
  BoundsRecord r{};
  const cudaError_t e = cudaMemcpyFromSymbol(&r, g_bounds, sizeof r);
  if (e != cudaSuccess) return (int)e;
  out3[0] = (long long)r.count;
  out3[1] = r.line;
  out3[2] = r.index;
#else
  out3[0] = -1;
  out3[1] = 0;
  out3[2] = 0;
#endif
  return 0;
}

}  // namespace sns
