// P5 of the large grids (N = 256, 512): forward z pass of the 10 (12) product fields and the whole
// k-space sweep in one persistent kernel, so the transformed products never return to HBM.
//
// A tile is 128 bytes of columns (TW = 8 complex doubles or 16 complex floats) x all mz at one
// my.  (64-byte tiles, two CTAs an SM at N = 512: 3.1 instead of 2.6 ms FP32, 5.7 instead of 4.0
// FP64; the strided rows cost by the piece.)  It arrives as a sequence of units through a ring
// of three shared-memory slots, each
// filled by TMA while the two before it are worked on:
//   units 0 .. 9   : the product fields, the plain grid's five first (work fields 0, 2, .. 8),
//                    then the shifted grid's (1, 3, .. 9); six each for the unprojected term
//   units 10 .. 17 : the state of an eighth of the tile's rows: u, and g after the first stage
// so memory is read at every moment, also while the sweep computes and stores.
//
// A field is transformed in place in its slot, N = 16 * R2: a 16-point butterfly per thread, a
// barrier, and an R2-point one that leaves 16 modes in the thread's registers.  (N = 512:
// R2 = 32 split over lane pairs, combined by a shuffle.)  Their -i k contributions accumulate
// into r_x, r_y, r_z in tensor memory.  The dealiased value is (P0 + conj(phase) Ps) / 2, and
// everything is linear in it: r accumulates the plain grid's, takes the phase once when the
// shifted grid's first contribution comes, and conj(phase) / 2 in the sweep.  Modes outside
// the sphere need no mask: the projection zeroes them.
//
// What bounds it: FP64 the memory (256^3: 0.41 ms a launch under ncu, 74 % of the copy
// bandwidth on the bytes it moves), FP32 instruction issue (61 % of the cycles, 860 instructions
// a mode of which 320 are FP32 arithmetic).  Before (three-stage transforms with five
// barriers a field, the sweep reading u and g itself, a phase product per pair), per stage:
// 256^3 0.58 -> 0.45 ms FP64, 0.35 -> 0.32 FP32; 512^3 5.39 -> 3.92 FP64, 2.82 -> 2.56 FP32.
#include "sns_p5.cuh"
#include "sns_sweep.cuh"
#include "sns_tma.cuh"

#include <algorithm>
#include <type_traits>

namespace sns {

namespace {

// The self-conjugate mode (N/2, 0, 0): one warp sums the x pass's per-CTA plane sums in a
// fixed order and runs the sweep on that single mode (column N/2 of row 0, which no P5 tile
// touches).
template <int N, class C, int NP>
__global__ void __launch_bounds__(32) k_nyq_mode(C* __restrict__ u, C* __restrict__ gbuf, C* __restrict__ rhs,
                                                 const double* __restrict__ nyq_part, int nparts,
                                                 const C* __restrict__ phase, SweepArgs a0, Geom g) {
  const SweepArgs a = resolve_step(a0);
  constexpr int NH = N / 2;
  const int tid = threadIdx.x;
  const bool load_g = a.stage > 0;
  double part[2 * NP];
#pragma unroll
  for (int f = 0; f < 2 * NP; ++f) {
    double acc = 0.0;
    for (int i = tid; i < nparts; i += 32) acc += nyq_part[f * nparts + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    part[f] = acc;
  }
  if (tid != 0) return;
  ModeIn<C, NP> in;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    in.p0[p] = cmk((real_of<C>)part[2 * p], real_of<C>(0));
    in.ps[p] = cmk((real_of<C>)part[2 * p + 1], real_of<C>(0));
  }
  C uu[3], gg[3], rr[3];
  CompWord lo[3] = {0, 0, 0};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    uu[c] = u[(long long)c * g.field + NH];
    gg[c] = load_g ? gbuf[(long long)c * g.field + NH] : czero<C>();
    if (a.ulo) lo[c] = a.ulo[(long long)c * g.field + NH];
  }
  sweep_mode(in, NH, 0, 0, N, phase[NH + 3 * N / 2], uu, gg, load_g, rr, a, lo);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (a.mode != 0) {
      rhs[(long long)c * g.field + NH] = rr[c];
    } else {
      u[(long long)c * g.field + NH] = uu[c];
      gbuf[(long long)c * g.field + NH] = gg[c];
      if (a.ulo) a.ulo[(long long)c * g.field + NH] = lo[c];
    }
  }
}

template <int N, class C, int PRODUCTS = 5>
struct P5 {
  static constexpr int NP = PRODUCTS;
  static constexpr int TW = (int)(128 / sizeof(C));
  static constexpr int LTW = TW == 16 ? 4 : 3;
  static constexpr int R2 = N / 16;
  static constexpr bool PAIR = R2 == 32;
  static constexpr int H = PAIR ? 2 : 1;        // lanes of one R2-point butterfly
  static constexpr int NT = TW * 16 * H;        // = TW * R2: one butterfly per thread in both passes
  static constexpr int M = 16;                  // modes per thread
  static constexpr int NCH = 8;                 // state units of a tile
  static constexpr int QC = M / NCH;            // modes of a thread per state unit
  static constexpr int CR = 16 * QC;            // consecutive rows of a state unit (H such runs)
  static constexpr int kF = 2 * NP, kU = kF + NCH;  // units of a tile
  static constexpr int SLOTS = 3;
  static constexpr int TILE = TW * N;
  static constexpr uint32_t kTileBytes = 128u * N;
  static constexpr int WPC = (int)(sizeof(C) / 4);
  static constexpr int CW = WPC * M;            // tensor-memory words per accumulator
  static constexpr uint32_t COLS = (NT / 32 + 3) / 4 * 3 * CW <= 256 ? 256u : 512u;
  static constexpr int BR = N < 256 ? N : 256;
  static constexpr size_t smem = (size_t)(SLOTS * TILE + N) * sizeof(C) + 128 + SLOTS * sizeof(uint64_t);
  static constexpr int MINB = N >= 512 ? 1 : 2;
  // a unit's values are in registers before they are worked on; with two CTAs an SM the slot is
  // refilled then and no barrier ends a unit (256^3 FP64 465 -> 450 us), with one CTA the
  // refill waits for the unit's end (512^3 FP32 2.60 -> 2.56 ms)
  static constexpr bool EARLY = MINB == 2;
  static_assert(NT == TW * R2 && (NT / 32 + 3) / 4 * 3 * CW <= 512, "one butterfly per thread");
  static_assert(6 * H * CR * TW <= TILE, "a state unit fits a slot");
};

template <int N, class C, int PRODUCTS = 5>
__global__ void __launch_bounds__(P5<N, C>::NT, P5<N, C>::MINB)
k_p5(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap smap, int f_u, C* __restrict__ u,
     C* __restrict__ gbuf, C* __restrict__ rhs, const C* __restrict__ tw, const C* __restrict__ phase, SweepArgs a0,
     int ncb, const int* __restrict__ live, int nlive, Geom g, int* err) {
  using P = P5<N, C, PRODUCTS>;
  using RT = real_of<C>;
  constexpr int NT = P::NT, TW = P::TW, R2 = P::R2, M = P::M, CW = P::CW, WPC = P::WPC, TILE = P::TILE, NH = N / 2;
  constexpr int QC = P::QC, CR = P::CR, H = P::H, NP = P::NP, kF = P::kF, kU = P::kU, SLOTS = P::SLOTS;
  const SweepArgs a = resolve_step(a0);
  extern __shared__ unsigned char smraw[];
  __shared__ uint32_t s_tmem;
  const uint32_t pad = (128u - (smem_u32(smraw) & 127u)) & 127u;
  C* const ring = reinterpret_cast<C*>(smraw + pad);
  C* const s_tw = ring + SLOTS * TILE;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(s_tw + N);
  const int tid = threadIdx.x, warp = tid >> 5;
  // pass-1 twiddles W_N^(n2 q) at [q][n2]: immediate offsets from the thread's column
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[SNS_IDX((t / R2) * (t % R2), N)];
  if (tid == 0) {
    for (int b = 0; b < SLOTS; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&s_tmem, P::COLS);
    tmem_relinquish();
  }
  __syncthreads();
  const uint32_t tbase = s_tmem;
  // this thread's lane and columns: r_x, r_y, r_z at CW * c
  const uint32_t tq = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 3 * CW);
  const bool load_g = a.stage > 0;

  // both passes: column s; pass 1: elements n2 + R2 r; pass 2: row k1 (its half h)
  const int s = tid & (TW - 1), n2 = tid >> P::LTW;
  const int h = P::PAIR ? (tid >> P::LTW) & 1 : 0, k1 = tid >> (P::LTW + (P::PAIR ? 1 : 0));
  // mode q of this thread: z index k1 + 16 (q + 16 h)
  auto mode_e = [&](int q) { return k1 + 16 * (q + 16 * h); };

  const int ntiles = live ? nlive : ncb * N;
  auto tile_of = [&](int t, int& cb, int& my) {
    const int idx = live ? __ldg(&live[SNS_IDX(t, nlive)]) : t;
    my = idx / ncb;
    cb = idx - my * ncb;
  };
  const int nstate = load_g ? 6 : 3;
  // the producer's place in the sequence: unit ik of tile it, into slot ib
  int it = blockIdx.x, ik = 0, ib = 0, icb = 0, imy = 0;
  auto issue = [&] {  // (thread 0)
    if (ik == 0) {
      if (it >= ntiles) return;
      tile_of(it, icb, imy);
    }
    C* const dst = ring + ib * TILE;
    if (ik < kF) {
      const int f = ik < NP ? 2 * ik : 2 * (ik - NP) + 1;
      mbar_arrive_expect_tx(&bars[ib], P::kTileBytes);
#pragma unroll
      for (int i = 0; i < N / P::BR; ++i)
        tma_load_4d(dst + i * P::BR * TW, &map, &bars[ib], icb * 2 * TW, imy, i * P::BR, f);
    } else {
      mbar_arrive_expect_tx(&bars[ib], (uint32_t)(nstate * H * CR * 128));
      for (int c = 0; c < nstate; ++c)
#pragma unroll
        for (int i = 0; i < H; ++i)
          tma_load_4d(dst + SNS_IDX((c * H + i) * CR * TW, TILE), &smap, &bars[ib], icb * 2 * TW, imy,
                      256 * i + CR * (ik - kF), c < 3 ? f_u + c : c);
    }
    ib = ib + 1 == SLOTS ? 0 : ib + 1;
    if (++ik == kU) {
      ik = 0;
      it += gridDim.x;
    }
  };
  if (tid == 0)
    for (int b = 0; b < SLOTS; ++b) issue();

  CompWord lo_n[QC][3] = {};
  bool fail = false;
  int b = 0;
  uint32_t parity = 0;
  for (int t = blockIdx.x; t < ntiles && !fail; t += gridDim.x) {
  int cb, my;
  tile_of(t, cb, my);
  const int ix = cb * TW + s, iy = signed_mode(my, N);
  const RT kx = (RT)ix, ky = (RT)iy, k1f = (RT)k1;
  // z wavenumber of mode q: index e = k1 + 16 (q + 16 h), minus N past N/2 (N/2 itself stays)
  auto kz = [&](int q) -> RT {
    if constexpr (P::PAIR) {
      if (q == 0 && h && k1 == 0) return RT(256);
      return k1f + (h ? RT(16 * q - 256) : RT(16 * q));
    } else {
      if (q == 8) return k1 == 0 ? RT(128) : k1f - RT(128);
      return k1f + RT(q < 8 ? 16 * q : 16 * q - 256);
    }
  };
  const C* const ph0 = phase + (ix + iy + 3 * N / 2);
  auto ph_of = [&](int iz) { return __ldg(ph0 + (SNS_IDX(ix + iy + iz + 3 * N / 2, 3 * N + 1) - (ix + iy + 3 * N / 2))); };
#pragma unroll 1
  for (int k = 0; k < kU; ++k) {
    // every thread polls; the next barrier tells all of them whether any wait ran out
    const bool late = !mbar_wait_bounded(&bars[b], parity);
    C* const S = ring + b * TILE;
    auto load_lo = [&](int c0) {
#pragma unroll
      for (int j = 0; j < QC; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          lo_n[j][c] = a.ulo[SNS_IDX(c * g.field + ((long long)mode_e(QC * c0 + j) * N + my) * g.pitch + ix,
                                     3 * g.field)];
    };
    auto release = [&] {  // true: a wait ran out
      fence_proxy_async_smem();
      if (__syncthreads_or(late)) return fail = true;
      if (tid == 0) issue();
      if (++b == SLOTS) {
        b = 0;
        parity ^= 1u;
      }
      return false;
    };
    if (k < kF) {
      C v[M];
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = S[SNS_IDX((n2 + R2 * r) * TW + s, TILE)];
      dft16<-1>(v);
      S[SNS_IDX(n2 * TW + s, TILE)] = v[0];
#pragma unroll
      for (int q = 1; q < 16; ++q) S[SNS_IDX((n2 + R2 * q) * TW + s, TILE)] = cmul(v[q], s_tw[SNS_IDX(q * R2 + n2, N)]);
      if (__syncthreads_or(late)) {
        fail = true;
        break;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = S[SNS_IDX((k1 * R2 + H * i + h) * TW + s, TILE)];
      if constexpr (P::EARLY) (void)release();  // (the vote above was this unit's)
      dft16<-1>(v);
      if constexpr (P::PAIR) {
        if (h) {
#pragma unroll
          for (int q = 1; q < 16; ++q) v[q] = cmul(v[q], w32<C>(q));
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const C o = shfl2_xor(v[q], TW);
          v[q] = h ? csub(o, v[q]) : cadd(v[q], o);
        }
      }
      // r_DST += -i k_KC v (first: =)
      auto add = [&](auto dst, auto kc, bool first) {
        constexpr int DST = decltype(dst)::value, KC = decltype(kc)::value;
        const uint32_t ta = tq + (uint32_t)(CW * DST);
#pragma unroll
        for (int q0 = 0; q0 < M; q0 += 8) {
          C r[8];
          (void)SNS_IDX((warp >> 2) * 3 * CW + CW * DST + WPC * q0 + 8 * WPC - 1, (long long)P::COLS);
          if (!first) tmem_ld<8>(ta + WPC * q0, r);
          else
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = czero<C>();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const RT kk = KC == 0 ? kx : (KC == 1 ? ky : kz(q0 + i));
            r[i] = cmk(r[i].x + kk * v[q0 + i].y, r[i].y - kk * v[q0 + i].x);
          }
          tmem_st<8>(ta + WPC * q0, r);
        }
      };
      using I0 = std::integral_constant<int, 0>;
      using I1 = std::integral_constant<int, 1>;
      using I2 = std::integral_constant<int, 2>;
      const bool f0 = k < NP;  // r_x, r_y, r_z are first touched by 00, 01, 02 of the plain grid
      switch (k < NP ? k : k - NP) {
        case 0: add(I0{}, I0{}, f0); break;                             // 00 (less 22 of 5)
        case 1: add(I0{}, I1{}, false); add(I1{}, I0{}, f0); break;     // 01
        case 2: add(I0{}, I2{}, false); add(I2{}, I0{}, f0); break;     // 02
        case 3: add(I1{}, I1{}, false); break;                          // 11 (less 22 of 5)
        case 4: add(I1{}, I2{}, false); add(I2{}, I1{}, false); break;  // 12
        default:
          if constexpr (NP == 6) add(I2{}, I2{}, false);                // 22
      }
      if (k == NP - 1) {  // the plain grid's part takes the phase before the shifted grid's comes
        tmem_wait_st();
#pragma unroll 1
        for (int q0 = 0; q0 < M; q0 += 4) {
          C ph[4], r[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) ph[i] = ph_of(signed_mode(mode_e(q0 + i), N));
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            tmem_ld<4>(tq + CW * c + WPC * q0, r);
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = cmul(r[i], ph[i]);
            tmem_st<4>(tq + CW * c + WPC * q0, r);
          }
        }
      }
      tmem_wait_st();
      if (k == kF - 1 && a.ulo) load_lo(0);
    } else {
      const int c0 = k - kF;
      CompWord lo[QC][3];
#pragma unroll
      for (int j = 0; j < QC; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c) lo[j][c] = lo_n[j][c];
      if (a.ulo && c0 + 1 < P::NCH) load_lo(c0 + 1);
      auto u_of = [&](int j, int c) { return S[SNS_IDX(((c * H + h) * CR + k1 + 16 * j) * TW + s, TILE)]; };
      auto g_of = [&](int j, int c) {
        return load_g ? S[SNS_IDX((((c + 3) * H + h) * CR + k1 + 16 * j) * TW + s, TILE)] : czero<C>();
      };
      [[maybe_unused]] C us[QC][3], gs[QC][3];
      if constexpr (P::EARLY) {
#pragma unroll
        for (int j = 0; j < QC; ++j)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            us[j][c] = u_of(j, c);
            gs[j][c] = g_of(j, c);
          }
        if (release()) break;
      }
#pragma unroll 1
      for (int j = 0; j < QC; ++j) {
        const int q = QC * c0 + j, ez = mode_e(q), iz = signed_mode(ez, N);
        __syncwarp();  // (tensor-memory loads are warp-wide)
        C uu[3], gg[3], rr[3], r3[3];
        CompWord l3[3];
        const C ph = ph_of(iz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if constexpr (P::EARLY) {
            uu[c] = j == 0 ? us[0][c] : us[QC - 1][c];
            gg[c] = j == 0 ? gs[0][c] : gs[QC - 1][c];
          } else {
            uu[c] = u_of(j, c);
            gg[c] = g_of(j, c);
          }
          r3[c] = cscale(cmulc(tmem_ld1<C>(tq + CW * c + WPC * q), ph), RT(0.5));
          l3[c] = j == 0 ? lo[0][c] : lo[QC - 1][c];
        }
        static_assert(QC == 2, "one of two is picked");
        finish_mode(r3, ix, iy, iz, N, uu, gg, load_g, rr, a, l3);
        if (ix < NH) {
          const long long row = (long long)ez * N + my;
          const long long idx = SNS_IDX(row * g.pitch + ix, g.field), inq = SNS_IDX(row * g.pitch + NH, g.field);
          const bool nyq_zero = ix == 0 && row != 0 && !a.frozen;  // the plane mx = N/2 is zero off (N/2,0,0)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (a.mode != 0) {
              rhs[c * g.field + idx] = rr[c];
              if (nyq_zero) rhs[c * g.field + inq] = czero<C>();
            } else {
              u[c * g.field + idx] = uu[c];
              gbuf[c * g.field + idx] = gg[c];
              if (a.ulo) a.ulo[c * g.field + idx] = l3[c];
              if (nyq_zero) {
                u[c * g.field + inq] = czero<C>();
                gbuf[c * g.field + inq] = czero<C>();
                if (a.ulo) a.ulo[c * g.field + inq] = 0;
              }
            }
          }
        }
      }
    }
    if constexpr (!P::EARLY) {
      if (release()) break;
    }
  }
  }
  if (fail) {
    if (tid == 0) {
      atomicExch(err, kErrTmaTimeout);
      // let every copy in flight land (bounded) before the CTA gives up its shared memory: each
      // slot holds one issued unit at most; a phase that already completed reads as landed
      for (int b = 0; b < SLOTS; ++b) {
        (void)mbar_wait_bounded(&bars[b], 0u);
        (void)mbar_wait_bounded(&bars[b], 1u);
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, P::COLS);
}

template <int N, class C>
struct LaunchP5 {
  using P = P5<N, C>;
  static C* F(void* p) { return static_cast<C*>(p); }
  static const C* F(const void* p) { return static_cast<const C*>(p); }
  template <int NP>
  static void prepare() {
    cudaFuncSetAttribute(k_p5<N, C, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::smem);
    cudaFuncSetAttribute(k_p5<N, C, NP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
  }
  static void init() {
    prepare<5>();
    prepare<6>();
  }
  // The runtime's occupancy query reports one CTA per SM for a tensor-memory kernel whatever
  // its allocation, so residency is computed from the kernel's own limits: shared memory,
  // registers, threads, and its tensor-memory columns (512 per SM).
  static int grid(int nsm) {
    int dev = 0, smem_sm = 0, smem_rsv = 0, regs_sm = 0, thr_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&smem_rsv, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, k_p5<N, C>);
    const long long smem_cta = (long long)P::smem + fa.sharedSizeBytes + smem_rsv;
    const long long regs_cta = (long long)((fa.numRegs + 7) / 8 * 8) * P::NT;
    int nb = 512 / (int)P::COLS;
    if (smem_cta > 0) nb = (int)std::min<long long>(nb, smem_sm / smem_cta);
    if (regs_cta > 0) nb = (int)std::min<long long>(nb, regs_sm / regs_cta);
    nb = std::min(nb, thr_sm / P::NT);
    return nsm * (nb < 1 ? 1 : nb);
  }
  template <int NP>
  static void go(const CUtensorMap& work, const CUtensorMap& state, int f_u, void* u, void* gbuf, void* rhs,
                 const double* nyq_part, int nparts, const void* tw, const void* phase, SweepArgs a, int ncb,
                 const int* live, int nlive, Geom g, int grid, int* err, cudaStream_t st) {
    k_nyq_mode<N, C, NP><<<1, 32, 0, st>>>(F(u), F(gbuf), F(rhs), nyq_part, nparts, F(phase), a, g);
    k_p5<N, C, NP><<<grid, P::NT, P::smem, st>>>(work, state, f_u, F(u), F(gbuf), F(rhs), F(tw), F(phase), a, ncb,
                                                 live, nlive, g, err);
  }
  static void run(const CUtensorMap& work, const CUtensorMap& state, int np, int f_u, void* u, void* gbuf, void* rhs,
                  const double* nyq_part, int nparts, const void* tw, const void* phase, SweepArgs a, int ncb,
                  const int* live, int nlive, Geom g, int grid, int* err, cudaStream_t st) {
    auto launch = np == 6 ? go<6> : go<5>;
    launch(work, state, f_u, u, gbuf, rhs, nyq_part, nparts, tw, phase, a, ncb, live, nlive, g, grid, err, st);
  }
  static const P5Ops* table() {
    static const P5Ops ops = {init, grid, P::CR, run};
    return &ops;
  }
};

}  // namespace

const P5Ops* p5_for(int n, int precision) {
  if (n == 256) return precision == 0 ? LaunchP5<256, double2>::table() : LaunchP5<256, float2>::table();
  if (n == 512) return precision == 0 ? LaunchP5<512, double2>::table() : LaunchP5<512, float2>::table();
  return nullptr;
}

int bounds_record_p5(long long* out3) {
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
