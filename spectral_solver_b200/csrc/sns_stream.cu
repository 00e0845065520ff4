// z and inverse y passes of the large grids (N = 256, 512), persistent and TMA-fed.  A tile is 128 bytes
// of columns (TW = 8 complex doubles or 16 complex floats) x the N elements of the axis; tiles
// land in a ring of shared-memory slots (no multicast) while the ones before are transformed
// in place: N = 16 * R2, a 16-point butterfly per thread, one barrier, an R2-point one (N = 512:
// R2 = 32 split over lane pairs, combined by a shuffle) whose outputs go straight to HBM as
// 128-byte row segments.  Variant 1 is the inverse z pass of u_hat with the phase shift: one
// read, two transforms (the shifted grid's through a work buffer beside the ring), two outputs.
//
// The truncation sphere saves traffic, bit for bit: pencils (mx, my) outside the disk
// 4 (mx^2 + my^2) <= N^2 hold nothing but modes that every stage zeroes.  With u known zero
// there, variant 1 skips their tiles and inverse y reads them as zeros, and does not load the
// row blocks that hold nothing else.
//
// What bounds it: memory (512^3 FP32: variant 1 4.8, inverse y 5.9 TB/s moved).  Per stage, three
// radix stages through a work buffer with five barriers a tile on all pencils (k_yz_tma) -> here:
//   variant 1  256^3 FP64 250 -> 202 us, FP32 126 -> 109; 512^3 FP64 2.26 -> 1.57 ms, FP32 1.02 -> 0.87
//   inverse y  256^3 FP64 298 -> 318 us, FP32 158 -> 159; 512^3 FP64 2.31 -> 1.95 ms, FP32 1.01 -> 1.02
// (inverse y must read the skipped pencils as zeros, so it goes with variant 1 at every size).
// Forward y keeps k_yz_tma, whose two butterflies per thread hide more latency: here, with the
// pencils outside not stored, 512^3 FP64 3.5 .. 3.9 ms (3.8), FP32 1.84 (1.72), 256^3 525 us (512)
// and 273 (266).
#include "sns_stream.cuh"
#include "sns_sweep.cuh"
#include "sns_tma.cuh"

namespace sns {

namespace {

template <int N, class C, int VARIANT>
struct YZ {
  static constexpr int TW = (int)(128 / sizeof(C));
  static constexpr int LTW = TW == 16 ? 4 : 3;
  static constexpr int R2 = N / 16;
  static constexpr bool PAIR = R2 == 32;
  static constexpr int H = PAIR ? 2 : 1;      // lanes of one R2-point butterfly
  static constexpr int NT = TW * R2;          // one butterfly per thread in both passes
  static constexpr int SLOTS = VARIANT ? 2 : 3;
  static constexpr int TILE = TW * N;
  static constexpr int PART = 64;             // rows of a partial box
  static constexpr size_t smem =
      (size_t)(3 * TILE + N) * sizeof(C) + 128 + SLOTS * sizeof(uint64_t) + (N / 2 + 1) * sizeof(int);
  static constexpr int MINB = N >= 512 ? 1 : 2;
  // both transforms' second inputs in registers at once, so that no barrier ends a tile: not at
  // 512 threads of 128 registers (variant 1 at 512^3 FP32: 0.91 ms; 0.84 with the barrier)
  static constexpr bool EARLY = !(VARIANT == 1 && NT == 512);
  static_assert(NT == TW * 16 * H, "one butterfly per thread");
};

// Pass 2 of the thread's column s, row k1, half h: its inputs from slot S, and the butterfly,
// which leaves v[q] = element k1 + 16 (q + 16 h).
template <class Y, class C>
__device__ __forceinline__ void pass2_load(const C* S, int s, int k1, int h, C v[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = S[SNS_IDX((k1 * Y::R2 + Y::H * i + h) * Y::TW + s, Y::TILE)];
}
template <int DIR, class Y, class C>
__device__ __forceinline__ void pass2(int h, C v[16]) {
  dft16<DIR>(v);
  if constexpr (Y::PAIR) {
    if (h) {
#pragma unroll
      for (int q = 1; q < 16; ++q) v[q] = DIR < 0 ? cmul(v[q], w32<C>(q)) : cmulc(v[q], w32<C>(q));
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const C o = shfl2_xor(v[q], Y::TW);
      v[q] = h ? csub(o, v[q]) : cadd(v[q], o);
    }
  }
}

template <int N, int DIR, class Y, class C>
__device__ __forceinline__ void pass1(C v[16], C* S, const C* s_tw, int s, int n2) {
  dft16<DIR>(v);
  S[SNS_IDX(n2 * Y::TW + s, Y::TILE)] = v[0];
#pragma unroll
  for (int q = 1; q < 16; ++q) {
    const C w = s_tw[SNS_IDX(q * Y::R2 + n2, N)];
    S[SNS_IDX((n2 + Y::R2 * q) * Y::TW + s, Y::TILE)] = DIR < 0 ? cmul(v[q], w) : cmulc(v[q], w);
  }
}

template <int N, int AXIS, int DIR, int VARIANT, bool PARTS, class C>
__global__ void __launch_bounds__(YZ<N, C, VARIANT>::NT, YZ<N, C, VARIANT>::MINB)
k_stream(const __grid_constant__ CUtensorMap map, TmaArgs a, const C* __restrict__ tw, const C* __restrict__ phase,
         Geom g) {
  using Y = YZ<N, C, VARIANT>;
  using RT = real_of<C>;
  constexpr int NT = Y::NT, TW = Y::TW, R2 = Y::R2, TILE = Y::TILE, SLOTS = Y::SLOTS, PART = Y::PART;
  constexpr int BR = PARTS ? PART : (N < 256 ? N : 256);
  static_assert(!PARTS || (AXIS == 1 && DIR > 0), "partial loads belong to the inverse y pass");
  static_assert(AXIS == 2 || DIR > 0, "forward y is k_yz_tma's");
  extern __shared__ unsigned char smraw[];
  const uint32_t pad = (128u - (smem_u32(smraw) & 127u)) & 127u;
  C* const ring = reinterpret_cast<C*>(smraw + pad);
  C* const W = ring + 2 * TILE;  // variant 1
  C* const s_tw = ring + 3 * TILE;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(s_tw + N);
  int* const s_disk = reinterpret_cast<int*>(bars + SLOTS);  // column mx: largest |my| inside the disk
  __shared__ int3 s_tile[SLOTS];                             // the slots' tiles: (cb, c, field)
  const int tid = threadIdx.x;
  // pass-1 twiddles W_N^(n2 q) at [q][n2]: immediate offsets from the thread's column
  for (int t = tid; t < N; t += NT) s_tw[t] = tw[SNS_IDX((t / R2) * (t % R2), N)];
  for (int mx = tid; mx <= N / 2; mx += NT) {  // 4 (mx^2 + my^2) <= N^2
    const int r2 = N * N / 4 - mx * mx;
    int m = (int)sqrtf((float)r2);
    while (m * m > r2) --m;
    while ((m + 1) * (m + 1) <= r2) ++m;
    s_disk[mx] = m;
  }
  if (tid == 0) {
    for (int b = 0; b < SLOTS; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const int s = tid & (TW - 1), n2 = tid >> Y::LTW;
  const int h = Y::PAIR ? (tid >> Y::LTW) & 1 : 0, k1 = tid >> (Y::LTW + (Y::PAIR ? 1 : 0));

  // tile t: column block cb (fastest), the other coordinate c, field f; with a live list the
  // listed (c, cb) of each field
  const int per = a.live ? a.nlive : N * a.ncb, ntiles = a.nf * per;
  auto tile_of = [&](int t, int& cb, int& c, int& f) {
    f = t / per;
    int idx = t - f * per;
    if (a.live) idx = __ldg(&a.live[SNS_IDX(idx, a.nlive)]);
    c = idx / a.ncb;
    cb = idx - c * a.ncb;
  };
  int it = blockIdx.x, ib = 0;  // the producer's place
  auto issue = [&] {            // (thread 0)
    if (it >= ntiles) return;
    int cb, c, f;
    tile_of(it, cb, c, f);
    s_tile[ib] = make_int3(cb, c, f);
    f += a.f_in0;
    C* const dst = ring + ib * TILE;
    if constexpr (PARTS) {
      // row blocks [BR i, BR i + BR): rows up to m, or from N - m
      const int m = s_disk[SNS_IDX(cb * TW, N / 2 + 1)];
      uint32_t bytes = 0;
#pragma unroll
      for (int i = 0; i < N / BR; ++i)
        if (BR * i <= m || BR * i + BR - 1 >= N - m) bytes += 128u * BR;
      mbar_arrive_expect_tx(&bars[ib], bytes);
#pragma unroll
      for (int i = 0; i < N / BR; ++i)
        if (BR * i <= m || BR * i + BR - 1 >= N - m)
          tma_load_4d(dst + i * BR * TW, &map, &bars[ib], cb * 2 * TW, i * BR, c, f);
    } else {
      mbar_arrive_expect_tx(&bars[ib], 128u * N);
#pragma unroll
      for (int i = 0; i < N / BR; ++i) {
        if constexpr (AXIS == 1) tma_load_4d(dst + i * BR * TW, &map, &bars[ib], cb * 2 * TW, i * BR, c, f);
        else tma_load_4d(dst + i * BR * TW, &map, &bars[ib], cb * 2 * TW, c, i * BR, f);
      }
    }
    ib = ib + 1 == SLOTS ? 0 : ib + 1;
    it += gridDim.x;
  };
  if (tid == 0)
    for (int b = 0; b < SLOTS; ++b) issue();
  __syncthreads();  // (s_tile)

  // distance between the thread's consecutive outputs (16 elements of the axis)
  const long long step = 16LL * g.pitch * (AXIS == 1 ? 1 : N);
  const RT sc = (RT)a.scale;
  bool fail = false;
  int b = 0;
  uint32_t parity = 0;
#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int3 tl = s_tile[b];
    const int c = tl.y, f = tl.z, mx = tl.x * TW + s;
    // every thread polls; the next barrier tells all of them whether any wait ran out
    const bool late = !mbar_wait_bounded(&bars[b], parity);
    C* const S = ring + b * TILE;
    C v[16];
    if constexpr (VARIANT == 1) {
      static_assert(AXIS == 2 || VARIANT == 0, "the phase variant is the inverse z pass");
      // shifted grid: phase exp(i pi (mx + my + mz) / N); modes with 0 < mx < N/2 and index N/2
      // in exactly one of y, z are anti-Hermitian in the reference and drop out; columns past
      // N/2 are padding
      C w[16];
      const int base = mx + signed_mode(c, N) + 3 * N / 2;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int e = n2 + R2 * r;
        v[r] = cscale(S[SNS_IDX(e * TW + s, TILE)], sc);
        const bool anti = mx > 0 && mx < N / 2 && ((c == N / 2) != (e == N / 2));
        w[r] = mx > N / 2 || anti ? czero<C>()
                                  : cmul(v[r], __ldg(&phase[SNS_IDX(base + signed_mode(e, N), 3 * N + 1)]));
      }
      pass1<N, DIR, Y>(v, S, s_tw, s, n2);
      pass1<N, DIR, Y>(w, W, s_tw, s, n2);
    } else {
      if constexpr (PARTS) {
        // row e = n2 + R2 r, |my| = e below N/2, N - e above
        const int m = s_disk[SNS_IDX(mx, N / 2 + 1)], lo = m - n2, hi = m + n2 - N;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const C x = S[SNS_IDX((n2 + R2 * r) * TW + s, TILE)];
          v[r] = (r < 8 ? lo >= R2 * r : hi >= -R2 * r) ? x : czero<C>();
        }
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = S[SNS_IDX((n2 + R2 * r) * TW + s, TILE)];
        if constexpr (AXIS == 2) {
#pragma unroll
          for (int r = 0; r < 16; ++r) v[r] = cscale(v[r], sc);
        }
      }
      pass1<N, DIR, Y>(v, S, s_tw, s, n2);
    }
    if (__syncthreads_or(late)) {
      fail = true;
      break;
    }
    const int e0 = k1 + 256 * h;
    const long long at = (AXIS == 1 ? (long long)c * N + e0 : (long long)e0 * N + c) * g.pitch + mx;
    C* out = static_cast<C*>(a.out) + (long long)(a.f_out0 + (VARIANT ? 2 : 1) * f) * g.field;
    pass2_load<Y>(S, s, k1, h, v);
    [[maybe_unused]] C w[VARIANT ? 16 : 1];
    if constexpr (VARIANT == 1 && Y::EARLY) pass2_load<Y>(W, s, k1, h, w);
    fence_proxy_async_smem();
    auto release = [&] {
      __syncthreads();
      if (tid == 0) issue();
      if (++b == SLOTS) {
        b = 0;
        parity ^= 1u;
      }
    };
    // the slot (and the work buffer) is in registers: refill it while the butterflies run and the
    // outputs are stored, which then overlap the next tile's first pass
    if constexpr (Y::EARLY) release();
    pass2<DIR, Y>(h, v);
#pragma unroll
    for (int q = 0; q < 16; ++q) out[SNS_IDX(at + q * step, g.field)] = v[q];
    if constexpr (VARIANT == 1) {
      if constexpr (!Y::EARLY) pass2_load<Y>(W, s, k1, h, w);
      pass2<DIR, Y>(h, w);
      out += g.field;
#pragma unroll
      for (int q = 0; q < 16; ++q) out[SNS_IDX(at + q * step, g.field)] = w[q];
    }
    if constexpr (!Y::EARLY) release();
  }
  if (fail) {
    if (tid == 0) {
      atomicExch(a.err, kErrTmaTimeout);
      // let every copy in flight land (bounded) before the CTA gives up its shared memory
      for (int i = 0; i < SLOTS; ++i) {
        (void)mbar_wait_bounded(&bars[i], 0u);
        (void)mbar_wait_bounded(&bars[i], 1u);
      }
    }
    __syncthreads();
  }
}

template <int N, class C>
struct LaunchStream {
  template <int AXIS, int DIR, int VARIANT, bool PARTS>
  static void prepare() {
    cudaFuncSetAttribute(k_stream<N, AXIS, DIR, VARIANT, PARTS, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)YZ<N, C, VARIANT>::smem);
    cudaFuncSetAttribute(k_stream<N, AXIS, DIR, VARIANT, PARTS, C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
  }
  static void init() {
    prepare<2, +1, 1, false>();
    prepare<1, +1, 0, true>();
    prepare<1, +1, 0, false>();
    prepare<2, +1, 0, false>();
    prepare<2, -1, 0, false>();
  }
  static int blocks_per_sm() {
    int nb = 0, lo = 1 << 30;
    auto occ = [&](auto k, int nt, size_t smem) {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, nt, smem) == cudaSuccess && nb < lo) lo = nb;
    };
    using Y0 = YZ<N, C, 0>;
    occ(k_stream<N, 2, +1, 1, false, C>, YZ<N, C, 1>::NT, YZ<N, C, 1>::smem);
    occ(k_stream<N, 1, +1, 0, true, C>, Y0::NT, Y0::smem);
    occ(k_stream<N, 1, +1, 0, false, C>, Y0::NT, Y0::smem);
    occ(k_stream<N, 2, +1, 0, false, C>, Y0::NT, Y0::smem);
    occ(k_stream<N, 2, -1, 0, false, C>, Y0::NT, Y0::smem);
    return lo > 0 && lo < (1 << 30) ? lo : 1;
  }
  template <int AXIS, int DIR, int VARIANT, bool PARTS>
  static void go(const CUtensorMap& map, TmaArgs a, const void* tw, const void* phase, Geom g, int grid,
                 cudaStream_t st) {
    using Y = YZ<N, C, VARIANT>;
    k_stream<N, AXIS, DIR, VARIANT, PARTS, C><<<grid, Y::NT, Y::smem, st>>>(map, a, static_cast<const C*>(tw),
                                                                            static_cast<const C*>(phase), g);
  }
  static void run(const CUtensorMap& map, int axis, int dir, int variant, int part, TmaArgs a, const void* tw,
                  const void* phase, Geom g, int grid, cudaStream_t st) {
    if (variant == 1) go<2, +1, 1, false>(map, a, tw, phase, g, grid, st);
    else if (axis == 1 && part) go<1, +1, 0, true>(map, a, tw, phase, g, grid, st);
    else if (axis == 1) go<1, +1, 0, false>(map, a, tw, phase, g, grid, st);
    else if (dir < 0) go<2, -1, 0, false>(map, a, tw, phase, g, grid, st);
    else go<2, +1, 0, false>(map, a, tw, phase, g, grid, st);
  }
  static const StreamOps* table() {
    static const StreamOps ops = {init, blocks_per_sm, run, YZ<N, C, 0>::PART};
    return &ops;
  }
};

}  // namespace

const StreamOps* stream_for(int n, int precision) {
  if (n == 256) return precision == 0 ? LaunchStream<256, double2>::table() : LaunchStream<256, float2>::table();
  if (n == 512) return precision == 0 ? LaunchStream<512, double2>::table() : LaunchStream<512, float2>::table();
  return nullptr;
}

int bounds_record_stream(long long* out3) {
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
