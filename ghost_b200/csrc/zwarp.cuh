// zwarp.cuh -- the Z pass with lines kept inside a warp.
//
// The same operations as zpipe_kernel (passes.cuh), but a line of N values is
// held by T = N/E lanes of one warp and a warp works for itself: it fetches
// LW = 32/T lines of every loaded field by bulk copies, transforms them with
// exchanges through a buffer of its own (__syncwarp only), stores the results
// from registers, and has the next lines on their way from the moment the
// operation has read the last of its inputs.  No barrier of the CTA after the
// twiddles.  us a step against CTAs of 128 or 256 threads: 256^3 FP64
// z_inv 940 -> 544; 1024 x 1024 x 256 Boussinesq z_fwd 7588 -> 5937; 128^3 FP32
// closure step z_inv 235 -> 199, z_fwd 115 -> 79, z_c2c 141 -> 100.
#pragma once
#include "f32x2.cuh"
#include "passes.cuh"
#include "xnl.cuh"

namespace gb {

// operations that update fields after their transforms
template <class Op> struct ZUpdate { static constexpr bool value = false; };
template <typename R> struct ZUpdate<ZFwdHD<R>> { static constexpr bool value = true; };
template <typename R> struct ZUpdate<ZFwdBouss<R>> { static constexpr bool value = true; };
template <typename R> struct ZUpdate<ZFwdMhd<R>> { static constexpr bool value = true; };
// The inverse operations, which write twice the fields they read.
template <class Op> struct ZWriter { static constexpr bool value = false; };
template <typename R, int P> struct ZWriter<ZInv<R, P>> { static constexpr bool value = true; };
template <typename R> struct ZWriter<ZGrad<R>> { static constexpr bool value = true; };
// Whether lines of N points are kept inside a warp, with z_warp_E values a lane.
// At 256 points the FP32 inverses stay with zpipe_kernel (us a step of 1024 x
// 1024 x 256: 6370 here, 6230 there; at 512, with 16 values a lane, 2430 and
// 2250), and so do the FP64 updates (256^3: 668 and 630), whose 4 values a lane
// would be two warps a line.  Updates take 4 values a lane: with 8 values of
// every component, and 255 registers, a 128^3 FP64 MHD step's z_fwd took 253
// us, with 4 it takes 106 (64^3 FP32: 58 and 47; 128^3 FP32: 79 and 74).
// FP64 operations of up to three loads take 512 points too, 16 values a lane:
// CTA-wide, 4 values a thread were four exchanges (512^3 z_inv 6180 -> 3380 us a
// step, 256 x 256 x 512 plain transforms 398 -> 202 us a pair).
template <typename R, class Op> constexpr bool z_warp_line(int N) {
  if (sizeof(R) == 4) return N >= 32 && N <= (ZWriter<Op>::value ? 128 : 256);
  return N >= 32 && N <= (ZUpdate<Op>::value ? 128 : (Op::NLOAD <= 3 ? 512 : 256));
}
template <typename R, class Op> constexpr int z_warp_E(int N) {
  return N == 512 ? 16 : (ZUpdate<Op>::value && N <= 128 ? 4 : 8);
}

template <typename R, int N, int E, int NL> struct ZWarpGeom {
  static constexpr int ES = 2 * sizeof(R), T = N / E, LW = 32 / T;
  // a line of the stage starts T values' worth of banks after the one before
  // it, where a shared-memory phase covers several lines
  static constexpr int PITCH = N * ES + (T * ES < 128 ? T * ES : 0);
  static constexpr int RX = E < 8 ? E : 8;  // radix of the stages
  static constexpr int PADL = N + N / RX;   // exchange slots of a line (zw_slot)
  static constexpr size_t warp = (size_t)NL * LW * PITCH + (size_t)LW * PADL * ES;
  static constexpr int tw_count(int L) {
    int n = 0;
    for (; L < N; L *= RX) n += (N / L < RX ? N / L - 1 : RX - 1) * L;
    return n;
  }
  static constexpr int TW = tw_count(RX);
  static constexpr size_t smem(int nw) { return nw * warp + (size_t)TW * ES + 16 * nw + 16; }
  static_assert(T >= 4 && T <= 32 && E >= 4 && E <= 16, "a line is 4 to 32 lanes of a warp");
};

// Exchange slot of value idx after the stage of span L: the lanes of a shared
// memory phase (16 values of FP32, 8 of FP64, from one line or several) write
// and read different banks.  The first stage writes idx = RX b + r, the
// ones after it RX L (b/L) + b%L + L r; all are read contiguously.
template <typename C, int T, int RX, int L> __device__ __forceinline__ constexpr int zw_slot(int idx) {
  constexpr int P = sizeof(C) == 8 && T >= 16 ? 16 : 8;
  return L == 1 ? idx + idx / P : idx + idx / (RX * RX) * RX;
}

// Stages of radix 8 (4 where a lane holds 4 values) and a last one of that or
// less, from span L on; tw: powers 1..Q-1 of the stage's
// twiddles, L of each.
template <int N, int E, int S, int L, typename C>
__device__ __forceinline__ void zw_fft(C (&x)[E], int t, C *xb, const C *tw) {
  constexpr int T = N / E, RX = E < 8 ? E : 8, Q = N / L < RX ? N / L : RX, NB = E / Q;
  constexpr bool LAST = L * Q == N;
  C y[E];
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const int b = t + T * q, k = b & (L - 1);
    C v[Q];
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      v[m] = x[q + NB * m];
      if (L > 1 && m > 0) v[m] = twmul<S>(v[m], tw[(m - 1) * L + k]);
    }
    if constexpr (Q == 8 && sizeof(C) == 8) pdft8<S>(v);
    else dftR<Q, S>(v);
#pragma unroll
    for (int r = 0; r < Q; ++r) {
      if (LAST) y[q + NB * r] = v[r];
      else {
        const int idx = (b / L) * L * Q + k + r * L;
        xb[zw_slot<C, T, RX, L>(idx)] = v[r];
      }
    }
  }
  if constexpr (LAST) {
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = y[e];
  } else {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int idx = t + T * e;
      x[e] = xb[zw_slot<C, T, RX, L>(idx)];
    }
    __syncwarp();
    zw_fft<N, E, S, L * Q>(x, t, xb, tw + (L > 1 ? (Q - 1) * L : 0));
  }
}
template <typename C> struct ZWarpBuf {
  C *xb;
  const C *tw;
  template <int N, int E, int S> __device__ __forceinline__ void fft(C (&x)[E], int t) const {
    zw_fft<N, E, S, 1>(x, t, xb, tw);
  }
};
template <typename C> struct is_warp_line<ZWarpBuf<C>> { static constexpr bool value = true; };

// The lines of warp w of nw (NWC warps in the CTA, this one's place in it wc;
// sm: the CTA's shared memory from a 16-byte boundary on).
template <typename R, int N, int E, int NWC, class Op>
__device__ __forceinline__ void zwarp_body(int w, int nw, int wc, unsigned char *sm, const Op &op,
                                           const cx<R> *__restrict__ twg, const int *__restrict__ lines, int nlines,
                                           PipeCtl ctl) {
  using C = cx<R>;
  constexpr int NL = Op::NLOAD;
  using G = ZWarpGeom<R, N, E, NL>;
  constexpr int T = G::T, LW = G::LW;
  unsigned char *mine = sm + wc * G::warp;
  C *tw = reinterpret_cast<C *>(sm + NWC * G::warp);
  uint64_t *full = reinterpret_cast<uint64_t *>(tw + G::TW) + 2 * wc, *never = full + 1;
  const int lane = threadIdx.x & 31, t = lane & (T - 1), li = lane / T;
  dep_go();
  if (lane == 0) {
    mbar_init(full, 1);
    mbar_init(never, 1);
    fence_barrier_init();
  }
  {
    int o = 0;
#pragma unroll
    for (int L = G::RX; L < N; L *= G::RX) {
      const int Q = N / L < G::RX ? N / L : G::RX;
      for (int q = threadIdx.x; q < (Q - 1) * L; q += 32 * NWC) tw[o + q] = twg[(q % L) * (q / L + 1) * (N / (L * Q))];
      o += (Q - 1) * L;
    }
  }
  __syncthreads();
  dep_wait();
  const int ngroups = (nlines + LW - 1) / LW;
  auto line_of = [&](int g, int l) -> long {
    const long idx = (long)g * LW + l;
    if (idx >= nlines) return -1;
    return lines ? (long)lines[idx] : idx;
  };
  // the whole warp: lane q fetches line q % LW of field q / LW
  auto issue = [&](int g) {
    if (g >= ngroups) return;
    fence_proxy_async();
    if (lane == 0) {
      uint32_t bytes = 0;
      for (int l = 0; l < LW; ++l)
        if (line_of(g, l) >= 0) bytes += NL * N * (uint32_t)sizeof(C);
      mbar_arrive_expect_tx(full, bytes);
    }
    __syncwarp();
    for (int q = lane; q < NL * LW; q += 32) {
      const int f = q / LW, l = q - f * LW;
      const long line = line_of(g, l);
      if (line >= 0) bulk_g2s(mine + (size_t)q * G::PITCH, op.load_src(f) + (size_t)line * N, N * (uint32_t)sizeof(C), full);
    }
  };
  issue(w);
  const unsigned char *in0 = mine + (size_t)li * G::PITCH;
  auto in = [in0](int f) -> const C * { return reinterpret_cast<const C *>(in0 + (size_t)f * LW * G::PITCH); };
  const ZWarpBuf<C> buf{reinterpret_cast<C *>(mine + (size_t)NL * LW * G::PITCH) + (size_t)li * G::PADL, tw};
  uint32_t par = 0;
  for (int g = w; g < ngroups; g += nw) {
    const bool got = (!ctl.stall || g > w || injected_stall_wait(never, ctl.cap)) && mbar_wait(full, par, ctl.cap);
    if (!__all_sync(0xffffffffu, got)) {
      if (lane == 0) record_timeout(ctl.status);
      mbar_wait(full, par, kDrainPolls);
      return;
    }
    par ^= 1u;
    const long line = line_of(g, li);
    op.template body<N, E>(line >= 0 ? line : 0, line >= 0, t, tw, buf, [] { __syncwarp(); }, in, [&] {
      __syncwarp();
      issue(g + nw);
    });
    __syncwarp();
  }
}

template <typename R, int N, int E, int NWC, int MINB, class Op>
__global__ void __launch_bounds__(32 * NWC, MINB) zwarp_kernel(Op op, const cx<R> *__restrict__ twg,
                                                               const int *__restrict__ lines, int nlines, PipeCtl ctl) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int wc = threadIdx.x >> 5;
  zwarp_body<R, N, E, NWC>(blockIdx.x * NWC + wc, gridDim.x * NWC, wc, smem_raw, op, twg, lines, nlines, ctl);
}

}  // namespace gb
