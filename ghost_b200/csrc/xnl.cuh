// xnl.cuh -- the fused X pass of a substep, lines kept inside a warp.
//
// Complex-to-real x lines of every input field, the real-space products in
// registers, real-to-complex lines of the products (prodre3,
// pseudospec3D_hd.f90:316-396; advect3, pseudospec3D_phd.f90:23-114):
//   PHYS 0 (HD):    in v, curl v (6)              -> out omega x v (3)
//   PHYS 1 (BOUSS): in v, curl v, grad theta (9)  -> out omega x v (3), -v.grad(theta) (1)
//
// A tile is BZ z-values x the live kx rows of one y, one TMA box sequence per
// field into a STAGES-deep ring (swizzled: 128-byte rows with SWIZZLE_128B,
// 64-byte rows with SWIZZLE_64B).  A line of M = NX/2 complex values is held
// by T = M/E lanes of one warp, E values each, so that a transform's
// exchanges go through a buffer of the warp's own and need __syncwarp only.
// With E = 16 a 256-point transform is 16 x 16: one exchange.
//
// What bounds it: shared-memory wavefronts and issue slots, about equally.
// So per line it (a) reads the tile once for X_k and once for X_{M-k}, only
// the rows that exist (LE of the E row groups: the 2/3 truncation leaves 11
// of 16), (b) takes one exchange where radix 8 took two, (c) fetches the
// mirror Z_{M-k} of the real-to-complex unpacking by shuffles, (d) adds in
// packed FP32, and (e) sends the results out by TMA from a staging tile; the
// CTA meets at three or four barriers a tile. ms a launch, by lines of a CTA with
// radix-8 (FP64: radix-4) stages and by this kernel: 512^3 FP32 1.48 and 1.22,
// 1024 x 1024 x 256 Boussinesq FP32 6.60 and 4.95, 256^3 FP64 0.515 and 0.430.
// Small grids stay with the lines of a CTA (xnl_takes, xnl.cu).
#pragma once
#include "f32x2.cuh"
#include "passes.cuh"

namespace gb {

// ------------------------------------------------------------ transforms
// In-register DFTs on packed complex numbers, y_r = sum_m x_m exp(S 2 pi i m r / R).
template <int S, typename C> __device__ __forceinline__ void pdft4(C &x0, C &x1, C &x2, C &x3) {
  const C a0 = add2(x0, x2), a1 = sub2(x0, x2), b0 = add2(x1, x3), d = sub2(x1, x3);
  x0 = add2(a0, b0);
  x2 = sub2(a0, b0);
  if (S > 0) {
    x1 = mk(a1.x - d.y, a1.y + d.x);
    x3 = mk(a1.x + d.y, a1.y - d.x);
  } else {
    x1 = mk(a1.x + d.y, a1.y - d.x);
    x3 = mk(a1.x - d.y, a1.y + d.x);
  }
}
// a * (c + S i s), constants
template <int S, typename C> __device__ __forceinline__ C cmulk(C a, double c0, double s0) {
  typedef decltype(C{}.x) R;
  const R c = (R)c0, t = (R)(S > 0 ? s0 : -s0);
  return mk(a.x * c - a.y * t, a.y * c + a.x * t);
}
// a * exp(S 2 pi i / 8) and a * exp(S 2 pi i 3/8)
template <int S, typename C> __device__ __forceinline__ C mulw8(C a) {
  const auto h = rsqrt2_of<C>::v();
  return S > 0 ? mul2(mk(a.x - a.y, a.y + a.x), both(h)) : mul2(mk(a.x + a.y, a.y - a.x), both(h));
}
template <int S, typename C> __device__ __forceinline__ C mulw83(C a) {
  const auto h = rsqrt2_of<C>::v();
  return S > 0 ? mul2(mk(-a.x - a.y, a.x - a.y), both(h)) : mul2(mk(a.y - a.x, -a.x - a.y), both(h));
}
template <int S, typename C> __device__ __forceinline__ void pdft8(C (&v)[8]) {
  C u0 = add2(v[0], v[4]), d0 = sub2(v[0], v[4]), u1 = add2(v[1], v[5]), d1 = sub2(v[1], v[5]);
  C u2 = add2(v[2], v[6]), d2 = sub2(v[2], v[6]), u3 = add2(v[3], v[7]), d3 = sub2(v[3], v[7]);
  C e1 = mulw8<S>(d1), e2 = mul_si<S>(d2), e3 = mulw83<S>(d3);
  pdft4<S>(u0, u1, u2, u3);
  pdft4<S>(d0, e1, e2, e3);
  v[0] = u0; v[2] = u1; v[4] = u2; v[6] = u3;
  v[1] = d0; v[3] = e1; v[5] = e2; v[7] = e3;
}
template <int S, typename C> __device__ __forceinline__ void pdft16(C (&x)[16]) {
  // cos and sin of 2 pi/16
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
#pragma unroll
  for (int m = 0; m < 4; ++m) pdft4<S>(x[m], x[m + 4], x[m + 8], x[m + 12]);
  // x[m + 4 r] is output r of column m: times W16^(m r)
  x[5] = cmulk<S>(x[5], c1, s1);
  x[9] = mulw8<S>(x[9]);
  x[13] = cmulk<S>(x[13], s1, c1);
  x[6] = mulw8<S>(x[6]);
  x[10] = mul_si<S>(x[10]);
  x[14] = mulw83<S>(x[14]);
  x[7] = cmulk<S>(x[7], s1, c1);
  x[11] = mulw83<S>(x[11]);
  x[15] = cmulk<S>(x[15], -c1, -s1);  // W16^9
#pragma unroll
  for (int r = 0; r < 4; ++r) pdft4<S>(x[4 * r], x[4 * r + 1], x[4 * r + 2], x[4 * r + 3]);
  // x[4 r + q] is now output r + 4 q
  C y[16];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) y[r + 4 * q] = x[4 * r + q];
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = y[q];
}

template <typename R, int NX, int E, int BZ, int LE> struct XnlGeom {
  static constexpr int ES = 2 * sizeof(R);  // bytes of a complex value
  static constexpr int M = NX / 2, T = M / E, LW = 32 / T, NW = BZ / LW, NT = 32 * NW;
  static constexpr int RB = BZ * ES;  // bytes of a tile row
  static constexpr int ROWS = ((LE == E ? M + 1 : LE * T + 1) + 7) / 8 * 8;  // rows of a tile buffer
  static constexpr size_t tile = (size_t)ROWS * RB;
  static constexpr int PAD = E == 16 && M <= 256 ? 16 : 8;  // exchange slots: idx + idx/PAD
  static constexpr int XL = M + M / PAD;                    // slots of a line
  static constexpr size_t xch = (size_t)XL * ES * LW;
  // twiddles between stages.  E = 16: pairs of powers (2j, 2j+1) side by side
  // (M = 256: 16 powers x 16 lanes; 128: 8 x 16; 512: 8 x 8 and 8 x 64).
  // E = 8: per stage of span L > 1 and radix Q, powers 1..Q-1 x L.
  static constexpr int tw8(int L) {
    int n = 0;
    for (; L < M; L *= 8) n += (M / L < 8 ? M / L - 1 : 7) * L;
    return n;
  }
  static constexpr int TW2 = E == 8 ? tw8(8) : (M == 256 ? 256 : (M == 128 ? 128 : 64)), TW3 = E == 16 && M == 512 ? 512 : 0;
  static constexpr size_t fixed = 2 * tile + NW * xch + (size_t)(M + TW2 + TW3) * ES + 1024 + 256;
  static constexpr int stages(size_t cap) {
    return fixed + 5 * tile <= cap ? 5 : (fixed + 4 * tile <= cap ? 4 : (fixed + 3 * tile <= cap ? 3 : 2));
  }
  static_assert(T >= 4 && T <= 32 && BZ % LW == 0 && (NW & (NW - 1)) == 0, "a line is 4 to 32 lanes of a warp");
};

// E = 8: radix 8 stages and a last one of radix 2 or 4, from span L on.
// tw: powers 1..Q-1 of the stage's twiddles, L of each; xb: the line's
// exchange buffer (slot idx at xb[(idx + idx/8) STR]).
template <int M, int S, int STR, int L, typename C>
__device__ __forceinline__ void xnl_fft8(C (&x)[8], int t, C *xb, const C *tw) {
  constexpr int T = M / 8, Q = M / L < 8 ? M / L : 8, NB = 8 / Q;
  constexpr bool LAST = L * Q == M;
  C y[8];
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
        xb[(idx + idx / 8) * STR] = v[r];
      }
    }
  }
  if constexpr (LAST) {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = y[e];
  } else {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int idx = t + T * e;
      x[e] = xb[(idx + idx / 8) * STR];
    }
    __syncwarp();
    xnl_fft8<M, S, STR, L * Q>(x, t, xb, tw + (L > 1 ? (Q - 1) * L : 0));
  }
}

// E = 16 (FP32): 16 x 16, 16 x 8 or 8 x 8 x 8.  xb: the line's exchange
// buffer (M + M/PAD slots); t2, t3: this lane's twiddle
// pairs (see XnlGeom).
template <int M, int S, int STR>
__device__ __forceinline__ void xnl_fft16(float2 (&x)[16], int t, float2 *xb, const float4 *t2, const float4 *t3) {
  constexpr int T = M / 16;
  auto tw = [](float2 &v, float2 w) { v = twmul<S>(v, w); };
  if constexpr (M == 256) {
    pdft16<S>(x);
    float2 *w = xb + (size_t)(17 * t) * STR;
#pragma unroll
    for (int r = 0; r < 16; ++r) w[r * STR] = x[r];
    __syncwarp();
    const float2 *q = xb + (size_t)t * STR;
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = q[17 * e * STR];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 p = t2[16 * j];
      if (j > 0) tw(x[2 * j], mk(p.x, p.y));
      tw(x[2 * j + 1], mk(p.z, p.w));
    }
    pdft16<S>(x);
    __syncwarp();
  } else if constexpr (M == 128) {
    pdft16<S>(x);
    float2 *w = xb + (size_t)(17 * t) * STR;
#pragma unroll
    for (int r = 0; r < 16; ++r) w[r * STR] = x[r];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = xb[(size_t)(t + 8 * e + e / 2) * STR];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      float2 v[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) v[m] = x[b + 2 * m];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 p = t2[16 * j + 8 * b];
        if (j > 0) tw(v[2 * j], mk(p.x, p.y));
        tw(v[2 * j + 1], mk(p.z, p.w));
      }
      pdft8<S>(v);
#pragma unroll
      for (int r = 0; r < 8; ++r) x[b + 2 * r] = v[r];
    }
    __syncwarp();
  } else {
    static_assert(M == 512, "line length");
    // 8 x 8 x 8, two butterflies per lane and stage: b = t, t + 32.  The 16
    // lanes of a shared-memory phase use 16 banks: the first stage writes
    // idx = 8 b + r to slot idx + idx/16, the second 64 (b/8) + b%8 + 8 r to
    // idx + 8 (idx/64), and both are read contiguously.  (With idx + idx/8 for
    // both the reads took twice the phases: 22.2 -> 19.8 ms a step of 1024 x 1024 x 256
    // Boussinesq.)
    auto slot = [&](int st, int idx) -> float2 & { return xb[(st == 0 ? idx + idx / 16 : idx + idx / 64 * 8) * STR]; };
#pragma unroll
    for (int st = 0; st < 3; ++st) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        float2 v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = x[b + 2 * m];
        if (st > 0) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 p = st == 1 ? t2[8 * j] : t3[64 * j + 32 * b];
            if (j > 0) tw(v[2 * j], mk(p.x, p.y));
            tw(v[2 * j + 1], mk(p.z, p.w));
          }
        }
        pdft8<S>(v);
        if (st == 2) {
#pragma unroll
          for (int r = 0; r < 8; ++r) x[b + 2 * r] = v[r];
        } else {
          const int bb = t + 32 * b;
          const int base = st == 0 ? 8 * bb : 64 * (bb / 8) + (bb & 7);
#pragma unroll
          for (int r = 0; r < 8; ++r) slot(st, base + (st == 0 ? r : 8 * r)) = v[r];
        }
      }
      if (st < 2) {
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = slot(st, t + T * e);
        __syncwarp();
      }
    }
  }
}

// ---------------------------------------------------------------- kernel
// The rows of a field a tile moves, [0, rows), as nbox boxes of rb rows; box q
// starts at row min(8 floor(rb/8) q, rows - rb), always a multiple of 8 (the
// swizzle pattern's period), so boxes may overlap but never leave the rows.
struct XnlBoxes {
  int nbox, rb;
  explicit XnlBoxes(int rows) : nbox((rows + 255) / 256) {
    for (;; ++nbox) {
      rb = (rows + nbox - 1) / nbox;
      rb += ((rows - rb) % 8 + 8) % 8;
      if (rb <= 256 && (nbox - 1) * (rb & ~7) + rb >= rows) return;
    }
  }
};

__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
// c2r_pack of two values, with every rounding spelt out: a line whose known
// zeros the compiler sees must come out bit for bit as one that loads them.
template <typename C> __device__ __forceinline__ C xnl_pack(C xk, C xm, C w) {
  const C a = addc2(xk, xm), b = subc2(xk, xm);
  // i b e^{+2 pi i k/NX}
  const C u = mk(rfma(-b.y, w.x, rmul(b.x, w.y)), rfma(b.x, w.x, rmul(b.y, w.y)));
  return add2(a, u);
}
// twice r2c_unpack
template <typename C> __device__ __forceinline__ C xnl_unpack2(C zk, C zm, C w) {
  const C s = addc2(zk, zm), d = subc2(zk, zm);
  const C u = mk(rfma(d.y, w.x, rmul(d.x, w.y)), rfma(d.y, w.y, rmul(-d.x, w.x)));  // w (d.y, -d.x)
  return add2(s, u);
}

// One lane's part of the lines of a tile: where it sits, its transforms and
// their tables (shared by the group).
template <typename R, int NX, int E, int BZ> struct XLine {
  using C = cx<R>;
  using G = XnlGeom<R, NX, E, BZ, E>;
  static constexpr int M = G::M, T = G::T, LW = G::LW, RB = G::RB, NT = G::NT;
  static constexpr bool F32 = sizeof(R) == 4;
  static constexpr int STR = F32 && LW > 1 ? 2 : 1;  // FP32: two lines share an exchange buffer's 16-byte slots
  static constexpr uint32_t ESTEP = (uint32_t)T * RB;
  int t, z, mlane;  // place in the line, line of the tile, the lane that holds M - k
  C *xb, *twp, *tw2, *tw3;
  uint32_t off_k[2], off_m[2];

  // byte offset of (k, z) in a swizzled tile.  k = t + T e and M - k keep
  // their swizzle over e where T is a multiple of 8; with T = 4 it alternates.
  static __device__ __forceinline__ uint32_t toff(int k, int zz) {
    if constexpr (!F32) return (uint32_t)k * 128 + ((uint32_t)(zz ^ (k & 7)) << 4);
    else
      return RB == 128 ? (uint32_t)k * 128 + ((uint32_t)((zz >> 1) ^ (k & 7)) << 4) + (uint32_t)(zz & 1) * 8
                       : (uint32_t)k * 64 + ((uint32_t)((zz >> 1) ^ ((k >> 1) & 3)) << 4) + (uint32_t)(zz & 1) * 8;
  }
  // xall: the group's exchange buffers, then its tables (M + TW2 + TW3 values);
  // a barrier of the group must follow before the first transform
  __device__ __forceinline__ XLine(int tid, C *xall, const C *__restrict__ twg) {
    const int lane = tid & 31, wp = tid >> 5;
    // The lanes of one shared-memory phase (16 of 8 bytes, 8 of 16) touch
    // different banks of the swizzled rows: 8 consecutive t, or 4 t of lines
    // whose 16-byte chunks differ in bit 2; in FP32 of both lines of a chunk.
    int zi;
    if constexpr (F32) {
      t = T == 32 ? lane : (lane >> 1) & (T - 1);
      zi = T == 32 ? 0 : (T == 16 ? lane & 1 : (T == 8 ? (lane & 1) + 2 * (lane >> 4) : (lane & 1) + 2 * (lane >> 3)));
      z = T == 4 ? (lane & 1) + 8 * ((lane >> 3) & 1) + 2 * (lane >> 4) + 4 * wp : wp * LW + zi;
    } else {
      t = lane & (T - 1);
      zi = lane / T;
      z = T == 4 ? 4 * (zi & 1) + (zi >> 1) : wp * LW + zi;
    }
    const int mt = (T - t) & (T - 1);
    mlane = F32 && T < 32 ? (lane & ~(2 * (T - 1))) | (2 * mt) : (lane & ~(T - 1)) | mt;
    xb = reinterpret_cast<C *>(reinterpret_cast<unsigned char *>(xall) + (size_t)wp * G::xch) +
         (STR == 2 ? (size_t)(zi >> 1) * G::XL * 2 + (zi & 1) : (size_t)zi * G::XL);
    // exp(-2 pi i k/NX), k = t + T e: E = 16 in pairs (e, e+1), else one by one
    twp = reinterpret_cast<C *>(reinterpret_cast<unsigned char *>(xall) + G::NW * G::xch);
    tw2 = twp + M;
    tw3 = tw2 + G::TW2;
    off_k[0] = toff(t, z);
    off_k[1] = T == 4 ? toff(t + T, z) - ESTEP : off_k[0];
    off_m[0] = toff(M - t, z);
    off_m[1] = T == 4 ? toff(M - t - T, z) + ESTEP : off_m[0];
    if constexpr (E == 16) {
      for (int q = tid; q < M; q += NT) {  // twp[((e/2) T + t) 2 + (e & 1)]
        const int e = 2 * (q / (2 * T)) + (q & 1), tt = (q >> 1) % T;
        twp[q] = twg[tt + T * e];
      }
      // tw2[(j W + b) 2 + p] = W_M^(b (2j + p) M/(L Q)) for the second stage's b < W
      constexpr int W = M == 512 ? 8 : 16, SC = M == 512 ? 8 : 1;
      for (int q = tid; q < G::TW2; q += NT) {
        const int m = 2 * (q / (2 * W)) + (q & 1), b = (q >> 1) % W;
        tw2[q] = twg[(2 * SC * b * m) % NX];
      }
      for (int q = tid; q < G::TW3; q += NT) {
        const int m = 2 * (q / 128) + (q & 1), b = (q >> 1) % 64;
        tw3[q] = twg[(2 * b * m) % NX];
      }
    } else {
      for (int q = tid; q < M; q += NT) twp[q] = twg[q];
      int o = 0;
#pragma unroll
      for (int L = 8; L < M; L *= 8) {
        const int Q = M / L < 8 ? M / L : 8;
        for (int q = tid; q < (Q - 1) * L; q += NT) tw2[o + q] = twg[2 * (q % L) * (q / L + 1) * (M / (L * Q))];
        o += (Q - 1) * L;
      }
    }
  }
  template <int S> __device__ __forceinline__ void fft(C (&x)[E]) const {
    if constexpr (E == 16)
      xnl_fft16<M, S, STR>(x, t, xb, reinterpret_cast<const float4 *>(tw2) + (M == 512 ? (t & 7) : t),
                           reinterpret_cast<const float4 *>(tw3) + t);
    else
      xnl_fft8<M, S, STR, 1>(x, t, xb, tw2);
  }
  // exp(-2 pi i k/NX) of k = t + T e, for two e at a time
  __device__ __forceinline__ void pack_tw(int e, C (&w)[2]) const {
    if constexpr (E == 16) {
      const float4 q = reinterpret_cast<const float4 *>(twp)[T * (e / 2) + t];
      w[0] = mk(q.x, q.y);
      w[1] = mk(q.z, q.w);
    } else {
      w[0] = twp[t + T * e];
      w[1] = twp[t + T * (e + 1)];
    }
  }
  // the line's packed half spectrum from a swizzled tile with LE row groups
  template <int LE> __device__ __forceinline__ void load_packed(C (&x)[E], const unsigned char *tb) const {
#pragma unroll
    for (int e0 = 0; e0 < E; e0 += 2) {
      C w[2];
      pack_tw(e0, w);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int e = e0 + p;
        C xk = e < LE ? *reinterpret_cast<const C *>(tb + off_k[e & 1] + e * ESTEP) : mk((R)0, (R)0);
        C xm = LE == E || e >= E - LE ? *reinterpret_cast<const C *>(tb + off_m[e & 1] - e * ESTEP) : mk((R)0, (R)0);
        if (e == 0 && t == 0) {
          xk.y = (R)0;
          xm.y = (R)0;
        }
        x[e] = xnl_pack(xk, xm, w[p]);
      }
    }
  }
  // twice the transformed line's half spectrum into a swizzled tile with LE row groups
  template <int LE> __device__ __forceinline__ void store_unpacked(const C (&P)[E], unsigned char *ob) const {
#pragma unroll
    for (int e0 = 0; e0 < LE; e0 += 2) {
      C w[2];
      pack_tw(e0, w);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int e = e0 + p;
        if (e < LE) {
          const C src = t == 0 ? P[(E - e) % E] : P[E - 1 - e];
          const C zm = mk(__shfl_sync(0xffffffffu, src.x, mlane), __shfl_sync(0xffffffffu, src.y, mlane));
          *reinterpret_cast<C *>(ob + off_k[e & 1] + e * ESTEP) = xnl_unpack2(P[e], zm, w[p]);
          if (LE == E && e == 0 && t == 0) *reinterpret_cast<C *>(ob + toff(M, z)) = xnl_unpack2(P[0], zm, mk((R)-1, (R)0));
        }
      }
    }
  }
};

// A pass's share of one group of NT threads (warps NW g .. NW g + NW - 1 of
// the CTA, shared memory from sm on): tiles vb, vb + nvb, ...  omaps: tensor
// maps of the output fields (the same boxes).
template <typename R, int NX, int E, int BZ, int PHYS, int LE, int STAGES>
__device__ __forceinline__ void xnl_body(int vb, int nvb, int g, unsigned char *sm, const FieldMaps &maps,
                                         const FieldMaps &omaps, const cx<R> *__restrict__ twg, int ny, int nz, R scale,
                                         int rows, int nbox, int rb, int nruns, int nxh, PipeCtl ctl) {
  using C = cx<R>;
  using G = XnlGeom<R, NX, E, BZ, LE>;
  constexpr int NW = G::NW, NT = G::NT, RB = G::RB;
  constexpr int NIN = PHYS == 0 ? 6 : 9;
  unsigned char *obuf = sm + STAGES * G::tile;
  C *xall = reinterpret_cast<C *>(obuf + 2 * G::tile);
  const int tid = threadIdx.x - g * NT, lane = tid & 31;
  const XLine<R, NX, E, BZ> ln(tid, xall, twg);
  uint64_t *full = reinterpret_cast<uint64_t *>(ln.tw3 + G::TW3), *never = full + STAGES;
  unsigned *cnt = reinterpret_cast<unsigned *>(never + 1);
  volatile int *failed = reinterpret_cast<int *>(cnt + STAGES);  // ring_wait
  auto group_sync = [g] {
    if (NT == 32) __syncwarp();
    else named_sync(1 + g, NT);
  };
  const int nzb = nz / BZ, ntiles = nzb * ny * nruns;
  dep_go();
  if (tid == 0) {
    mbar_init(never, 1);
    for (int q = 0; q < STAGES; ++q) {
      mbar_init(&full[q], 1);
      cnt[q] = 0;
    }
    *failed = 0;
    fence_barrier_init();
  }
  // rows beyond the live ones are zero and stay so: no load reaches them
  for (int s = 0; s < STAGES; ++s)
    for (int q = tid; q < (G::ROWS - rows) * (RB / 16); q += NT)
      reinterpret_cast<uint4 *>(sm + s * G::tile + (size_t)rows * RB)[q] = make_uint4(0, 0, 0, 0);
  group_sync();
  // input order: v, then (BOUSS) grad theta, then curl v
  auto field_of = [](int f) { return PHYS == 0 || f < 3 ? f : (f < 6 ? f + 3 : f - 3); };
  // box q of a field: rows min(8 floor(rb/8) q, rows - rb) onwards, always a multiple of 8
  const int bstep = rb & ~7;
  constexpr int U = G::ES / 8;
  auto issue = [&](int L) {
    const int k = L / NIN, f = L - k * NIN;
    const int tile = vb + k * nvb;
    if (tile >= ntiles) return;
    const int s = L % STAGES;
    fence_proxy_async();
    mbar_arrive_expect_tx(&full[s], (uint32_t)(nbox * rb) * RB);
    for (int q = 0; q < nbox; ++q) {
      const int r0 = min(q * bstep, rows - rb);
      tma_load_3d(sm + s * G::tile + (size_t)r0 * RB, &maps.m[field_of(f)], (tile % nzb) * BZ * U, (tile / nzb) % ny,
                  (tile / nzb / ny) * nxh + r0, &full[s]);
    }
  };
  dep_wait();
  if (tid == 0)
    for (int L = 0; L < STAGES; ++L) issue(L);
  int nout = 0;
  bool alive = true;  // no wait of this thread has run out
  // forward line of a product and its way out as output field c, unless a wait
  // of the group has run out
  auto emit = [&](C(&P)[E], int tile, int c) {
    ln.template fft<-1>(P);
    unsigned char *ob = obuf + (size_t)(nout & 1) * G::tile;
    ln.template store_unpacked<LE>(P, ob);
    fence_proxy_async();                  // the tile's generic writes, before the store reads them
    if (tid == 0) bulk_wait_read_all();   // the store before this one has read its buffer
    group_sync();
    if (tid == 0 && !*failed) {
      for (int q = 0; q < nbox; ++q) {
        const int r0 = min(q * bstep, rows - rb);
        tma_store_3d(&omaps.m[c], ob + (size_t)r0 * RB, (tile % nzb) * BZ * U, (tile / nzb) % ny,
                     (tile / nzb / ny) * nxh + r0);
      }
      bulk_commit();
    }
    ++nout;
  };
  for (int k = 0;; ++k) {
    const int tile = vb + k * nvb;
    if (tile >= ntiles) break;
    // inverse line of load f of the tile: x[e] = (r_{2m}, r_{2m+1}) at m = t + T e
    auto inverse = [&](int f, C(&x)[E]) {
      const int L = k * NIN + f, s = L % STAGES;
      // after a wait that ran out the line is computed from whatever the slot
      // holds and goes nowhere
      alive = alive && ring_wait(&full[s], (uint32_t)(L / STAGES) & 1u, never, ctl.stall && L == 0, ctl, failed);
      ln.template load_packed<LE>(x, sm + s * G::tile);
      // the last warp to read a slot refills it
      __syncwarp();
      if (lane == 0 && alive && ring_read<STAGES, NW>(cnt, L)) issue(L + STAGES);
      ln.template fft<+1>(x);
    };
    // Loops where the live registers allow it: nine unrolled lines were 90 KB
    // of code, and the warps waited for instructions half as long as they
    // issued them.  The three curl components stay unrolled, as not all of V
    // and P is live in any one of them.
    C V[3][E], P[3][E];
    const R half = scale * (R)0.5;  // store_unpacked gives twice the spectrum
    const C sc = both(half);
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
      C x[E];
      inverse(f, x);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (f == 0) V[0][e] = x[e];
        else if (f == 1) V[1][e] = x[e];
        else V[2][e] = x[e];
      }
    }
    if constexpr (PHYS == 1) {
      // advect3: vx th_x + vy th_y + vz th_z, times -1/(nx ny nz)^2
      C Q[E];
#pragma unroll 1
      for (int f = 0; f < 3; ++f) {
        C x[E];
        inverse(3 + f, x);
#pragma unroll
        for (int e = 0; e < E; ++e)
          Q[e] = f == 0 ? mul2(V[0][e], x[e]) : (f == 1 ? fma2(V[1][e], x[e], Q[e]) : mul2(fma2(V[2][e], x[e], Q[e]), both(-half)));
      }
      emit(Q, tile, 3);
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      C x[E];
      inverse(NIN - 3 + f, x);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (f == 0) {  // wx: (w x v)_y = wz vx - vz wx ; (w x v)_z = wx vy - vx wy
          P[1][e] = mul2(V[2][e], x[e]);
          P[2][e] = mul2(x[e], V[1][e]);
        } else if (f == 1) {  // wy: (w x v)_x = wy vz - vy wz
          P[0][e] = mul2(x[e], V[2][e]);
          P[2][e] = mul2(fnma2(V[0][e], x[e], P[2][e]), sc);
        } else {  // wz
          P[0][e] = mul2(fnma2(V[1][e], x[e], P[0][e]), sc);
          P[1][e] = mul2(fnma2(V[0][e], x[e], P[1][e]), both(-half));
        }
      }
    }
    // The FP32 pass of six loads is short enough to keep its three emissions
    // unrolled (128^3: 117 -> 111 us a step); with nine loads that was 22.7 -> 27.7 ms
    // at 1024 x 1024 x 256.
    if constexpr (PHYS == 0 && sizeof(R) == 4) {
      emit(P[0], tile, 0);
      emit(P[1], tile, 1);
      emit(P[2], tile, 2);
    } else {
#pragma unroll 1
      for (int c = 0; c < 3; ++c) {
        emit(P[0], tile, c);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          P[0][e] = P[1][e];
          P[1][e] = P[2][e];
        }
      }
    }
  }
  if (tid == 0) {
    if (*failed) ring_drain<STAGES, NW>(full, cnt, [&](int L) { return vb + L / NIN * nvb < ntiles; });
    bulk_wait_all();
  }
}

template <typename R, int NX, int E, int BZ, int PHYS, int LE, int STAGES, int MINB>
__global__ void __launch_bounds__(XnlGeom<R, NX, E, BZ, LE>::NT, MINB)
    xnl_kernel(const __grid_constant__ FieldMaps maps, const __grid_constant__ FieldMaps omaps,
               const cx<R> *__restrict__ twg, int ny, int nz, R scale, int rows, int nbox, int rb, int nruns, int nxh,
               PipeCtl ctl) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *sm = align1024(smem_raw);
  xnl_body<R, NX, E, BZ, PHYS, LE, STAGES>(blockIdx.x, gridDim.x, 0, sm, maps, omaps, twg, ny, nz, scale, rows, nbox, rb,
                                           nruns, nxh, ctl);
}

}  // namespace gb
