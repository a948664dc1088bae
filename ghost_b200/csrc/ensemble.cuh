// ensemble.cuh -- one launch per pass for every size class of an ensemble.
//
// An ensemble holds batched contexts of different grids (config 3: 128 runs
// of 32^3, 96 of 64^3, 32 of 128^3).  Each pass of the fused substep (Z
// inverse, Y inverse, X, Y forward, Z forward) runs as ONE kernel over all
// classes.  The launch has per CTAs for each of nsm SM slots; class c owns
// the slots [b0[c], b0[c] + nb[c]), and CTA b (slot b % nsm, round b / nsm)
// works for the class owning its slot, as CTA round nb[c] + slot - b0[c] of
// that class's per nb[c] persistent CTAs, with the class's own line length
// (a switch over the supported lengths picks the templated pass body).  The
// hardware fills the SMs slot by slot, round after round, so the CTAs
// resident on one SM tend to run one class's code: the instruction cache
// then holds one pass body per SM instead of several.  Every class runs the same CTA size, NTH threads:
//   Z pass: NTH / (N/E) lines of N points per tile;
//   Y pass: BZ z-lines of NTH / (BZ N/E) consecutive kx per tile;
//   X pass: BZ z-values of NTH / (BZ (N/2)/E) consecutive y per tile;
// so the arithmetic of a line is the one of the class's own launch.
#pragma once
#include "passes.cuh"
#include "xnl.cuh"
#include "ywarp.cuh"
#include "zwarp.cuh"

namespace gb {

constexpr int kEnsMaxCls = 4;   // classes one launch covers
constexpr int kEnsThreads = 128;  // CTA size of every class

template <typename R> constexpr int ens_zE() { return sizeof(R) == 4 ? 8 : 4; }
template <typename R> constexpr int ens_xE() { return sizeof(R) == 4 ? 8 : 4; }
template <typename R> constexpr int ens_xBZ() { return sizeof(R) == 4 ? 8 : 4; }
constexpr int kEnsYBZ = 8;
constexpr int kEnsXStages = 4;  // the X pass's ring: four fields in flight, as the classes' own launches

// the class a CTA works for, its index among that class's CTAs, and their number
struct EnsCta {
  int c, vb, nvb;
};
template <class P> __device__ __forceinline__ EnsCta ens_cta(const P &p) {
  const int slot = (int)blockIdx.x % p.nsm, round = (int)blockIdx.x / p.nsm;
  int c = 0;
  while (c + 1 < p.ncls && slot >= p.b0[c + 1]) ++c;
  return EnsCta{c, round * p.nb[c] + (slot - p.b0[c]), p.per * p.nb[c]};
}

// ------------------------------------------------------------------ Z
template <typename R, class Op> struct ZClass {
  Op op;
  const cx<R> *tw;
  const int *lines;
  int nlines;
  PipeCtl ctl;
};
template <typename R, class Op> struct ZMulti {
  int ncls, nsm, per;
  int n[kEnsMaxCls], b0[kEnsMaxCls], nb[kEnsMaxCls];
  ZClass<R, Op> cl[kEnsMaxCls];
};
template <typename R, int N, int NTH> constexpr int ens_z_lpb() { return NTH / (N / (ens_zE<R>() < N ? ens_zE<R>() : N)); }
template <typename R, int N, class Op> constexpr size_t ens_z_smem(int stages) {
  if constexpr (z_warp_line<R, Op>(N)) return ZWarpGeom<R, N, z_warp_E<R, Op>(N), Op::NLOAD>::smem(kEnsThreads / 32);
  constexpr int E = ens_zE<R>() < N ? ens_zE<R>() : N;
  return ZGeom<R, N, E, ens_z_lpb<R, N, kEnsThreads>(), Op::NLOAD>::smem_bytes(stages);
}

template <typename R, int N, class Op> __device__ __forceinline__ void ens_z_run(const ZClass<R, Op> &k, int vb, int nvb) {
  if constexpr (z_warp_line<R, Op>(N)) {  // as the class's own launches (zwarp.cuh)
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int NWC = kEnsThreads / 32;
    const int wc = (int)threadIdx.x >> 5;
    zwarp_body<R, N, z_warp_E<R, Op>(N), NWC>(vb * NWC + wc, nvb * NWC, wc, smem_raw, k.op, k.tw, k.lines, k.nlines, k.ctl);
  } else {
    constexpr int E = ens_zE<R>() < N ? ens_zE<R>() : N;
    zpipe_body<R, N, E, ens_z_lpb<R, N, kEnsThreads>(), 2>(vb, nvb, k.op, k.tw, k.lines, k.nlines, k.ctl);
  }
}

template <typename R, class Op>
__global__ void __launch_bounds__(kEnsThreads) zmulti_kernel(const __grid_constant__ ZMulti<R, Op> P) {
  const EnsCta k = ens_cta(P);
  switch (P.n[k.c]) {
    case 16: ens_z_run<R, 16>(P.cl[k.c], k.vb, k.nvb); break;
    case 32: ens_z_run<R, 32>(P.cl[k.c], k.vb, k.nvb); break;
    case 64: ens_z_run<R, 64>(P.cl[k.c], k.vb, k.nvb); break;
    case 128: ens_z_run<R, 128>(P.cl[k.c], k.vb, k.nvb); break;
  }
}

// ------------------------------------------------------------------ Y
template <typename R> struct YClass {
  FieldMaps maps, omaps;  // omaps: the warp-line body's store boxes
  Fields<R> fld;
  const cx<R> *tw;
  int nz, ni, nf, nruns, nxh, rb, rbo;
  const int *jpos, *jneg;
  PipeCtl ctl;
};
template <typename R> struct YMulti {
  int ncls, nsm, per;
  int n[kEnsMaxCls], b0[kEnsMaxCls], nb[kEnsMaxCls];
  YClass<R> cl[kEnsMaxCls];
};
template <int N> constexpr int ens_y_kb() {
  constexpr int E = N < 8 ? N : 8;
  return kEnsThreads / (kEnsYBZ * (N / E));
}
// Lines the warp-line body takes: as many groups of its size as make up the CTA.
template <typename R> constexpr int ens_y_warp_BZ() { return sizeof(R) == 4 ? 16 : 8; }
constexpr int ens_y_warp_E(int N) { return N == 64 ? 8 : 16; }
template <typename R, int N> struct EnsYWarp {
  using G = YWarpGeom<R, N, ens_y_warp_E(N), ens_y_warp_BZ<R>()>;
  static constexpr int groups = kEnsThreads / G::NT;
  static constexpr size_t group = (G::smem + 1023) / 1024 * 1024;
  static_assert(groups * G::NT == kEnsThreads, "one CTA size for all classes");
};
template <typename R, int N> constexpr size_t ens_y_smem() {
  if constexpr (y_warp_line<R>(N)) return EnsYWarp<R, N>::groups * EnsYWarp<R, N>::group + 1024;
  else {
    constexpr int E = N < 8 ? N : 8;
    return YGeom<R, N, E, kEnsYBZ, ens_y_kb<N>()>::smem_bytes(3);
  }
}

template <typename R, int N, int S> __device__ __forceinline__ void ens_y_run(const YClass<R> &k, int vb, int nvb) {
  if constexpr (y_warp_line<R>(N)) {
    using W = EnsYWarp<R, N>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int g = (int)threadIdx.x / W::G::NT;
    ywarp_body<R, N, ens_y_warp_E(N), ens_y_warp_BZ<R>(), S>(
        vb * W::groups + g, nvb * W::groups, g, align1024(smem_raw) + g * W::group, k.maps, k.omaps, k.tw,
        k.nz / ens_y_warp_BZ<R>(), k.ni, k.nf, k.nruns, k.nxh, k.jpos, k.jneg, k.rb, k.rbo, k.ctl);
  } else {
    constexpr int E = N < 8 ? N : 8;
    ypipe_body<R, N, E, kEnsYBZ, 3, S, ens_y_kb<N>()>(vb, nvb, k.maps, k.fld, k.tw, k.nz, k.ni, k.nf, k.nruns, k.nxh,
                                                      k.jpos, k.jneg, k.rb, k.ctl);
  }
}

template <typename R, int S>
__global__ void __launch_bounds__(kEnsThreads) ymulti_kernel(const __grid_constant__ YMulti<R> P) {
  const EnsCta k = ens_cta(P);
  switch (P.n[k.c]) {
    case 16: ens_y_run<R, 16, S>(P.cl[k.c], k.vb, k.nvb); break;
    case 32: ens_y_run<R, 32, S>(P.cl[k.c], k.vb, k.nvb); break;
    case 64: ens_y_run<R, 64, S>(P.cl[k.c], k.vb, k.nvb); break;
    case 128: ens_y_run<R, 128, S>(P.cl[k.c], k.vb, k.nvb); break;
  }
}

// ------------------------------------------------------------------ X
template <typename R> struct XClass {
  FieldMaps maps;
  Fields<R> out;
  const cx<R> *tw;
  int ny, nz, rows, nbox, rb, nruns, nxh;
  R scale;
  PipeCtl ctl;
};
template <typename R> struct XMulti {
  int ncls, nsm, per;
  int n[kEnsMaxCls], b0[kEnsMaxCls], nb[kEnsMaxCls];
  XClass<R> cl[kEnsMaxCls];
};
template <typename R, int NX> constexpr int ens_x_E() { return ens_xE<R>() < NX / 2 ? ens_xE<R>() : NX / 2; }
template <typename R, int NX> constexpr int ens_x_yb() {
  return kEnsThreads / (ens_xBZ<R>() * (NX / 2 / ens_x_E<R, NX>()));
}
// Lines of 64 points and more run the warp-line body of their own launches
// (xnl.cuh), in as many groups of its size as make up the CTA.  Its outputs
// replace its first inputs, so one set of tensor maps serves both.
constexpr bool ens_warp_lines(int nx) { return nx >= 64; }
template <typename R> constexpr int ens_warp_BZ() { return sizeof(R) == 4 ? 16 : 8; }
template <typename R, int NX> struct EnsWarp {
  template <int LE> using G = XnlGeom<R, NX, 8, ens_warp_BZ<R>(), LE>;
  static constexpr int NT = G<8>::NT, groups = kEnsThreads / NT;
  // FP64 groups with four stages left one CTA of four warps on an SM (64 runs of
  // 64^3: 2.12 ms a step; with two stages, two CTAs, 1.71)
  static constexpr int STAGES = sizeof(R) == 4 ? kEnsXStages : 2;
  static constexpr size_t group = (G<8>::fixed + STAGES * G<8>::tile + 1023) / 1024 * 1024;
  static_assert(groups * NT == kEnsThreads, "one CTA size for all classes");
};
template <typename R, int NX> constexpr size_t ens_x_smem() {
  if constexpr (ens_warp_lines(NX)) return EnsWarp<R, NX>::groups * EnsWarp<R, NX>::group + 1024;
  else
  return XGeom<R, NX, ens_xBZ<R>(), ens_x_yb<R, NX>()>::smem_bytes(kEnsXStages);
}

template <typename R, int NX> __device__ __forceinline__ void ens_x_run(const XClass<R> &k, int vb, int nvb) {
  if constexpr (ens_warp_lines(NX)) {
    using W = EnsWarp<R, NX>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int g = (int)threadIdx.x / W::NT;
    unsigned char *sm = align1024(smem_raw) + g * W::group;
    vb = vb * W::groups + g;
    nvb *= W::groups;
    constexpr int BZ = ens_warp_BZ<R>();
    if (k.rows <= 6 * W::template G<6>::T)
      xnl_body<R, NX, 8, BZ, 0, 6, W::STAGES>(vb, nvb, g, sm, k.maps, k.maps, k.tw, k.ny, k.nz, k.scale, k.rows, k.nbox,
                                                k.rb, k.nruns, k.nxh, k.ctl);
    else
      xnl_body<R, NX, 8, BZ, 0, 8, W::STAGES>(vb, nvb, g, sm, k.maps, k.maps, k.tw, k.ny, k.nz, k.scale, k.rows, k.nbox,
                                                k.rb, k.nruns, k.nxh, k.ctl);
  } else {
    xpipe_nl_body<R, NX, ens_x_E<R, NX>(), ens_xBZ<R>(), 0, kEnsXStages, ens_x_yb<R, NX>()>(
        vb, nvb, k.maps, k.out, k.tw, k.ny, k.nz, k.scale, k.rows, k.nbox, k.rb, k.nruns, k.nxh, k.ctl);
  }
}

template <typename R>
__global__ void __launch_bounds__(kEnsThreads) xmulti_kernel(const __grid_constant__ XMulti<R> P) {
  const EnsCta k = ens_cta(P);
  switch (P.n[k.c]) {
    case 16: ens_x_run<R, 16>(P.cl[k.c], k.vb, k.nvb); break;
    case 32: ens_x_run<R, 32>(P.cl[k.c], k.vb, k.nvb); break;
    case 64: ens_x_run<R, 64>(P.cl[k.c], k.vb, k.nvb); break;
    case 128: ens_x_run<R, 128>(P.cl[k.c], k.vb, k.nvb); break;
  }
}

}  // namespace gb
