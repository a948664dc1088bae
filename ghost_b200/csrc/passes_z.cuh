// passes_z.cuh -- launches of the Z passes (passes.cuh), one template instance
// per line length; passes_z32.cu and passes_z64.cu instantiate them.
#pragma once
#include <algorithm>

#include "internal.cuh"
#include "zwarp.cuh"

namespace gb {

template <class Op> struct ZKind;
template <typename R, int S, int NF> struct ZKind<ZC2C<R, S, NF>> { static constexpr int value = GHOST_TIMER_Z_C2C; };
template <typename R, int P> struct ZKind<ZInv<R, P>> { static constexpr int value = GHOST_TIMER_Z_INV; };
template <typename R> struct ZKind<ZGrad<R>> { static constexpr int value = GHOST_TIMER_Z_INV; };
template <typename R> struct ZKind<ZNorm<R>> { static constexpr int value = GHOST_TIMER_Z_INV; };
template <typename R> struct ZKind<ZInvMhd<R>> { static constexpr int value = GHOST_TIMER_Z_INV; };
template <typename R> struct ZKind<ZFwdMhd<R>> { static constexpr int value = GHOST_TIMER_Z_FWD; };
template <typename R> struct ZKind<ZFwdHD<R>> { static constexpr int value = GHOST_TIMER_Z_FWD; };
template <typename R> struct ZKind<ZFwdBouss<R>> { static constexpr int value = GHOST_TIMER_Z_FWD; };

template <typename R, int N, int LPB, int STAGES0, int MINB, class Op>
int launch_z_cfg(ghost_ctx *c, const Op &op, const Prune &pr) {
  constexpr int E = zE<R>() < N ? zE<R>() : N, T = N / E;
  using G = ZGeom<R, N, E, LPB, Op::NLOAD>;
  // (six fields of 1024-point FP64 lines: two stages are 249 KB, one is 151)
  constexpr int STAGES = G::smem_bytes(STAGES0) <= 200 * 1024 ? STAGES0 : (G::smem_bytes(2) <= 227 * 1024 ? 2 : 1);
  constexpr size_t smem = G::smem_bytes(STAGES);
  static_assert(smem <= 227 * 1024, "shared memory");
  const int nlines = pr.lines ? pr.nlines : c->ny * c->nxh * c->nruns;
  auto kern = zpipe_kernel<R, N, E, LPB, STAGES, MINB, Op>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = persistent_grid(c, kern, LPB * T, smem, (nlines + LPB - 1) / LPB);
  const int ts = timer_begin(c, ZKind<Op>::value);
  GB_CHECK(launch_dep(c, Op::NLOAD, kern, grid, LPB * T, smem, op, (const cx<R> *)c->tw_z, pr.lines, nlines, pipe_ctl(c)));
  timer_end(c, ts);
  return post_launch(c);
}

// lines per CTA, halved from want until a two-stage ring of NL fields fits
template <typename R, int N, int NL> constexpr int fit_lines(int want) {
  int lpb = want;
  while (lpb > 1 && ((size_t)2 * NL * lpb * N + N + (size_t)2 * lpb * (N + N / 8)) * sizeof(cx<R>) + 24 > 220 * 1024)
    lpb /= 2;
  return lpb;
}

// whether the one-stage ring with four CTAs per SM is an Op's better one at
// lines of N points.  us a step with two stages and three CTAs, and with one and
// four: HD z_fwd FP32 256 x 128 x 512 246 and 218, x 1024 482 and 448, FP64 128 x
// 128 x 256 123.3 and 120.3, x 512 252.4 and 253.6; Boussinesq z_inv FP32 256 x
// 128 x 512 315 and 284, x 1024 745 and 696, its z_fwd x 512 339 and 309.  Not for
// the plain transforms (0.178 and 0.199 ms at 512^3 FP32), the FP64 inverse (0.235
// and 0.238 at 256^3), and the Boussinesq update where its 128 registers spill
// four components: FP64 (128 x 128 x 256 176 and 193, x 512 387 and 423) and
// FP32 at 1024 points (704 and 865).
template <class Op, int N> struct OneStage { static constexpr bool value = true; };
template <typename R, int S, int NF, int N> struct OneStage<ZC2C<R, S, NF>, N> { static constexpr bool value = false; };
template <int P, int N> struct OneStage<ZInv<double, P>, N> { static constexpr bool value = false; };
template <int N> struct OneStage<ZFwdBouss<double>, N> { static constexpr bool value = false; };
template <> struct OneStage<ZFwdBouss<float>, 1024> { static constexpr bool value = false; };

// CTAs of NWC warps (zwarp.cuh)
template <typename R, int N, int E, int NWC, int MINB, class Op>
int launch_zwarp_cfg(ghost_ctx *c, const Op &op, const Prune &pr) {
  using G = ZWarpGeom<R, N, E, Op::NLOAD>;
  const size_t smem = G::smem(NWC);
  static_assert(G::smem(NWC) <= 227 * 1024, "shared memory");
  const int nlines = pr.lines ? pr.nlines : c->ny * c->nxh * c->nruns;
  auto kern = zwarp_kernel<R, N, E, NWC, MINB, Op>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = persistent_grid(c, kern, 32 * NWC, smem, (nlines + G::LW * NWC - 1) / (G::LW * NWC));
  const int ts = timer_begin(c, ZKind<Op>::value);
  GB_CHECK(launch_dep(c, Op::NLOAD, kern, grid, 32 * NWC, smem, op, (const cx<R> *)c->tw_z, pr.lines, nlines, pipe_ctl(c)));
  timer_end(c, ts);
  return post_launch(c);
}
template <typename R, int N, class Op> int launch_zwarp(ghost_ctx *c, const Op &op, const Prune &pr) {
  constexpr int E = z_warp_E<R, Op>(N);
  // the forward updates hold three or four components: 255 registers in FP64
  constexpr int MINB = ZUpdate<Op>::value && sizeof(R) == 8 ? 2 : 3;
  const int nlines = pr.lines ? pr.nlines : c->ny * c->nxh * c->nruns;
  // few lines: one warp per CTA, so that every SM has work (a 64^3 FP64 step
  // has 740 live lines)
  if (nlines < 8 * ZWarpGeom<R, N, E, Op::NLOAD>::LW * sm_count(c))
    return launch_zwarp_cfg<R, N, E, 1, (N == 512 ? 6 : 4 * MINB)>(c, op, pr);
  // 512 points: three warps and their lines of three fields are half an SM's shared memory
  if constexpr (N == 512) return launch_zwarp_cfg<R, N, E, 3, 2>(c, op, pr);
  else return launch_zwarp_cfg<R, N, E, 4, MINB>(c, op, pr);
}

// The CTA-wide pass of an Op at lines of N points, and the tile variant's
// choice of it.  0: CTAs of 256 threads; 1 (bit 1): of 128 threads; 2 (bits 1
// and 2, lines of 256 points or more): of 128 threads with a two-stage ring and
// at most 170 registers, so that three CTAs share an SM; 3 (bit 5 too): a
// one-stage ring and four CTAs.
template <typename R, int N, class Op> struct ZRing {
  static constexpr int T = N / (zE<R>() < N ? zE<R>() : N);
  static constexpr int L256 = fit_lines<R, N, Op::NLOAD>(256 / T > 0 ? 256 / T : 1);
  static constexpr int L128 = fit_lines<R, N, Op::NLOAD>(128 / T > 0 ? 128 / T : 1);
  static constexpr bool sizes = !z_warp_line<R, Op>(N) && L128 != L256, stages = sizes && N >= 256;
  static constexpr bool one = stages && OneStage<Op, N>::value;
  static int of(int cfg) {
    if (one && (cfg & 38) == 38) return 3;
    if (stages && (cfg & 6) == 6) return 2;
    return sizes && (cfg & 2) ? 1 : 0;
  }
};
template <typename R, int N, class Op> int launch_z_n(ghost_ctx *c, const Op &op, const Prune &pr) {
  if constexpr (z_warp_line<R, Op>(N)) {
    return launch_zwarp<R, N>(c, op, pr);
  } else {
    using Z = ZRing<R, N, Op>;
    const int ring = Z::of(c->tile_cfg);
    if constexpr (Z::one)
      if (ring == 3) return launch_z_cfg<R, N, Z::L128, 1, 4>(c, op, pr);
    if constexpr (Z::stages)
      if (ring == 2) return launch_z_cfg<R, N, Z::L128, 2, 3>(c, op, pr);
    if constexpr (Z::sizes)
      if (ring == 1) return launch_z_cfg<R, N, Z::L128, 3, 1>(c, op, pr);
    return launch_z_cfg<R, N, Z::L256, 3, 1>(c, op, pr);
  }
}

template <typename R, class Op> int launch_z(ghost_ctx *c, const Op &op, const Prune &pr) {
  switch (c->nz) {
    case 16: return launch_z_n<R, 16>(c, op, pr);
    case 32: return launch_z_n<R, 32>(c, op, pr);
    case 64: return launch_z_n<R, 64>(c, op, pr);
    case 128: return launch_z_n<R, 128>(c, op, pr);
    case 256: return launch_z_n<R, 256>(c, op, pr);
    case 512: return launch_z_n<R, 512>(c, op, pr);
    case 1024: return launch_z_n<R, 1024>(c, op, pr);
  }
  return fail(GHOST_ERR_SIZE, "nz=%d unsupported", c->nz);
}

// the rings of an HD step's two z passes with a tile variant
template <typename R> int hd_z_rings(const ghost_ctx *c, int cfg) {
  switch (c->nz) {
#define GB_NZ(N) \
  case N: return ZRing<R, N, ZInv<R, 0>>::of(cfg) + 4 * ZRing<R, N, ZFwdHD<R>>::of(cfg);
    GB_NZ(16) GB_NZ(32) GB_NZ(64) GB_NZ(128) GB_NZ(256) GB_NZ(512) GB_NZ(1024)
#undef GB_NZ
  }
  return 0;
}

#define GB_INST(R)                                                                    \
  template int hd_z_rings<R>(const ghost_ctx *, int);                                 \
  template int launch_z<R, ZInv<R, 0>>(ghost_ctx *, const ZInv<R, 0> &, const Prune &);   \
  template int launch_z<R, ZInv<R, 1>>(ghost_ctx *, const ZInv<R, 1> &, const Prune &);   \
  template int launch_z<R, ZGrad<R>>(ghost_ctx *, const ZGrad<R> &, const Prune &);       \
  template int launch_z<R, ZFwdHD<R>>(ghost_ctx *, const ZFwdHD<R> &, const Prune &);     \
  template int launch_z<R, ZFwdBouss<R>>(ghost_ctx *, const ZFwdBouss<R> &, const Prune &); \
  template int launch_z<R, ZNorm<R>>(ghost_ctx *, const ZNorm<R> &, const Prune &);       \
  template int launch_z<R, ZInvMhd<R>>(ghost_ctx *, const ZInvMhd<R> &, const Prune &);   \
  template int launch_z<R, ZFwdMhd<R>>(ghost_ctx *, const ZFwdMhd<R> &, const Prune &);   \
  template int launch_z<R, ZC2C<R, -1, 1>>(ghost_ctx *, const ZC2C<R, -1, 1> &, const Prune &); \
  template int launch_z<R, ZC2C<R, -1, 3>>(ghost_ctx *, const ZC2C<R, -1, 3> &, const Prune &); \
  template int launch_z<R, ZC2C<R, -1, 6>>(ghost_ctx *, const ZC2C<R, -1, 6> &, const Prune &); \
  template int launch_z<R, ZC2C<R, +1, 1>>(ghost_ctx *, const ZC2C<R, +1, 1> &, const Prune &);

}  // namespace gb
