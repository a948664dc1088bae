// passes_y.cu -- launches of the Y passes (passes.cuh), one template instance
// per line length.
#include <algorithm>

#include "internal.cuh"
#include "ywarp.cuh"

namespace gb {

// y tile width: BZ0 z-lines, at most 1024 threads, narrowed until a
// two-stage ring fits in shared memory (FP64 with 1024-point lines)
template <typename R, int N, int BZ0> constexpr int y_tile_width() {
  constexpr int E = N < 8 ? N : 8, T = N / E;
  int bz = BZ0 * T <= 1024 ? BZ0 : 1024 / T;
  while (bz > 1 && ((size_t)3 * bz * N + N) * sizeof(cx<R>) + 24 > 220 * 1024) bz /= 2;
  return bz;
}

// kx indices per y tile: short lines put several kx in one tile so that a
// CTA has at least 128 threads
template <int N, int E, int BZ> constexpr int y_kb() {
  return BZ * (N / E) >= 128 ? 1 : 128 / (BZ * (N / E));
}

template <typename R, int N, int S, int BZ0>
int launch_y_cfg(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr) {
  constexpr int E = N < 8 ? N : 8, T = N / E;
  constexpr int BZ = y_tile_width<R, N, BZ0>();
  constexpr int KB = y_kb<N, E, BZ>();
  using G = YGeom<R, N, E, BZ, KB>;
  constexpr int STAGES = G::smem_bytes(3) <= 200 * 1024 ? 3 : 2;
  if (c->nz < BZ) return fail(GHOST_ERR_SIZE, "nz=%d below the y-pass tile width %d", c->nz, BZ);
  constexpr size_t smem = G::smem_bytes(STAGES);
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = ypipe_kernel<R, N, E, BZ, STAGES, S, KB>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int ni = pr.jpos ? pr.ni : c->nxh;
  const long ntiles = (long)(c->nz / BZ) * ((ni + KB - 1) / KB) * c->nruns * nf;
  const int grid = persistent_grid(c, kern, KB * BZ * T, smem, ntiles);
  // box rows: 32 (or N/2) for the pruned inverse, whole halves otherwise
  const int rb = (pr.jpos && S > 0) ? std::min(32, N / 2) : std::min(N, 256);
  const unsigned U = sizeof(R) == 4 ? 1 : 2;
  FieldMaps maps;
  for (int q = 0; q < nf; ++q) GB_CHECK(field_map(c, f.p[q], BZ * U, rb, 1, &maps.m[q]));
  const int ts = timer_begin(c, S > 0 ? GHOST_TIMER_Y_INV : GHOST_TIMER_Y_FWD);
  GB_CHECK(launch_dep(c, nf, kern, grid, KB * BZ * T, smem, maps, f, (const cx<R> *)c->tw_y, c->nz, ni, nf, c->nruns,
                      c->nxh, pr.jpos, pr.jneg, rb, pipe_ctl(c)));
  timer_end(c, ts);
  return post_launch(c);
}

// whether lines of N points have a choice of tiles: the 16-wide one needs two
// stages of 16 lines in shared memory (which leaves out FP64 lines of 512
// points and more)
template <typename R, int N> constexpr bool y_has_wide() {
  constexpr int E = N < 8 ? N : 8, T = N / E;
  return !y_warp_line<R>(N) && YGeom<R, N, E, (16 * T <= 1024 ? 16 : 1024 / T)>::smem_bytes(2) <= 227 * 1024;
}
template <typename R> bool y_wide_choice(const ghost_ctx *c) {
  switch (c->ny) {
#define GB_NY(N) \
  case N: return y_has_wide<R, N>();
    GB_NY(16) GB_NY(32) GB_NY(64) GB_NY(128) GB_NY(256) GB_NY(512) GB_NY(1024)
#undef GB_NY
  }
  return false;
}

// tiles 8 z-lines wide, or 16 with tile variant bit 0
template <typename R, int N, int S> int launch_y_n(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr) {
  // lines the warp-line kernel takes, whatever the tile variant (its y bit
  // chooses between the tiles of other line lengths)
  if constexpr (y_warp_line<R>(N)) {
    return launch_ywarp<R, S>(c, f, nf, pr);
  } else {
    if constexpr (y_has_wide<R, N>()) {
      if ((c->tile_cfg & 1) && c->nz >= 16) return launch_y_cfg<R, N, S, 16>(c, f, nf, pr);
    }
    return launch_y_cfg<R, N, S, 8>(c, f, nf, pr);
  }
}

template <typename R, int S> int launch_y(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr) {
  switch (c->ny) {
    case 16: return launch_y_n<R, 16, S>(c, f, nf, pr);
    case 32: return launch_y_n<R, 32, S>(c, f, nf, pr);
    case 64: return launch_y_n<R, 64, S>(c, f, nf, pr);
    case 128: return launch_y_n<R, 128, S>(c, f, nf, pr);
    case 256: return launch_y_n<R, 256, S>(c, f, nf, pr);
    case 512: return launch_y_n<R, 512, S>(c, f, nf, pr);
    case 1024: return launch_y_n<R, 1024, S>(c, f, nf, pr);
  }
  return fail(GHOST_ERR_SIZE, "ny=%d unsupported", c->ny);
}

#define GB_INST(R)                                                            \
  template bool y_wide_choice<R>(const ghost_ctx *);                              \
  template int launch_y<R, +1>(ghost_ctx *, const Fields<R> &, int, const Prune &); \
  template int launch_y<R, -1>(ghost_ctx *, const Fields<R> &, int, const Prune &);
GB_INST(float)
GB_INST(double)
#undef GB_INST

}  // namespace gb
