// ywarp.cu -- launches of the warp-line Y pass (ywarp.cuh).
#include "ywarp.cuh"

#include "internal.cuh"

namespace gb {

template <typename R, int N, int E, int BZ, int S, int MINB>
static int launch(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr) {
  using G = YWarpGeom<R, N, E, BZ>;
  constexpr size_t smem = G::smem + 1024;
  auto kern = ywarp_kernel<R, N, E, BZ, S, MINB>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int ni = pr.jpos ? pr.ni : c->nxh;
  const int grid = persistent_grid(c, kern, G::NT, smem, (long)(c->nz / BZ) * ni * c->nruns * nf);
  const YWarpBoxes bx(N, pr.jpos != nullptr, S);
  const CUtensorMapSwizzle swz = G::RB == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  constexpr unsigned U = G::ES / 8;
  FieldMaps maps, omaps;
  for (int q = 0; q < nf; ++q) {
    GB_CHECK(field_map(c, f.p[q], BZ * U, bx.rb, 1, &maps.m[q], swz));
    GB_CHECK(field_map(c, f.p[q], BZ * U, bx.rbo, 1, &omaps.m[q], swz));
  }
  const int ts = timer_begin(c, S > 0 ? GHOST_TIMER_Y_INV : GHOST_TIMER_Y_FWD);
  GB_CHECK(launch_dep(c, nf, kern, grid, G::NT, smem, maps, omaps, (const cx<R> *)c->tw_y, c->nz / BZ, ni, nf, c->nruns,
                      c->nxh, pr.jpos, pr.jneg, bx.rb, bx.rbo, pipe_ctl(c)));
  timer_end(c, ts);
  return post_launch(c);
}

template <typename R, int S> int launch_ywarp(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr) {
  if constexpr (sizeof(R) == 4) {
    switch (c->ny) {
      case 64: return launch<R, 64, 8, 16, S, 6>(c, f, nf, pr);
      case 128: return launch<R, 128, 16, 16, S, 4>(c, f, nf, pr);
      case 256: return launch<R, 256, 16, 16, S, 2>(c, f, nf, pr);
      case 512: return launch<R, 512, 32, 16, S, 1>(c, f, nf, pr);
      case 1024: return launch<R, 1024, 32, 8, S, 1>(c, f, nf, pr);
    }
  } else {
    switch (c->ny) {
      case 64: return launch<R, 64, 8, 8, S, 8>(c, f, nf, pr);
      case 128: return launch<R, 128, 16, 8, S, 4>(c, f, nf, pr);
      case 256: return launch<R, 256, 16, 8, S, 2>(c, f, nf, pr);
    }
  }
  return fail(GHOST_ERR_SIZE, "ny=%d has no warp-line Y pass", c->ny);
}
#define GB_INST(R)                                                                \
  template int launch_ywarp<R, +1>(ghost_ctx *, const Fields<R> &, int, const Prune &); \
  template int launch_ywarp<R, -1>(ghost_ctx *, const Fields<R> &, int, const Prune &);
GB_INST(float)
GB_INST(double)
#undef GB_INST

}  // namespace gb
