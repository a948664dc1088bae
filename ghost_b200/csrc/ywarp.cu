// ywarp.cu -- launches of the warp-line Y pass (ywarp.cuh).
#include "ywarp.cuh"

#include "internal.cuh"

namespace gb {

template <int N, int E, int BZ, int S>
static int launch(ghost_ctx *c, const Fields<float> &f, int nf, const Prune &pr) {
  using G = YWarpGeom<N, E, BZ>;
  auto kern = ywarp_kernel<N, E, BZ, S>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem));
  const int ni = pr.jpos ? pr.ni : c->nxh;
  const int grid = persistent_grid(c, kern, G::NT, G::smem, (long)(c->nz / BZ) * ni * c->nruns * nf);
  // the pruned inverse loads, and the pruned forward pass stores, boxes of 32
  // rows that cover the live ones; everything else moves in boxes of 256
  const int rb = (pr.jpos && S > 0) ? 32 : 256, rbo = (pr.jpos && S < 0) ? 32 : 256;
  const CUtensorMapSwizzle swz = G::RB == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  FieldMaps maps, omaps;
  for (int q = 0; q < nf; ++q) {
    GB_CHECK(field_map(c, f.p[q], BZ, rb, 1, &maps.m[q], swz));
    GB_CHECK(field_map(c, f.p[q], BZ, rbo, 1, &omaps.m[q], swz));
  }
  const int ts = timer_begin(c, S > 0 ? GHOST_TIMER_Y_INV : GHOST_TIMER_Y_FWD);
  GB_CHECK(launch_dep(c, nf, kern, grid, G::NT, G::smem, maps, omaps, (const float2 *)c->tw_y, c->nz / BZ, ni, nf, c->nruns, c->nxh, pr.jpos, pr.jneg, rb, rbo, pipe_ctl(c)));
  timer_end(c, ts);
  return post_launch(c);
}

template <int S> int launch_ywarp(ghost_ctx *c, const Fields<float> &f, int nf, const Prune &pr) {
  switch (c->ny) {
    case 256: return launch<256, 16, 16, S>(c, f, nf, pr);
    case 512: return launch<512, 32, 16, S>(c, f, nf, pr);
    case 1024: return launch<1024, 32, 8, S>(c, f, nf, pr);
  }
  return fail(GHOST_ERR_SIZE, "ny=%d has no warp-line Y pass", c->ny);
}
template int launch_ywarp<+1>(ghost_ctx *, const Fields<float> &, int, const Prune &);
template int launch_ywarp<-1>(ghost_ctx *, const Fields<float> &, int, const Prune &);

}  // namespace gb
