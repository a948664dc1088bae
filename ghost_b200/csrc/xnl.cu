// xnl.cu -- launches of the warp-line X pass (xnl.cuh).
#include "xnl.cuh"

#include <algorithm>

#include "internal.cuh"

namespace gb {

template <typename R, int NX, int E, int BZ, int PHYS, int LE, int MINB>
static int launch(ghost_ctx *c, const void *const *ins, void *const *outs, int rows) {
  using G = XnlGeom<R, NX, E, BZ, LE>;
  constexpr int NIN = PHYS == 0 ? 6 : 9, NOUT = PHYS == 0 ? 3 : 4;
  constexpr int STAGES = G::stages(226 * 1024 / MINB - 1024);
  constexpr size_t smem = G::fixed + STAGES * G::tile;
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = xnl_kernel<R, NX, E, BZ, PHYS, LE, STAGES, MINB>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const XnlBoxes bx(rows);
  const CUtensorMapSwizzle swz = G::RB == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  constexpr unsigned U = G::ES / 8;
  FieldMaps maps, omaps;
  for (int q = 0; q < NIN; ++q) GB_CHECK(field_map(c, ins[q], BZ * U, 1, bx.rb, &maps.m[q], swz));
  for (int q = 0; q < NOUT; ++q) GB_CHECK(field_map(c, outs[q], BZ * U, 1, bx.rb, &omaps.m[q], swz));
  const R nn = (R)c->nx * (R)c->ny * (R)c->nz_glob;
  const int grid = persistent_grid(c, kern, G::NT, smem, (long)(c->nz / BZ) * c->ny * c->nruns);
  GB_CHECK(launch_dep(c, NIN, kern, grid, G::NT, smem, maps, omaps, (const cx<R> *)c->tw_x, c->ny, c->nz, (R)1 / (nn * nn),
                      rows, bx.nbox, bx.rb, c->nruns, c->nxh, pipe_ctl(c)));
  return GHOST_OK;
}

// row groups that exist: 11 of 16 (6 of 8) when the 2/3 truncation leaves no
// more rows than that, all of them otherwise
template <typename R, int NX, int E, int BZ, int MINB>
static int pick(ghost_ctx *c, bool bouss, const void *const *ins, void *const *outs, int rows) {
  constexpr int M = NX / 2, T = M / E, LP = E == 16 ? 11 : 6;
  const int n = rows > 0 ? rows : M + 1;
  if (n <= LP * T)
    return bouss ? launch<R, NX, E, BZ, 1, LP, MINB>(c, ins, outs, n) : launch<R, NX, E, BZ, 0, LP, MINB>(c, ins, outs, n);
  return bouss ? launch<R, NX, E, BZ, 1, E, MINB>(c, ins, outs, n) : launch<R, NX, E, BZ, 0, E, MINB>(c, ins, outs, n);
}

// Lines of 64 points and more (shorter ones leave a warp's lines nothing to
// exchange with); FP64 up to 512 (a 1024-point line would be 64 lanes).  The
// tiles must divide nz, which only a rank's z-slab of a decomposed run can fail.
// Where a lane holds twice the values that a thread of the CTA-wide kernel
// does (FP64, and FP32 from 256 points on), its chains are twice as long, and a
// grid that gives a multiprocessor four warps or fewer is faster CTA-wide: us of
// X a Boussinesq step, CTA-wide and here, FP64 64 x 64 x 32 (256 warps) 33.7 and
// 39.8, 256 x 64 x 16 (512) 42.3 and 48.9, x 32 (1024) 72.4 and 56.5; FP32 1024 x
// 16 x 16 (256) 58 and 69, 256 x 64 x 64 (1024) 74 and 50.  The classes of an
// ensemble share the GPU, and their one launch a pass has this body only.
bool xnl_takes(ghost_ctx *c) {
  const bool sp = c->precision == GHOST_SINGLE;
  const int bz = sp && c->nx < 1024 ? 16 : 8;
  if (c->nx < 64 || c->nz % bz != 0 || (!sp && c->nx == 1024)) return false;
  if (c->shares_gpu || (sp && c->nx < 256)) return true;
  // warps of a tile at these lengths (XnlGeom::NW)
  const int nw = c->nx >= 512 ? 8 : c->nx / 64;
  return (long)(c->nz / bz) * c->ny * c->nruns * nw > 4L * sm_count(c);
}

int launch_xnl(ghost_ctx *c, bool bouss, const void *const *ins, void *const *outs, int rows) {
  if (c->precision == GHOST_SINGLE) {
    switch (c->nx) {
      case 64: return pick<float, 64, 8, 16, 6>(c, bouss, ins, outs, rows);
      case 128: return pick<float, 128, 8, 16, 4>(c, bouss, ins, outs, rows);
      case 256: return pick<float, 256, 16, 16, 2>(c, bouss, ins, outs, rows);
      case 512: return pick<float, 512, 16, 16, 1>(c, bouss, ins, outs, rows);
      case 1024: return pick<float, 1024, 16, 8, 1>(c, bouss, ins, outs, rows);
    }
  } else {
    switch (c->nx) {
      case 64: return pick<double, 64, 8, 8, 6>(c, bouss, ins, outs, rows);
      case 128: return pick<double, 128, 8, 8, 4>(c, bouss, ins, outs, rows);
      case 256: return pick<double, 256, 8, 8, 2>(c, bouss, ins, outs, rows);
      case 512: return pick<double, 512, 8, 8, 1>(c, bouss, ins, outs, rows);
    }
  }
  return fail(GHOST_ERR_SIZE, "nx=%d has no warp-line X pass", c->nx);
}

}  // namespace gb
