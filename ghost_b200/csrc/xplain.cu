// xplain.cu -- launches of the warp-line plain x transforms (xplain.cuh).
#include "xplain.cuh"

#include "internal.cuh"

namespace gb {

// Lines of 64 points and more in both precisions, except where the warp-wide
// lines of xwarp.cuh (FP32, 512 points) or nothing fits (FP64, 1024 points).
// Every device array of the C ABI starts on 16 bytes, as the bulk copies need.
bool xline_takes(const ghost_ctx *c) {
  const bool sp = c->precision == GHOST_SINGLE;
  if (c->nruns != 1 || c->nx < 64 || (sp ? c->nx == 512 : c->nx == 1024)) return false;
  return c->nz % (sp && c->nx < 1024 ? 16 : 8) == 0;
}

static CUtensorMapSwizzle swizzle_of(int row_bytes) {
  return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
}

template <typename R, int NX, int E, int BZ> static int r2c(ghost_ctx *c, const void *const *in, void *const *out, int nf) {
  using G = XnlGeom<R, NX, E, BZ, E>;
  using P = XPlainGeom<R, NX, E, BZ>;
  constexpr int STAGES = P::r2c(3) <= 110 * 1024 ? 3 : 2;
  auto kern = xline_r2c_kernel<R, NX, E, BZ, STAGES>;
  constexpr size_t smem = P::r2c(STAGES);
  static_assert(smem <= 227 * 1024, "shared memory");
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const XnlBoxes bx(G::M + 1);
  CFields<R> f{};
  FieldMaps maps;
  for (int q = 0; q < nf; ++q) {
    f.p[q] = (const cx<R> *)in[q];
    GB_CHECK(field_map(c, out[q], BZ * G::ES / 8, 1, bx.rb, &maps.m[q], swizzle_of(G::RB)));
  }
  const int grid = persistent_grid(c, kern, G::NT, smem, (long)(c->nz / BZ) * c->ny * nf);
  GB_CHECK(launch_dep(c, nf, kern, grid, G::NT, smem, f, maps, (const cx<R> *)c->tw_x, c->ny, c->nz, nf, bx.nbox, bx.rb,
                      pipe_ctl(c)));
  return GHOST_OK;
}

template <typename R, int NX, int E, int BZ> static int c2r(ghost_ctx *c, const void *in, void *out) {
  using G = XnlGeom<R, NX, E, BZ, E>;
  using P = XPlainGeom<R, NX, E, BZ>;
  constexpr int STAGES = P::c2r(3) <= 110 * 1024 ? 3 : 2;
  auto kern = xline_c2r_kernel<R, NX, E, BZ, STAGES>;
  constexpr size_t smem = P::c2r(STAGES);
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const XnlBoxes bx(G::M + 1);
  CUtensorMap m;
  GB_CHECK(field_map(c, in, BZ * G::ES / 8, 1, bx.rb, &m, swizzle_of(G::RB)));
  const int grid = persistent_grid(c, kern, G::NT, smem, (long)(c->nz / BZ) * c->ny);
  GB_CHECK(launch_dep(c, 1, kern, grid, G::NT, smem, m, (R *)out, (const cx<R> *)c->tw_x, c->ny, c->nz, bx.nbox, bx.rb, pipe_ctl(c)));
  return GHOST_OK;
}

template <typename R, int NX, int E, int BZ>
static int features(ghost_ctx *c, const void *const *spec, float *x, float gs, float delta) {
  using G = XnlGeom<R, NX, E, BZ, E>;
  using P = XPlainGeom<R, NX, E, BZ>;
  constexpr int STAGES = P::feat(3) <= 112 * 1024 ? 3 : 2;
  auto kern = xline_features_kernel<R, NX, E, BZ, STAGES>;
  constexpr size_t smem = P::feat(STAGES);
  static_assert(smem <= 227 * 1024, "shared memory");
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const XnlBoxes bx(G::M + 1);
  FieldMaps maps;
  for (int q = 0; q < 9; ++q) GB_CHECK(field_map(c, spec[q], BZ * G::ES / 8, 1, bx.rb, &maps.m[q], swizzle_of(G::RB)));
  const int grid = persistent_grid(c, kern, G::NT, smem, (long)(c->nz / BZ) * c->ny);
  // nine fields, but started early as three would be (launch_dep): with nine a
  // closure step (RK2) of 128^3 FP32 took 773 us instead of 771, FP64 1245 instead of 1236
  GB_CHECK(launch_dep(c, 3, kern, grid, G::NT, smem, maps, x, (const cx<R> *)c->tw_x, c->ny, c->nz, bx.nbox, bx.rb, (R)(1.0 / (double)c->nreal), gs, delta, pipe_ctl(c)));
  return GHOST_OK;
}

#define GB_LINES(F, ...)                                              \
  if (c->precision == GHOST_SINGLE) {                                 \
    switch (c->nx) {                                                  \
      case 64: return F<float, 64, 8, 16>(c, __VA_ARGS__);            \
      case 128: return F<float, 128, 8, 16>(c, __VA_ARGS__);          \
      case 256: return F<float, 256, 16, 16>(c, __VA_ARGS__);         \
      case 1024: return F<float, 1024, 16, 8>(c, __VA_ARGS__);        \
    }                                                                 \
  } else {                                                            \
    switch (c->nx) {                                                  \
      case 64: return F<double, 64, 8, 8>(c, __VA_ARGS__);            \
      case 128: return F<double, 128, 8, 8>(c, __VA_ARGS__);          \
      case 256: return F<double, 256, 8, 8>(c, __VA_ARGS__);          \
      case 512: return F<double, 512, 8, 8>(c, __VA_ARGS__);          \
    }                                                                 \
  }                                                                   \
  return fail(GHOST_ERR_SIZE, "nx=%d has no warp-line x transform", c->nx);

int launch_xline_r2c(ghost_ctx *c, const void *const *in, void *const *out, int nf) { GB_LINES(r2c, in, out, nf) }
int launch_xline_c2r(ghost_ctx *c, const void *in, void *out) { GB_LINES(c2r, in, out) }

// the closure's rows of a tile fit shared memory up to 128-point lines, and
// leave it by bulk copies; rows that start elsewhere (a caller's float array)
// take the element-wise kernel
bool xline_features_takes(const ghost_ctx *c, const void *x) {
  return c->nx <= 128 && xline_takes(c) && reinterpret_cast<uintptr_t>(x) % 16 == 0;
}
int launch_xline_features(ghost_ctx *c, const void *const *spec, float *x, float gs, float delta) {
  if (c->precision == GHOST_SINGLE)
    return c->nx == 64 ? features<float, 64, 8, 16>(c, spec, x, gs, delta) : features<float, 128, 8, 16>(c, spec, x, gs, delta);
  return c->nx == 64 ? features<double, 64, 8, 8>(c, spec, x, gs, delta) : features<double, 128, 8, 8>(c, spec, x, gs, delta);
}

}  // namespace gb
