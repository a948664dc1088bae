// passes_x.cu -- launches of the X passes (passes.cuh), one template instance
// per line length.
#include <algorithm>

#include "internal.cuh"
#include "xwarp.cuh"

namespace gb {

// y rows per x tile: short lines put several y rows in one tile so that a
// CTA has at least 128 threads
template <typename R, int NX, int BZ> constexpr int x_yb() {
  constexpr int E = xE<R>() < NX / 2 ? xE<R>() : NX / 2;
  return BZ * (NX / 2 / E) >= 128 ? 1 : 128 / (BZ * (NX / 2 / E));
}

// The fused X pass with tiles of BZ z-values (MINB CTAs per SM).
template <typename R, int NX, int KIND, int BZ, int MINB>
int launch_x_fused(ghost_ctx *c, const void *const *ins, void *const *outs, int rows) {
  constexpr int E = xE<R>() < NX / 2 ? xE<R>() : NX / 2;
  constexpr int YB = x_yb<R, NX, BZ>();
  if (c->ny % YB != 0) return fail(GHOST_ERR_SIZE, "ny=%d not a multiple of the x tile's %d rows", c->ny, YB);
  constexpr int M = NX / 2, T = M / E, NT = YB * BZ * T;
  typedef cx<R> C;
  constexpr int PHYS = KIND == X_HD ? 0 : (KIND == X_BOUSS ? 1 : (KIND == X_MHD ? 2 : 3));
  constexpr int NIN = PHYS == 0 ? 6 : (PHYS == 1 ? 9 : (PHYS == 2 ? 12 : 3));
  constexpr int NOUT = PHYS == 0 ? 3 : (PHYS == 1 ? 4 : (PHYS == 2 ? 6 : 1));
  const int nruns = KIND == X_NORM ? 1 : c->nruns;  // maxabs is of the first run's field
  using G = XGeom<R, NX, BZ, YB>;
  constexpr size_t cap = 220 * 1024 / MINB;  // four stages while MINB CTAs fit an SM
  constexpr int STAGES = G::smem_bytes(4) <= cap ? 4 : (G::smem_bytes(3) <= 200 * 1024 ? 3 : 2);
  constexpr size_t smem = G::smem_bytes(STAGES);
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = xpipe_nl_kernel<R, NX, E, BZ, PHYS, STAGES, MINB, YB>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  Fields<R> fo{};
  for (int q = 0; q < NOUT; ++q) fo.p[q] = (C *)outs[q];
  const R nn = (R)c->nx * (R)c->ny * (R)c->nz_glob;
  const int nrows = rows > 0 ? rows : M + 1;
  // tensor boxes: nbox boxes of rb kx-rows; rb keeps every box 128-byte aligned in shared memory
  const int nbox = (nrows + 255) / 256;
  const int align = std::max(1, 128 / (YB * BZ * (int)sizeof(C)));
  const int rb = ((nrows + nbox - 1) / nbox + align - 1) / align * align;
  if (nbox * rb > M + 8 || rb > 256) return fail(GHOST_ERR_STATE, "x-pass box plan %d x %d exceeds the tile", nbox, rb);
  const unsigned U = sizeof(R) == 4 ? 1 : 2;
  FieldMaps maps;
  for (int q = 0; q < NIN; ++q) GB_CHECK(field_map(c, ins[q], BZ * U, YB, rb, &maps.m[q]));
  const int pgrid = persistent_grid(c, kern, NT, smem, (long)(c->nz / BZ) * (c->ny / YB) * nruns);
  // A step's pass with fewer CTAs than multiprocessors is slower started early
  // (us a step, early and not, 256 x 32 x 16 FP32 Boussinesq 150 and 142, 512 x 32 x
  // 16 FP64 HD 106 and 93; 64^3 FP64 HD, 256 CTAs, 81 and 87).
  const bool alone = NX >= 64 && (KIND == X_HD || KIND == X_BOUSS) && pgrid < sm_count(c);
  GB_CHECK(launch_dep(c, alone ? kAlone : NIN, kern, pgrid, NT, smem, maps, fo, (const C *)c->tw_x, c->ny, c->nz, (R)1 / (nn * nn), nrows,
                      nbox, rb, nruns, c->nxh, pipe_ctl(c)));
  return GHOST_OK;
}

// TMA map of a real FP32 field (x fastest) as 8-byte pairs: a box of
// nx/2 pairs x 1 y-row x 8 z-values, the tiles of the plain x transforms.
static int real_map(ghost_ctx *c, const void *base, CUtensorMap *out) {
  PFN_cuTensorMapEncodeTiled_v12000 enc;
  GB_CHECK(encode_fn(&enc));
  const cuuint64_t dims[3] = {(cuuint64_t)c->nx / 2, (cuuint64_t)c->ny, (cuuint64_t)c->nz};
  const cuuint64_t strides[2] = {(cuuint64_t)c->nx * 4, (cuuint64_t)c->nx * c->ny * 4};
  const cuuint32_t box[3] = {(cuuint32_t)c->nx / 2, 1, 8};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(GHOST_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return GHOST_OK;
}

// The plain x transforms with one warp per line (FP32, nx = 512, one run).
static bool xw_plain_ok(const ghost_ctx *c) {
  return c->precision == GHOST_SINGLE && c->nx == 512 && c->nruns == 1 && c->nz % 8 == 0;
}
static int launch_xw_r2c(ghost_ctx *c, const void *in, void *out) {
  constexpr int NX = 512, M = NX / 2, STAGES = 3;
  using G = XWPlainGeom<NX, STAGES>;
  auto kern = xwarp_r2c_kernel<NX, STAGES>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::r2c_bytes));
  const int rb = ((M + 1 + 1) / 2 + 15) / 16 * 16;  // 2 x 144 rows cover the M+1 kx rows
  static_assert(2 * (((M + 2) / 2 + 15) / 16 * 16) <= G::OROWS, "r2c store boxes exceed the output tile");
  CUtensorMap rm, cm;
  GB_CHECK(real_map(c, in, &rm));
  GB_CHECK(field_map(c, out, 8, 1, rb, &cm, CU_TENSOR_MAP_SWIZZLE_64B));
  const int grid = persistent_grid(c, kern, 256, G::r2c_bytes, (long)(c->nz / 8) * c->ny);
  GB_CHECK(launch_dep(c, 1, kern, grid, 256, G::r2c_bytes, rm, cm, (const float2 *)c->tw_x, c->ny, c->nz, rb, pipe_ctl(c)));
  return GHOST_OK;
}
static int launch_xw_c2r(ghost_ctx *c, const void *in, void *out) {
  constexpr int NX = 512, M = NX / 2, STAGES = 4;
  using G = XWPlainGeom<NX, STAGES>;
  auto kern = xwarp_c2r_kernel<NX, STAGES>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::c2r_bytes));
  const int nbox = 2, rb = ((M + 1 + 1) / 2 + 15) / 16 * 16;  // 2 x 144 rows cover the M+1 kx rows
  static_assert(2 * (((M + 2) / 2 + 15) / 16 * 16) <= G::SROWS, "c2r box plan exceeds the slot");
  CUtensorMap m;
  GB_CHECK(field_map(c, in, 8, 1, rb, &m, CU_TENSOR_MAP_SWIZZLE_64B));
  const int grid = persistent_grid(c, kern, 256, G::c2r_bytes, (long)(c->nz / 8) * c->ny);
  GB_CHECK(launch_dep(c, 1, kern, grid, 256, G::c2r_bytes, m, (float *)out, (const float2 *)c->tw_x, c->ny, c->nz, nbox, rb, pipe_ctl(c)));
  return GHOST_OK;
}

template <typename R, int NX, int KIND> int launch_x_n(ghost_ctx *c, const void *in, void *out, const void *const *ins,
                                                       void *const *outs, int rows) {
  constexpr int E = xE<R>() < NX / 2 ? xE<R>() : NX / 2;
  constexpr int M = NX / 2, T = M / E;
  // rows of BZ z values; at most 256 threads so the register-resident
  // real fields of the fused pass fit the register file
  constexpr int BZ = xBZ<R>() * T <= 256 ? xBZ<R>() : (256 / T > 0 ? 256 / T : 1);
  constexpr int NT = BZ * T;
  typedef cx<R> C;
  dim3 grid(c->nz / BZ, c->ny);
  const C *tw = (const C *)c->tw_x;
  const int ts = timer_begin(c, KIND == X_C2R || KIND == X_NORM ? GHOST_TIMER_X_C2R : (KIND == X_R2C ? GHOST_TIMER_X_R2C : GHOST_TIMER_X_NL));
  if constexpr (KIND == X_NORM) {
    GB_CHECK((launch_x_fused<R, NX, KIND, BZ, 2>(c, ins, outs, rows)));
  } else if constexpr (KIND == X_MHD) {
    // v, b and both products of a line live in registers: 255 a thread
    constexpr int YB = x_yb<R, NX, BZ>();
    GB_CHECK((launch_x_fused<R, NX, KIND, BZ, (YB * NT <= 128 ? 2 : 1)>(c, ins, outs, rows)));
  } else if constexpr (KIND == X_HD || KIND == X_BOUSS) {
    // the warp-line kernel (xnl.cuh) where it takes the grid
    if (xnl_takes(c)) {
      GB_CHECK(launch_xnl(c, KIND == X_BOUSS, ins, outs, rows));
      timer_end(c, ts);
      return post_launch(c);
    }
    GB_CHECK((launch_x_fused<R, NX, KIND, BZ, 2>(c, ins, outs, rows)));
  } else if (KIND == X_C2R && xw_plain_ok(c)) {
    GB_CHECK(launch_xw_c2r(c, in, out));
  } else if (KIND == X_R2C && xw_plain_ok(c)) {
    GB_CHECK(launch_xw_r2c(c, in, out));
  } else if (KIND == X_C2R && xline_takes(c)) {
    GB_CHECK(launch_xline_c2r(c, in, out));
  } else if (KIND == X_R2C && xline_takes(c)) {
    GB_CHECK(launch_xline_r2c(c, &in, &out, 1));
  } else if (KIND == X_C2R) {
    const size_t smem = (size_t)(NX + (M + 1) * BZ + M * BZ) * sizeof(C);
    auto kern = xpass_c2r_kernel<R, NX, E, BZ>;
    GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, NT, smem, c->stream>>>((const C *)in, (R *)out, tw, c->ny, c->nz);
  } else {
    const size_t smem = (size_t)(NX + M * BZ) * sizeof(C);
    auto kern = xpass_r2c_kernel<R, NX, E, BZ>;
    GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, NT, smem, c->stream>>>((const R *)in, (C *)out, tw, c->ny, c->nz);
  }
  timer_end(c, ts);
  return post_launch(c);
}

template <typename R, int KIND>
int launch_x(ghost_ctx *c, const void *in, void *out, const void *const *ins, void *const *outs, int rows) {
  switch (c->nx) {
    case 16: return launch_x_n<R, 16, KIND>(c, in, out, ins, outs, rows);
    case 32: return launch_x_n<R, 32, KIND>(c, in, out, ins, outs, rows);
    case 64: return launch_x_n<R, 64, KIND>(c, in, out, ins, outs, rows);
    case 128: return launch_x_n<R, 128, KIND>(c, in, out, ins, outs, rows);
    case 256: return launch_x_n<R, 256, KIND>(c, in, out, ins, outs, rows);
    case 512: return launch_x_n<R, 512, KIND>(c, in, out, ins, outs, rows);
    case 1024: return launch_x_n<R, 1024, KIND>(c, in, out, ins, outs, rows);
  }
  return fail(GHOST_ERR_SIZE, "nx=%d unsupported", c->nx);
}

// The LES closure's input rows from a spectral velocity: the nine gradients
// through z and y passes over all nine, then one x pass that writes
// x[q][3a+b] = (d v_a / d x_b) * gs and x[q][9] = delta directly.
template <typename R, int NX>
int grad9_features_n(ghost_ctx *c, void *const spec[9], float *x, float gs, float delta) {
  constexpr int E = xE<R>() < NX / 2 ? xE<R>() : NX / 2;
  constexpr int M = NX / 2, T = M / E;
  constexpr int BZ = xBZ<R>() * T <= 256 ? xBZ<R>() : (256 / T > 0 ? 256 / T : 1);
  typedef cx<R> C;
  const size_t smem = (size_t)(NX + (M + 1) * BZ + M * BZ) * sizeof(C);
  auto kern = xpass_c2r_features_kernel<R, NX, E, BZ>;
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  Fields<R> in{};
  for (int q = 0; q < 9; ++q) in.p[q] = (C *)spec[q];
  const int ts = timer_begin(c, GHOST_TIMER_X_C2R);
  kern<<<dim3(c->nz / BZ, c->ny), BZ * T, smem, c->stream>>>(in, x, (const C *)c->tw_x, c->ny, c->nz,
                                                              (R)(1.0 / (double)c->nreal), gs, delta);
  timer_end(c, ts);
  return post_launch(c);
}

template <typename R>
int grad9_features_dev(ghost_ctx *c, const void *const v[3], void *const spec[9], float *x, float gs, float delta) {
  ZGrad<R> zg{};
  for (int a = 0; a < 3; ++a) zg.v.p[a] = (const cx<R> *)v[a];
  for (int q = 0; q < 9; ++q) zg.w.p[q] = (cx<R> *)spec[q];
  zg.kp = kparams<R>(c);
  GB_CHECK(launch_z<R>(c, zg));
  Fields<R> fy{};
  for (int q = 0; q < 9; ++q) fy.p[q] = (cx<R> *)spec[q];
  GB_CHECK((launch_y<R, +1>(c, fy, 9)));
  if (xline_features_takes(c, x)) {
    const int ts = timer_begin(c, GHOST_TIMER_X_C2R);
    GB_CHECK(launch_xline_features(c, (const void *const *)spec, x, gs, delta));
    timer_end(c, ts);
    return post_launch(c);
  }
  switch (c->nx) {
    case 16: return grad9_features_n<R, 16>(c, spec, x, gs, delta);
    case 32: return grad9_features_n<R, 32>(c, spec, x, gs, delta);
    case 64: return grad9_features_n<R, 64>(c, spec, x, gs, delta);
    case 128: return grad9_features_n<R, 128>(c, spec, x, gs, delta);
    case 256: return grad9_features_n<R, 256>(c, spec, x, gs, delta);
    case 512: return grad9_features_n<R, 512>(c, spec, x, gs, delta);
    case 1024: return grad9_features_n<R, 1024>(c, spec, x, gs, delta);
  }
  return fail(GHOST_ERR_SIZE, "nx=%d unsupported", c->nx);
}

#define GB_INST(R)                                                                                                  \
  template int launch_x<R, X_HD>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);       \
  template int launch_x<R, X_BOUSS>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);    \
  template int launch_x<R, X_MHD>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);      \
  template int launch_x<R, X_NORM>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);     \
  template int launch_x<R, X_C2R>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);      \
  template int launch_x<R, X_R2C>(ghost_ctx *, const void *, void *, const void *const *, void *const *, int);      \
  template int grad9_features_dev<R>(ghost_ctx *, const void *const[3], void *const[9], float *, float, float);
GB_INST(float)
GB_INST(double)
#undef GB_INST

}  // namespace gb
