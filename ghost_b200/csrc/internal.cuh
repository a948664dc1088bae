// internal.cuh -- device-path entry points of api.cu shared with the other
// translation units of the library (les.cu).  Explicit instantiations for
// float and double live at the end of api.cu's gb namespace.
#pragma once
#include <cudaTypedefs.h>

#include <algorithm>
#include <utility>

#include "common.cuh"
#include "passes.cuh"

namespace gb {

int dalloc(void **p, size_t bytes);
// scratch spectral fields 0..n-1 of the context (each cbytes); the 3D
// transforms and substeps below use them, so callers keep their own
// buffers for anything that must survive a call
int scratch(ghost_ctx *c, int n, void **out);
int post_launch(ghost_ctx *c);
int check_status(ghost_ctx *c);
bool is_device_ptr(const void *p);
int grid1d(size_t n);

template <typename R> const KParams<R> &kparams(const ghost_ctx *c);
// unnormalised 3D transforms on device arrays (c2r keeps its input)
template <typename R> int r2c_dev(ghost_ctx *c, const void *in, void *out);
template <typename R> int c2r_dev(ghost_ctx *c, const void *in, void *out);
// the LES closure's input rows x[q][10] (gradients times gs, delta) of a
// spectral velocity, through spectral work fields spec[9]
template <typename R>
int grad9_features_dev(ghost_ctx *c, const void *const v[3], void *const spec[9], float *x, float gs, float delta);
// six real fields to spectra (x per field, one y and one z pass for all six)
template <typename R> int r2c6_dev(ghost_ctx *c, const void *const in[6], void *const out[6]);
// one fused HD substep (include/hd_rkstep2.f90; hd_rkstep1 folded in with copy)
template <typename R>
int hd_substep_dev(ghost_ctx *c, int o, double dt, double nu, void *const v[3], void *const C[3], const void *const f[3],
                   int copy, bool prune = false);
// E of the X and Z passes and z-values of an X tile
template <typename R> constexpr int xE() { return sizeof(R) == 4 ? 8 : 4; }
template <typename R> constexpr int xBZ() { return sizeof(R) == 4 ? 8 : 4; }

template <typename R> constexpr int zE() { return sizeof(R) == 4 ? 8 : 4; }

// Pruning state for one substep: null tables = every line.
struct Prune {
  const int *lines = nullptr;
  int nlines = 0;
  const int *jpos = nullptr, *jneg = nullptr;
  int ni = 0;    // kx indices processed by the y passes
  int rows = 0;  // kx rows present in / written by the x pass
};

// X pass kinds
enum XKind { X_HD = 0, X_C2R = 1, X_R2C = 2, X_BOUSS = 3, X_MHD = 4, X_NORM = 5 };

// the passes: Op of passes.cuh over z-lines; nf fields along y (in place);
// an X pass of kind KIND (in, out: the plain transforms; ins, outs: the fused
// ones, whose output fields may be any of the inputs that a tile has consumed)
template <typename R, class Op> int launch_z(ghost_ctx *c, const Op &op, const Prune &pr = Prune());
template <typename R, int S> int launch_y(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr = Prune());
template <typename R, int KIND>
int launch_x(ghost_ctx *c, const void *in, void *out, const void *const *ins = nullptr, void *const *outs = nullptr,
             int rows = 0);
// what a tile variant chooses for an HD step: the z passes' rings, and whether
// the y passes have a choice (bit 0)
template <typename R> int hd_z_rings(const ghost_ctx *c, int cfg);
template <typename R> bool y_wide_choice(const ghost_ctx *c);
int encode_fn(PFN_cuTensorMapEncodeTiled_v12000 *fn);
int sm_count(ghost_ctx *c);
// Persistent grid: as many CTAs as fit on the device at once, or fewer
// when there are fewer tiles.
template <class K> int persistent_grid(ghost_ctx *c, K kern, int threads, size_t smem, long ntiles) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (per_sm < 1) per_sm = 1;
  const long g = (long)per_sm * sm_count(c);
  return (int)std::max<long>(1, std::min<long>(g, ntiles));
}
// Launch of a pass over nf fields whose kernel calls dep_wait (pipeline.cuh).
// A small pass starts its prologue (barriers, twiddles) while the kernel before
// it in the stream ends, instead of after the launch latency: a 256 x 128 x 64
// FP64 transform pair took 60 us without and 48 us with, a 128^3 FP32 closure
// step 1697 and 1623.  Large ones are slower for it (256^3 FP64 step: 4055 us
// without, 4236 with; 128^3 FP64 MHD: 905 and 945), so the attribute is left
// out above kDepBytes of input, for batched contexts (256 runs: 5758 and 6377),
// and for the classes of an ensemble, one-run ones too, whose streams share the
// GPU already (4 + 2 + 1 runs of 16^3, 32^3, 64^3 FP32: 162 without, 182 with).
// Neither do the passes over several fields gain with 16-point y lines, whose
// CTAs hold eight kx each: 256 x 16 x 64 FP32 HD 89 without and 99 with, 1024 x 16 x
// 16 FP64 118 and 134 (with 32 points, 1024 x 32 x 16 FP64: 160 and 145).
constexpr size_t kDepBytes = (size_t)64 << 20;
constexpr int kAlone = 1 << 20;  // as nf: a pass that starts when the one before it has ended
template <class... P, class... A>
int launch_dep(ghost_ctx *c, int nf, void (*kern)(P...), int grid, int block, size_t smem, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = c->nruns == 1 && !c->shares_gpu && (c->ny > 16 || nf == 1) && nf * c->cbytes <= kDepBytes ? 1 : 0;
  GB_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
  return GHOST_OK;
}
// TMA tensor map of a spectral field: a 3D tensor (z in 8-byte units, y, kx)
// over one field, with the box the pass moves
int field_map(ghost_ctx *c, const void *base, unsigned box0, unsigned box1, unsigned box2, CUtensorMap *out,
              CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_NONE);
PipeCtl pipe_ctl(ghost_ctx *c);
// the fused X pass with lines kept inside a warp (xnl.cuh): whether it
// takes this grid, and its launch (ins: v, curl v (, grad theta); rows: live
// kx rows, 0 for all)
bool xnl_takes(ghost_ctx *c);
int launch_xnl(ghost_ctx *c, bool bouss, const void *const *ins, void *const *outs, int rows);
// plain x transforms with lines kept inside a warp (xplain.cuh): whether they
// take this grid, and their launches
bool xline_takes(const ghost_ctx *c);
int launch_xline_r2c(ghost_ctx *c, const void *const *in, void *const *out, int nf);  // nf <= 12 fields
int launch_xline_c2r(ghost_ctx *c, const void *in, void *out);
bool xline_features_takes(const ghost_ctx *c, const void *x);
int launch_xline_features(ghost_ctx *c, const void *const *spec, float *x, float gs, float delta);
// the Y pass with lines kept inside a warp (ywarp.cuh)
template <typename R, int S> int launch_ywarp(ghost_ctx *c, const Fields<R> &f, int nf, const Prune &pr);
// FP64 partial sums owned by the context, grown on demand
int partials(ghost_ctx *c, size_t n, double **out);
// per-kernel timers around a launch (kind GHOST_TIMER_*)
int timer_begin(ghost_ctx *c, int kind);
void timer_end(ghost_ctx *c, int slot);
// out[b] = sum over q < nparts of part[q][b], in a fixed order
int finalize_dev(ghost_ctx *c, const double *part, int nparts, int nbins, double *out);
// reductions (reduce.cu; kinds of ops.cuh, kind 0: <|v|^2>) into host doubles:
// one kind, or the kinds of a mask in one pass over the fields
template <typename R>
int reduce_dev(ghost_ctx *c, int kind, const void *a, const void *b, const void *cc, const void *d, const void *e,
               const void *f, double *out_host);
template <typename R>
int sums_dev(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
             const void *f, double *out_host);
// shell spectra of the kinds of a mask, on the device without synchronising
// (shells_dev) or into host arrays
template <typename R>
int shells_dev(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
               const void *f, double *out_dev, R rnd, double *part = nullptr, int maxblk = 0, double **fin = nullptr);
template <typename R>
int shells_host(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
                const void *f, double *const *out_host, R rnd, double *part = nullptr, int maxblk = 0);

}  // namespace gb

namespace gb {
template <> const KParams<float> &kparams<float>(const ghost_ctx *c);
template <> const KParams<double> &kparams<double>(const ghost_ctx *c);
}  // namespace gb
