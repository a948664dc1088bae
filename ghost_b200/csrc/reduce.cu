// reduce.cu -- global sums and shell spectra of spectral fields
// (energy, helicity, cross, hdcheck, spectrumc, entrans, heltrans, ... of
// pseudo/pseudospec3D_hd.f90), deterministic, accumulated in FP64.
//
// All quantities asked for in one call are formed in one pass over the
// fields, so a call is bound by reading its fields once.  Wavenumbers come
// from the line a warp works on, not from dividing a flat mode index.
#include <algorithm>
#include <type_traits>

#include "internal.cuh"
#include "ops.cuh"

namespace gb {

constexpr int kKinds = RED_SC_VAR_K2 + 1;
__host__ __device__ constexpr int kinds_of(unsigned mask) {
  int n = 0;
  for (int q = 0; q < kKinds; ++q) n += (mask >> q) & 1;
  return n;
}
__host__ __device__ constexpr bool wants_bc(unsigned mask) {
  return (mask & ~((1u << RED_SC_CROSS) | (1u << RED_SC_VAR) | (1u << RED_SC_VAR_K2))) != 0;
}
__host__ __device__ constexpr bool wants_d(unsigned mask) {
  return (mask & ((1u << RED_CROSS) | (1u << RED_CROSS_K2) | (1u << RED_CURL_CROSS) | (1u << RED_SC_CROSS))) != 0;
}
__host__ __device__ constexpr bool wants_ef(unsigned mask) {
  return (mask & ((1u << RED_CROSS) | (1u << RED_CROSS_K2) | (1u << RED_CURL_CROSS))) != 0;
}

// the fields of mode p that the kinds of MASK read
template <unsigned MASK, typename R> __device__ __forceinline__ RedVals<R> red_load(const RedArgs<R> &ra, size_t p) {
  RedVals<R> v{};
  v.a = ra.a[p];
  if constexpr (wants_bc(MASK)) {
    v.b = ra.b[p];
    v.c = ra.c[p];
  }
  if constexpr (wants_d(MASK)) v.d = ra.d[p];
  if constexpr (wants_ef(MASK)) {
    v.e = ra.e[p];
    v.f = ra.f[p];
  }
  return v;
}
// acc[n] += w * term of the n-th kind of MASK; on != 0
template <unsigned MASK, int Q, int N, bool IN_R, typename R>
__device__ __forceinline__ void red_add(const KParams<R> &kp, const RedVals<R> &v, int i, int j, int k, R w, bool on,
                                        double *acc) {
  if constexpr (Q < kKinds) {
    if constexpr ((MASK >> Q) & 1) {
      const R t = red_value(kp, v, Q, i, j, k);
      // spectra weight the term in the working precision, sums in FP64
      const double x = IN_R ? (double)(w * t) : (double)w * (double)t;
      acc[N] += on ? x : 0.0;
      red_add<MASK, Q + 1, N + 1, IN_R>(kp, v, i, j, k, w, on, acc);
    } else {
      red_add<MASK, Q + 1, N, IN_R>(kp, v, i, j, k, w, on, acc);
    }
  }
}

// Sums over all modes: a warp takes z-lines (i, j) in turn, its lanes
// consecutive kz; partials[block][kind].
template <typename R, unsigned MASK>
__global__ void __launch_bounds__(256) sums_kernel(KParams<R> kp, RedArgs<R> ra, unsigned nlines, double *partials) {
  __shared__ double sh[32];
  constexpr int NK = kinds_of(MASK);
  double acc[NK];
#pragma unroll
  for (int q = 0; q < NK; ++q) acc[q] = 0.0;
  const int lane = threadIdx.x & 31;
  const unsigned nw = gridDim.x * (blockDim.x >> 5);
  for (unsigned L = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); L < nlines; L += nw) {
    const int j = (int)(L % (unsigned)kp.ny), i = (int)(L / (unsigned)kp.ny) % kp.nxh;
    const R w = i == 0 ? (R)1 : (R)2;
    const size_t base = (size_t)L * kp.nz;
#pragma unroll 4
    for (int k = lane; k < kp.nz; k += 32) {
      const RedVals<R> v = red_load<MASK>(ra, base + k);
      red_add<MASK, 0, 0, false>(kp, v, i, j, k, w, true, acc);
    }
  }
#pragma unroll
  for (int q = 0; q < NK; ++q) {
    const double s = block_sum(acc[q], sh);
    if (threadIdx.x == 0) partials[(size_t)blockIdx.x * NK + q] = s;
  }
}

// Shell spectra (spectrumc, pseudospec3D_hd.f90:1190-1415).  A warp takes
// the lines (i, j) and (i, ny - j); lane k adds the modes (+-ky, +-kz), which
// have one shell, and the shells do not decrease along the lanes.  So the
// lanes of a shell are neighbours: a segmented scan sums them in five
// shuffles and the last lane of each run adds the sum to the warp's own
// histogram, no two lanes to one slot.  Warps are combined in warp order and
// blocks in block order: reproducible bit for bit.
// Bound by reading the fields: energy and helicity of 512^3 FP32 fields
// are one pass over 1.6 GB; a kernel that summed each chunk of 32 modes by 32 rounds
// of shuffles took 1.2 ms for each of the two.
template <typename R, unsigned MASK>
__global__ void __launch_bounds__(256) shells_kernel(KParams<R> kp, RedArgs<R> ra, unsigned npairs, int nb, R Dkk, R rnd,
                                                     double *partials) {
  extern __shared__ double hist[];  // [warps][kinds][nb]
  constexpr int NK = kinds_of(MASK);
  const int nwb = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = threadIdx.x; q < nwb * NK * nb; q += blockDim.x) hist[q] = 0.0;
  __syncthreads();
  double *hw = hist + (size_t)w * NK * nb;
  const unsigned njp = (unsigned)kp.ny / 2 + 1, nw = gridDim.x * nwb;
  const int nzh = kp.nz / 2;
  auto shell_of = [&](int i, int j, int k) {
    const int kmn = (int)(sqrt(kk2_of(kp, i, j, k)) / Dkk + rnd);  // rnd: .501 rounding of the caller's GHOST routine
    return (kmn > 0 && kmn <= nb) ? kmn - 1 : -1;
  };
  for (unsigned P = blockIdx.x * nwb + w; P < npairs; P += nw) {
    const int j = (int)(P % njp), ib = (int)(P / njp), i = ib % kp.nxh;
    const bool two = j > 0 && 2 * j < kp.ny;  // ky = 0 and ny/2 have no mirror line
    const int j2 = two ? kp.ny - j : j;
    const R wgt = i == 0 ? (R)1 : (R)2;
    const size_t l1 = ((size_t)ib * kp.ny + j) * kp.nz, l2 = ((size_t)ib * kp.ny + j2) * kp.nz;
    for (int k0 = 0; k0 < nzh; k0 += 32) {
      const bool on = k0 + lane < nzh;
      const int k = on ? k0 + lane : nzh - 1, km = k > 0 ? kp.nz - k : 0;
      // all loads before any use (a mode without a mirror loads itself again)
      const RedVals<R> v0 = red_load<MASK>(ra, l1 + k), v1 = red_load<MASK>(ra, l1 + km),
                       v2 = red_load<MASK>(ra, l2 + k), v3 = red_load<MASK>(ra, l2 + km);
      double s[NK];
#pragma unroll
      for (int q = 0; q < NK; ++q) s[q] = 0.0;
      red_add<MASK, 0, 0, true>(kp, v0, i, j, k, wgt, on, s);
      red_add<MASK, 0, 0, true>(kp, v1, i, j, km, wgt, on && k > 0, s);
      red_add<MASK, 0, 0, true>(kp, v2, i, j2, k, wgt, on && two, s);
      red_add<MASK, 0, 0, true>(kp, v3, i, j2, km, wgt, on && two && k > 0, s);
      // lanes past the line's half continue the last shell with zeros
      const int bin = shell_of(i, j, k);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int bo = __shfl_up_sync(0xffffffffu, bin, o);
        const bool same = lane >= o && bo == bin;
#pragma unroll
        for (int q = 0; q < NK; ++q) {
          const double x = __shfl_up_sync(0xffffffffu, s[q], o);
          if (same) s[q] += x;
        }
      }
      const int bn = __shfl_down_sync(0xffffffffu, bin, 1);
      if (bin >= 0 && (lane == 31 || bn != bin)) {
#pragma unroll
        for (int q = 0; q < NK; ++q) hw[q * nb + bin] += s[q];
      }
      __syncwarp();
    }
    // kz = nz/2 has no mirror: lanes 0 and 1 take it on the two lines
    double s[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) s[q] = 0.0;
    if (lane < (two ? 2 : 1)) {
      const RedVals<R> v = red_load<MASK>(ra, (lane == 0 ? l1 : l2) + nzh);
      red_add<MASK, 0, 0, true>(kp, v, i, lane == 0 ? j : j2, nzh, wgt, true, s);
    }
    const int bin = shell_of(i, j, nzh);
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      const double x = __shfl_down_sync(0xffffffffu, s[q], 1);
      if (lane == 0 && bin >= 0) hw[q * nb + bin] += s[q] + x;
    }
    __syncwarp();
  }
  __syncthreads();
  for (int b = threadIdx.x; b < NK * nb; b += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < nwb; ++q) s += hist[(size_t)q * NK * nb + b];
    partials[(size_t)blockIdx.x * NK * nb + b] = s;
  }
}

// out[b] = sum over q of partials[q][b]: a block takes 32 columns, its warps
// every 32nd row in order, and the first warp the 32 sums in order.  (One
// block taking the bins one after the other took 0.5 ms for 257 bins.)
__global__ void __launch_bounds__(1024) finalize_kernel(const double *__restrict__ partials, int nparts, int nbins,
                                                        double *out) {
  __shared__ double sh[32][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x * 32 + lane;
  double a = 0.0;
  if (b < nbins)
    for (int q = w; q < nparts; q += 32) a += partials[(size_t)q * nbins + b];
  sh[w][lane] = a;
  __syncthreads();
  if (w == 0 && b < nbins) {
    double s = 0.0;
    for (int q = 0; q < 32; ++q) s += sh[q][lane];
    out[b] = s;
  }
}

int finalize_dev(ghost_ctx *c, const double *part, int nparts, int nbins, double *out) {
  finalize_kernel<<<(nbins + 31) / 32, 1024, 0, c->stream>>>(part, nparts, nbins, out);
  return post_launch(c);
}

template <typename R>
static RedArgs<R> red_args(const void *a, const void *b, const void *cc, const void *d, const void *e, const void *f) {
  return RedArgs<R>{(const cx<R> *)a, (const cx<R> *)b, (const cx<R> *)cc,
                    (const cx<R> *)d, (const cx<R> *)e, (const cx<R> *)f};
}

// one of the listed masks, or a failure
template <unsigned M, unsigned... Rest, class F> static int for_mask(unsigned mask, F f) {
  if (mask == M) return f(std::integral_constant<unsigned, M>{});
  if constexpr (sizeof...(Rest) > 0) return for_mask<Rest...>(mask, f);
  return fail(GHOST_ERR_STATE, "no reduction kernel for the kinds %u", mask);
}
#define B(k) (1u << (k))

// sums of the kinds of mask, in ascending order of kind, into out_host
template <typename R>
int sums_dev(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
             const void *f, double *out_host) {
  const unsigned nlines = (unsigned)((size_t)c->nxh * c->nruns * c->ny);
  const int nblk = (int)std::min<unsigned>((nlines + 7) / 8, 148 * 6);
  const int nk = kinds_of(mask);
  double *part;
  GB_CHECK(partials(c, (size_t)(nblk + 1) * nk, &part));
  const RedArgs<R> ra = red_args<R>(a, b, cc, d, e, f);
  const int ts = timer_begin(c, GHOST_TIMER_REDUCE);
  constexpr unsigned HD = B(RED_ENERGY) | B(RED_ENSTROPHY) | B(RED_CROSS);
  GB_CHECK((for_mask<B(RED_ENERGY), B(RED_ENSTROPHY), B(RED_LAPLACIAN), B(RED_HELICITY), B(RED_CROSS), B(RED_CROSS_K2),
                     B(RED_DIVERGENCE), B(RED_CURL_CROSS), B(RED_SC_CROSS), B(RED_SC_VAR), B(RED_SC_VAR_K2), HD,
                     HD | B(RED_HELICITY), HD | B(RED_DIVERGENCE), HD | B(RED_HELICITY) | B(RED_DIVERGENCE)>(
      mask, [&](auto m) {
        sums_kernel<R, m.value><<<nblk, 256, 0, c->stream>>>(kparams<R>(c), ra, nlines, part);
        return post_launch(c);
      })));
  double *fin = part + (size_t)nblk * nk;
  GB_CHECK(finalize_dev(c, part, nblk, nk, fin));
  timer_end(c, ts);
  GB_CUDA(cudaMemcpyAsync(out_host, fin, sizeof(double) * nk, cudaMemcpyDeviceToHost, c->stream));
  GB_CUDA(cudaStreamSynchronize(c->stream));
  return check_status(c);
}

template <typename R>
int reduce_dev(ghost_ctx *c, int kind, const void *a, const void *b, const void *cc, const void *d, const void *e,
               const void *f, double *out_host) {
  return sums_dev<R>(c, 1u << kind, a, b, cc, d, e, f, out_host);
}

// Shell spectra of the kinds of mask (ascending order of kind, nmax/2+1
// shells each) into out_dev, or (null) behind the partial sums, *fin saying
// where; part: room for (maxblk + 1) rows of kinds x shells, or null (the
// context's buffer).  rnd is the shell rounding: GHOST's
// spectra add the default-REAL literal .501 (0.501f), spectrscc adds shift +
// .501 in GP.
template <typename R>
int shells_dev(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
               const void *f, double *out_dev, R rnd, double *part, int maxblk, double **fin) {
  const int nb = c->nmax / 2 + 1, nk = kinds_of(mask);
  constexpr size_t kMostShared = 227 * 1024;
  if ((size_t)8 * nb * sizeof(double) > kMostShared)
    return fail(GHOST_ERR_CUDA, "%d shells exceed the shared-memory histograms", nb);
  // as many warps per block (8 at most) as leave three blocks on an SM
  int nw = 8;
  while (nw > 1 && (size_t)nw * nk * nb * sizeof(double) > 72 * 1024) nw /= 2;
  const size_t smem = (size_t)nw * nk * nb * sizeof(double);
  const unsigned npairs = (unsigned)((size_t)c->nxh * c->nruns * (c->ny / 2 + 1));
  const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(24 / nw, kMostShared / (smem + 1024)));
  int nblk = (int)std::min<unsigned>((npairs + nw - 1) / nw, 148u * per_sm);
  if (part) nblk = std::max(1, std::min(nblk, maxblk));
  else GB_CHECK(partials(c, (size_t)(nblk + 1) * nk * nb, &part));
  const RedArgs<R> ra = red_args<R>(a, b, cc, d, e, f);
  const int ts = timer_begin(c, GHOST_TIMER_REDUCE);
  GB_CHECK((for_mask<B(RED_ENERGY), B(RED_ENSTROPHY), B(RED_HELICITY), B(RED_CROSS), B(RED_CROSS_K2), B(RED_CURL_CROSS),
                     B(RED_SC_CROSS), B(RED_SC_VAR), B(RED_ENERGY) | B(RED_HELICITY),
                     B(RED_ENSTROPHY) | B(RED_HELICITY)>(mask, [&](auto m) {
    auto kern = shells_kernel<R, m.value>;
    GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<nblk, 32 * nw, smem, c->stream>>>(kparams<R>(c), ra, npairs, nb, (R)c->Dkk, rnd, part);
    return post_launch(c);
  })));
  if (!out_dev) out_dev = part + (size_t)nblk * nk * nb;
  if (fin) *fin = out_dev;
  GB_CHECK(finalize_dev(c, part, nblk, nk * nb, out_dev));
  timer_end(c, ts);
  return GHOST_OK;
}

// the same into host arrays, one per kind
template <typename R>
int shells_host(ghost_ctx *c, unsigned mask, const void *a, const void *b, const void *cc, const void *d, const void *e,
                const void *f, double *const *out_host, R rnd, double *part, int maxblk) {
  const int nb = c->nmax / 2 + 1, nk = kinds_of(mask);
  double *fin = nullptr;
  GB_CHECK(shells_dev<R>(c, mask, a, b, cc, d, e, f, nullptr, rnd, part, maxblk, &fin));
  for (int q = 0; q < nk; ++q)
    GB_CUDA(cudaMemcpyAsync(out_host[q], fin + (size_t)q * nb, sizeof(double) * nb, cudaMemcpyDeviceToHost, c->stream));
  GB_CUDA(cudaStreamSynchronize(c->stream));
  return GHOST_OK;
}
#undef B

#define GB_INST(R)                                                                                                     \
  template int sums_dev<R>(ghost_ctx *, unsigned, const void *, const void *, const void *, const void *, const void *, \
                           const void *, double *);                                                                    \
  template int reduce_dev<R>(ghost_ctx *, int, const void *, const void *, const void *, const void *, const void *,   \
                             const void *, double *);                                                                  \
  template int shells_dev<R>(ghost_ctx *, unsigned, const void *, const void *, const void *, const void *,            \
                             const void *, const void *, double *, R, double *, int, double **);                       \
  template int shells_host<R>(ghost_ctx *, unsigned, const void *, const void *, const void *, const void *,           \
                              const void *, const void *, double *const *, R, double *, int);
GB_INST(float)
GB_INST(double)
#undef GB_INST

}  // namespace gb
