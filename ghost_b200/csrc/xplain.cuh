// xplain.cuh -- plain x transforms and the LES closure's inputs with the
// warp-line tools of xnl.cuh (fftp3d_real_to_complex / fftp3d_complex_to_real,
// the x stage of fftp-3/fftp3D.fpp).
//
// A tile is BZ z-lines at one y; a line of NX real values is held by T lanes
// of one warp as M = NX/2 complex ones.  Persistent groups stream tiles through
// a ring of bulk copies; a slot is refilled by the last warp to read it.
//   r2c       real lines come in as they lie (line-major), the half spectrum
//             goes out by TMA from a swizzled kx-row tile;
//   c2r       kx-row tiles in, each lane stores its real pairs;
//   features  the nine gradients of a tile in turn, collected as the closure's
//             rows x[point][10] in shared memory and sent out line by line.
// Against one tile per block, real data scattered through shared memory and
// (features) rows written four bytes at a time: 256 x 128 x 64 FP64 r2c 16.5
// -> 8 us, inputs of a 128^3 closure 137 -> 53 us.
#pragma once
#include "xnl.cuh"

namespace gb {

template <typename R, int NX, int E, int BZ> struct XPlainGeom {
  using G = XnlGeom<R, NX, E, BZ, E>;
  // real lines: a phase's two lines (FP32, T < 32) or four (T = 4) start on other banks
  static constexpr int PITCH = G::M * G::ES + (sizeof(R) == 8 ? 16 : (G::T < 32 ? 64 : 0));
  static constexpr size_t line_tile = ((size_t)BZ * PITCH + 127) / 128 * 128;
  static constexpr size_t tables = G::NW * G::xch + (size_t)(G::M + G::TW2 + G::TW3) * G::ES + 256 + 1024;
  static constexpr size_t r2c(int st) { return st * line_tile + 2 * G::tile + tables; }
  static constexpr size_t c2r(int st) { return st * G::tile + tables; }
  static constexpr int ROWF = NX * 10 + 4;  // floats of a line's closure inputs
  static constexpr size_t feat(int st) { return st * G::tile + (size_t)BZ * ROWF * 4 + tables; }
};

// Ring bookkeeping of a group: bounded waits, refills by the last reader.
template <int STAGES, int NW> struct XRing {
  uint64_t *full, *never;
  unsigned *cnt;
  volatile int *failed;  // ring_wait
  __device__ __forceinline__ XRing(void *at, int tid) {
    full = reinterpret_cast<uint64_t *>(at);
    never = full + STAGES;
    cnt = reinterpret_cast<unsigned *>(never + 1);
    failed = reinterpret_cast<int *>(cnt + STAGES);
    if (tid == 0) {
      mbar_init(never, 1);
      for (int q = 0; q < STAGES; ++q) {
        mbar_init(&full[q], 1);
        cnt[q] = 0;
      }
      *failed = 0;
      fence_barrier_init();
    }
  }
  __device__ __forceinline__ bool wait(int L, const PipeCtl &ctl) const {
    return ring_wait(&full[L % STAGES], (uint32_t)(L / STAGES) & 1u, never, ctl.stall && L == 0, ctl, failed);
  }
  // every lane has read the slot of load L (alive: as ring_wait asks); true in
  // one lane of the group, which refills it
  __device__ __forceinline__ bool read(int L, int lane, bool alive) const {
    __syncwarp();
    return lane == 0 && alive && ring_read<STAGES, NW>(cnt, L);
  }
  // one thread at the end, per loads a tile of a CTA that takes every gridDim.x-th of ntiles
  __device__ __forceinline__ void drain(int per, int ntiles) const {
    if (*failed)
      ring_drain<STAGES, NW>(full, cnt, [&](int L) { return (int)(blockIdx.x + L / per * gridDim.x) < ntiles; });
  }
};

// nf fields in one launch: the six stresses of a 128^3 FP32 closure substep
// took 65 us one by one, 31 together
template <typename R, int NX, int E, int BZ, int STAGES>
__global__ void __launch_bounds__(XnlGeom<R, NX, E, BZ, E>::NT)
    xline_r2c_kernel(const __grid_constant__ CFields<R> in, const __grid_constant__ FieldMaps cmaps,
                     const cx<R> *__restrict__ twg, int ny, int nz, int nf, int nbox, int rb, PipeCtl ctl) {
  using C = cx<R>;
  using G = XnlGeom<R, NX, E, BZ, E>;
  using P = XPlainGeom<R, NX, E, BZ>;
  constexpr int M = G::M, T = G::T, RB = G::RB, U = G::ES / 8;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *sm = align1024(smem_raw);
  unsigned char *obuf = sm, *ibuf = sm + 2 * G::tile;
  const int tid = threadIdx.x, lane = tid & 31;
  dep_go();
  const XLine<R, NX, E, BZ> ln(tid, reinterpret_cast<C *>(ibuf + STAGES * P::line_tile), twg);
  const XRing<STAGES, G::NW> ring(ln.tw3 + G::TW3, tid);
  __syncthreads();
  const int nzb = nz / BZ, nft = nzb * ny, ntiles = nft * nf, bstep = rb & ~7;
  auto issue = [&](int k) {
    const int tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) return;
    const int s = k % STAGES, ft = tile % nft;
    const R *src = reinterpret_cast<const R *>(in.p[tile / nft]);
    fence_proxy_async();
    mbar_arrive_expect_tx(&ring.full[s], BZ * NX * (uint32_t)sizeof(R));
    for (int z = 0; z < BZ; ++z)
      bulk_g2s(ibuf + s * P::line_tile + (size_t)z * P::PITCH,
               src + (size_t)NX * ((size_t)(ft / nzb) + (size_t)ny * ((ft % nzb) * BZ + z)), NX * (uint32_t)sizeof(R),
               &ring.full[s]);
  };
  dep_wait();
  if (tid == 0)
    for (int k = 0; k < STAGES; ++k) issue(k);
  bool alive = true;  // no wait of this thread has run out
  for (int k = 0;; ++k) {
    const int tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) break;
    alive = alive && ring.wait(k, ctl);
    const C *src = reinterpret_cast<const C *>(ibuf + (k % STAGES) * P::line_tile + (size_t)ln.z * P::PITCH) + ln.t;
    C x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = src[T * e];
    if (ring.read(k, lane, alive)) issue(k + STAGES);
    ln.template fft<-1>(x);
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = mul2(x[e], both((R)0.5));  // store_unpacked gives twice the spectrum
    unsigned char *ob = obuf + (size_t)(k & 1) * G::tile;
    ln.template store_unpacked<E>(x, ob);
    fence_proxy_async();                 // the tile's generic writes, before the store reads them
    if (tid == 0) bulk_wait_read_all();  // the store before this one has read its buffer
    __syncthreads();
    if (tid == 0 && !*ring.failed) {
      const int ft = tile % nft;
      for (int q = 0; q < nbox; ++q) {
        const int r0 = min(q * bstep, M + 1 - rb);
        tma_store_3d(&cmaps.m[tile / nft], ob + (size_t)r0 * RB, (ft % nzb) * BZ * U, ft / nzb, r0);
      }
      bulk_commit();
    }
  }
  if (tid == 0) {
    ring.drain(1, ntiles);
    bulk_wait_all();
  }
}

template <typename R, int NX, int E, int BZ, int STAGES>
__global__ void __launch_bounds__(XnlGeom<R, NX, E, BZ, E>::NT)
    xline_c2r_kernel(const __grid_constant__ CUtensorMap cmap, R *__restrict__ out, const cx<R> *__restrict__ twg, int ny,
                     int nz, int nbox, int rb, PipeCtl ctl) {
  using C = cx<R>;
  using G = XnlGeom<R, NX, E, BZ, E>;
  constexpr int M = G::M, T = G::T, RB = G::RB, U = G::ES / 8;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *sm = align1024(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31;
  dep_go();
  const XLine<R, NX, E, BZ> ln(tid, reinterpret_cast<C *>(sm + STAGES * G::tile), twg);
  const XRing<STAGES, G::NW> ring(ln.tw3 + G::TW3, tid);
  __syncthreads();
  const int nzb = nz / BZ, ntiles = nzb * ny, bstep = rb & ~7;
  auto issue = [&](int k) {
    const int tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) return;
    const int s = k % STAGES;
    fence_proxy_async();
    mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(nbox * rb) * RB);
    for (int q = 0; q < nbox; ++q) {
      const int r0 = min(q * bstep, M + 1 - rb);
      tma_load_3d(sm + s * G::tile + (size_t)r0 * RB, &cmap, (tile % nzb) * BZ * U, tile / nzb, r0, &ring.full[s]);
    }
  };
  dep_wait();
  if (tid == 0)
    for (int k = 0; k < STAGES; ++k) issue(k);
  for (int k = 0;; ++k) {
    const int tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) break;
    if (!__all_sync(0xffffffffu, ring.wait(k, ctl))) break;
    C x[E];
    ln.template load_packed<E>(x, sm + (k % STAGES) * G::tile);
    if (ring.read(k, lane, true)) issue(k + STAGES);
    ln.template fft<+1>(x);
    C *row = reinterpret_cast<C *>(out + (size_t)NX * ((size_t)(tile / nzb) + (size_t)ny * ((tile % nzb) * BZ + ln.z))) + ln.t;
#pragma unroll
    for (int e = 0; e < E; ++e) row[T * e] = x[e];
  }
  __syncthreads();
  if (tid == 0) ring.drain(1, ntiles);
}

// x[q][3a+b] = (real value / (nx ny nz)) * gs of the nine fields, x[q][9] = delta
template <typename R, int NX, int E, int BZ, int STAGES>
__global__ void __launch_bounds__(XnlGeom<R, NX, E, BZ, E>::NT)
    xline_features_kernel(const __grid_constant__ FieldMaps maps, float *__restrict__ xrows,
                          const cx<R> *__restrict__ twg, int ny, int nz, int nbox, int rb, R inv_n, float gs, float delta,
                          PipeCtl ctl) {
  using C = cx<R>;
  using G = XnlGeom<R, NX, E, BZ, E>;
  using P = XPlainGeom<R, NX, E, BZ>;
  constexpr int M = G::M, T = G::T, RB = G::RB, U = G::ES / 8;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *sm = align1024(smem_raw);
  float *st = reinterpret_cast<float *>(sm + STAGES * G::tile);
  const int tid = threadIdx.x, lane = tid & 31;
  dep_go();
  const XLine<R, NX, E, BZ> ln(tid, reinterpret_cast<C *>(st + BZ * P::ROWF), twg);
  const XRing<STAGES, G::NW> ring(ln.tw3 + G::TW3, tid);
  for (int q = tid; q < BZ * NX; q += G::NT) st[(q / NX) * P::ROWF + (q % NX) * 10 + 9] = delta;  // stays from tile to tile
  __syncthreads();
  const int nzb = nz / BZ, ntiles = nzb * ny, bstep = rb & ~7;
  auto issue = [&](int L) {
    const int k = L / 9, f = L - 9 * k, tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) return;
    const int s = L % STAGES;
    fence_proxy_async();
    mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(nbox * rb) * RB);
    for (int q = 0; q < nbox; ++q) {
      const int r0 = min(q * bstep, M + 1 - rb);
      tma_load_3d(sm + s * G::tile + (size_t)r0 * RB, &maps.m[f], (tile % nzb) * BZ * U, tile / nzb, r0, &ring.full[s]);
    }
  };
  dep_wait();
  if (tid == 0)
    for (int L = 0; L < STAGES; ++L) issue(L);
  float *mine = st + ln.z * P::ROWF + 20 * ln.t;
  bool alive = true;  // no wait of this thread has run out
  for (int k = 0;; ++k) {
    const int tile = blockIdx.x + k * gridDim.x;
    if (tile >= ntiles) break;
#pragma unroll 1
    for (int f = 0; f < 9; ++f) {
      const int L = 9 * k + f;
      alive = alive && ring.wait(L, ctl);
      C x[E];
      ln.template load_packed<E>(x, sm + (L % STAGES) * G::tile);
      if (ring.read(L, lane, alive)) issue(L + STAGES);
      ln.template fft<+1>(x);
      if (f == 0) {  // the last tile's rows have left shared memory
        if (tid == 0) bulk_wait_read_all();
        __syncthreads();
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        mine[20 * T * e + f] = (float)(x[e].x * inv_n) * gs;
        mine[20 * T * e + 10 + f] = (float)(x[e].y * inv_n) * gs;
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0 && !*ring.failed) {
      for (int z = 0; z < BZ; ++z)
        bulk_s2g(xrows + (size_t)10 * NX * ((size_t)(tile / nzb) + (size_t)ny * ((tile % nzb) * BZ + z)), st + z * P::ROWF,
                 NX * 40);
      bulk_commit();
    }
  }
  if (tid == 0) {
    ring.drain(9, ntiles);
    bulk_wait_all();
  }
}

}  // namespace gb
