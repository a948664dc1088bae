// ywarp.cuh -- the Y pass with lines kept inside a warp.
//
// A tile is the live y rows x BZ z-values (128 bytes, SWIZZLE_128B; 64 bytes
// with SWIZZLE_64B for 1024-point lines) of one field at one kx.  A line of N
// values is held by T = N/E lanes of one warp, E values each, and transformed
// as R1 x R2 points (R1 = E): one exchange, in place.  A warp owns its
// z-columns of the tile, so the exchange needs __syncwarp only: value idx goes
// to row idx ^ ((idx/R1) & 7), which puts the lanes of a shared-memory phase on
// different banks both when it is written (idx = R1 t + r) and when it is
// read (idx = t + T e).  The result replaces the tile in natural order and
// leaves by TMA; three tiles are in the ring: one coming, one being
// transformed, one going.  The CTA meets once a tile.
// ms a launch against 16 values a thread, two exchanges and three barriers a
// tile: 1024 x 1024 x 256 Boussinesq y_inv 3.4 and 2.6; 512^3 plain 0.196 and
// 0.176.
#pragma once
#include "f32x2.cuh"
#include "passes.cuh"
#include "xnl.cuh"

namespace gb {

// 32 points as 4 x 8: columns m, m + 8, m + 16, m + 24, then rows of 8
template <int S, typename C> __device__ __forceinline__ void pdft32(C (&x)[32]) {
  // W32^q, q = 0..21 (m r for m < 8, r < 4)
  constexpr double c[22] = {1., 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                           0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                           0.19509032201612826785, 0., -0.19509032201612826785, -0.38268343236508977173,
                           -0.55557023301960222474, -0.70710678118654752440, -0.83146961230254523708,
                           -0.92387953251128675613, -0.98078528040323044913, -1., -0.98078528040323044913,
                           -0.92387953251128675613, -0.83146961230254523708, -0.70710678118654752440,
                           -0.55557023301960222474};
  constexpr double s[22] = {0., 0.19509032201612826785, 0.38268343236508977173, 0.55557023301960222474,
                           0.70710678118654752440, 0.83146961230254523708, 0.92387953251128675613,
                           0.98078528040323044913, 1., 0.98078528040323044913, 0.92387953251128675613,
                           0.83146961230254523708, 0.70710678118654752440, 0.55557023301960222474,
                           0.38268343236508977173, 0.19509032201612826785, 0., -0.19509032201612826785,
                           -0.38268343236508977173, -0.55557023301960222474, -0.70710678118654752440,
                           -0.83146961230254523708};
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    pdft4<S>(x[m], x[m + 8], x[m + 16], x[m + 24]);
    // x[m + 8 r] is output r of column m: times W32^(m r)
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      const int q = m * r;
      if (q == 0) continue;
      if (q == 4) x[m + 8 * r] = mulw8<S>(x[m + 8 * r]);
      else if (q == 8) x[m + 8 * r] = mul_si<S>(x[m + 8 * r]);
      else if (q == 12) x[m + 8 * r] = mulw83<S>(x[m + 8 * r]);
      else x[m + 8 * r] = cmulk<S>(x[m + 8 * r], c[q], s[q]);
    }
  }
  C y[32];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    C v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = x[8 * r + q];
    pdft8<S>(v);
#pragma unroll
    for (int q = 0; q < 8; ++q) y[r + 4 * q] = v[q];
  }
#pragma unroll
  for (int q = 0; q < 32; ++q) x[q] = y[q];
}

template <int Q, int S, typename C> __device__ __forceinline__ void pdftR(C (&v)[Q]) {
  if constexpr (Q == 32) pdft32<S>(v);
  else if constexpr (Q == 16) pdft16<S>(v);
  else pdft8<S>(v);
}

template <typename R, int N, int E, int BZ> struct YWarpGeom {
  static constexpr int ES = 2 * sizeof(R);
  static constexpr int T = N / E, R1 = E, R2 = N / R1, NB = E / R2;
  static constexpr int LW = 32 / T, NW = BZ / LW, NT = 32 * NW, RB = BZ * ES;
  static constexpr size_t tile = (size_t)N * RB;
  static constexpr int STAGES = 3;
  static constexpr size_t smem = STAGES * tile + (size_t)N * ES + 64;  // from a 1024-byte boundary on
  static_assert(R2 <= R1 && T >= 8 && T <= 32 && BZ % LW == 0, "R1 x R2 points, a line is 8 to 32 lanes");
};

// Rows a tile moves at a time: the pruned inverse loads, and the pruned forward
// pass stores, boxes of 32 rows that cover the live ones; all else in boxes of
// up to 256.
struct YWarpBoxes {
  int rb, rbo;
  YWarpBoxes(int n, bool pruned, int s)
      : rb(pruned && s > 0 ? 32 : (n < 256 ? n : 256)), rbo(pruned && s < 0 ? 32 : (n < 256 ? n : 256)) {}
};
// whether lines of N points are kept inside a warp
template <typename R> constexpr bool y_warp_line(int N) { return N >= 64 && N <= (sizeof(R) == 4 ? 1024 : 256); }

// One group of NT threads (the g-th of the CTA, shared memory from sm on):
// tiles vb, vb + nvb, ...  rb: rows of a load box, rbo: of a store box (both
// divide N).
template <typename R, int N, int E, int BZ, int S>
__device__ __forceinline__ void ywarp_body(int vb, int nvb, int g, unsigned char *sm, const FieldMaps &maps,
                                           const FieldMaps &omaps, const cx<R> *__restrict__ twg, int nzb, int ni, int nf,
                                           int nruns, int nxh, const int *__restrict__ jpos,
                                           const int *__restrict__ jneg, int rb, int rbo, PipeCtl ctl) {
  using C = cx<R>;
  using G = YWarpGeom<R, N, E, BZ>;
  constexpr bool F32 = sizeof(R) == 4;
  constexpr int T = G::T, R1 = G::R1, R2 = G::R2, NB = G::NB, LW = G::LW, RB = G::RB, STAGES = G::STAGES, U = G::ES / 8;
  // W_N^(b m): FP32 pairs (2j, 2j+1) of m, [j][b]; FP64 [m][b]
  C *tw = reinterpret_cast<C *>(sm + STAGES * G::tile);
  uint64_t *full = reinterpret_cast<uint64_t *>(tw + N), *never = full + STAGES;
  volatile int *failed = reinterpret_cast<int *>(never + 1);  // ring_wait
  const int tid = threadIdx.x - g * G::NT, lane = tid & 31, wp = tid >> 5;
  auto group_sync = [g] { named_sync(1 + g, G::NT); };
  // the lanes of a shared-memory phase: 8 t of the two lines of a 16-byte
  // chunk in FP32 (16 t of one line with T = 32), 8 t of one line in FP64
  int t, z;
  if constexpr (F32) {
    t = T == 32 ? lane : (lane >> 1) & (T - 1);
    z = T == 32 ? wp : wp * LW + (T == 16 ? lane & 1 : (lane & 1) + 2 * (lane >> 4));
  } else {
    t = lane & (T - 1);
    z = wp * LW + lane / T;
  }
  const int ntiles = nzb * ni * nruns * nf;
  dep_go();
  if (tid == 0) {
    mbar_init(never, 1);
    for (int q = 0; q < STAGES; ++q) mbar_init(&full[q], 1);
    *failed = 0;
    fence_barrier_init();
  }
  for (int q = tid; q < N; q += G::NT) {
    const int m = F32 ? 2 * (q / (2 * R1)) + (q & 1) : q / R1, b = F32 ? (q >> 1) % R1 : q % R1;
    tw[q] = twg[(b * m) % N];
  }
  group_sync();
  struct Tile {
    int zb, ii, i, f;  // ii: kx index within the run, i: its plane of the batched field
  };
  auto tile_of = [&](int tile) {
    Tile r;
    r.zb = tile % nzb;
    int q = tile / nzb;
    r.ii = q % ni;
    q /= ni;
    r.i = (q % nruns) * nxh + r.ii;
    r.f = q / nruns;
    return r;
  };
  // load k: boxes of rb rows covering [0, jp) from the top and [N - jn, N)
  // from the bottom (rows of a box beyond those are masked below)
  auto issue = [&](int k) {
    const int tile = vb + k * nvb;
    if (tile >= ntiles) return;
    const Tile tl = tile_of(tile);
    const int s = k % STAGES;
    int jp = N, jn = 0;
    if (jpos && S > 0) {
      jp = jpos[tl.ii];
      jn = jneg[tl.ii];
    }
    const int nt = (jp + rb - 1) / rb, nb = min((jn + rb - 1) / rb, N / rb - nt);
    fence_proxy_async();
    mbar_arrive_expect_tx(&full[s], (uint32_t)(nt + nb) * rb * RB);
    unsigned char *dst = sm + s * G::tile;
    for (int q = 0; q < nt; ++q) tma_load_3d(dst + (size_t)q * rb * RB, &maps.m[tl.f], tl.zb * BZ * U, q * rb, tl.i, &full[s]);
    for (int q = 0; q < nb; ++q) {
      const int r0 = N - (q + 1) * rb;
      tma_load_3d(dst + (size_t)r0 * RB, &maps.m[tl.f], tl.zb * BZ * U, r0, tl.i, &full[s]);
    }
  };
  dep_wait();
  if (tid == 0)
    for (int k = 0; k < STAGES - 1; ++k) issue(k);
  int issued = STAGES - 2;  // the last load asked for; it and the one before may be in flight
  // off[c]: byte offset of this lane's column in row (t & 7) ^ c of an 8-row group
  uint32_t off[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int u = (t & 7) ^ c;
    off[c] = !F32 ? (uint32_t)u * 128 + ((uint32_t)(z ^ u) << 4)
             : RB == 128 ? (uint32_t)u * 128 + ((uint32_t)((z >> 1) ^ u) << 4) + (uint32_t)(z & 1) * 8
                         : (uint32_t)u * 64 + ((uint32_t)((z >> 1) ^ ((u >> 1) & 3)) << 4) + (uint32_t)(z & 1) * 8;
  }
  const uint32_t trow = (uint32_t)(t & ~7) * RB, wrow = (uint32_t)(R1 * t) * RB;
  for (int k = 0;; ++k) {
    const int tile = vb + k * nvb;
    if (tile >= ntiles) break;
    const int s = k % STAGES;
    ring_wait(&full[s], (uint32_t)(k / STAGES) & 1u, never, ctl.stall && k == 0, ctl, failed);
    const Tile tl = tile_of(tile);
    int jp = N, jn = 0;
    if (jpos) {
      jp = jpos[tl.ii];
      jn = jneg[tl.ii];
    }
    unsigned char *tb = sm + s * G::tile;
    C x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      x[e] = *reinterpret_cast<const C *>(tb + trow + off[0] + (uint32_t)(T * e) * RB);
      if (S > 0) {
        const int jj = t + T * e;
        if (!(jj < jp || jj >= N - jn)) x[e] = mk((R)0, (R)0);
      }
    }
    __syncwarp();
    pdftR<R1, S>(x);
#pragma unroll
    for (int r = 0; r < R1; ++r)
      *reinterpret_cast<C *>(tb + wrow + off[r & 7] + (uint32_t)(r & ~7) * RB) = x[r];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e)
      x[e] = *reinterpret_cast<const C *>(tb + trow + off[(T * e / R1) & 7] + (uint32_t)(T * e) * RB);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      C v[R2];
#pragma unroll
      for (int m = 0; m < R2; ++m) v[m] = x[b + NB * m];
      if constexpr (F32) {
        const float4 *w = reinterpret_cast<const float4 *>(tw) + t + T * b;
#pragma unroll
        for (int j = 0; j < R2 / 2; ++j) {
          const float4 q = w[R1 * j];
          if (j > 0) v[2 * j] = twmul<S>(v[2 * j], mk(q.x, q.y));
          v[2 * j + 1] = twmul<S>(v[2 * j + 1], mk(q.z, q.w));
        }
      } else {
#pragma unroll
        for (int m = 1; m < R2; ++m) v[m] = twmul<S>(v[m], tw[R1 * m + t + T * b]);
      }
      pdftR<R2, S>(v);
#pragma unroll
      for (int r = 0; r < R2; ++r) x[b + NB * r] = v[r];
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) *reinterpret_cast<C *>(tb + trow + off[0] + (uint32_t)(T * e) * RB) = x[e];
    fence_proxy_async();
    group_sync();
    if (tid == 0 && !*failed) {
      // rows written: all of them, or (pruned forward pass) boxes covering the
      // live rows; the extra rows of a box hold the transform's own values, in
      // rows nothing reads
      if (S > 0 || !jpos) {
        for (int r0 = 0; r0 < N; r0 += rbo) tma_store_3d(&omaps.m[tl.f], tb + (size_t)r0 * RB, tl.zb * BZ * U, r0, tl.i);
      } else {
        const int nt = (jp + rbo - 1) / rbo, nb = min((jn + rbo - 1) / rbo, N / rbo - nt);
        for (int q = 0; q < nt; ++q) tma_store_3d(&omaps.m[tl.f], tb + (size_t)q * rbo * RB, tl.zb * BZ * U, q * rbo, tl.i);
        for (int q = 0; q < nb; ++q) {
          const int r0 = N - (q + 1) * rbo;
          tma_store_3d(&omaps.m[tl.f], tb + (size_t)r0 * RB, tl.zb * BZ * U, r0, tl.i);
        }
      }
      bulk_commit();
      // the store of the tile before this one has read its slot: refill it
      asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
      issue(k + STAGES - 1);
      issued = k + STAGES - 1;
    }
  }
  if (tid == 0) {
    if (*failed)
      for (int q = max(0, issued - 1); q <= issued && vb + q * nvb < ntiles; ++q)
        mbar_wait(&full[q % STAGES], (uint32_t)(q / STAGES) & 1u, kDrainPolls);
    bulk_wait_all();
  }
}

template <typename R, int N, int E, int BZ, int S, int MINB>
__global__ void __launch_bounds__(YWarpGeom<R, N, E, BZ>::NT, MINB)
    ywarp_kernel(const __grid_constant__ FieldMaps maps, const __grid_constant__ FieldMaps omaps,
                 const cx<R> *__restrict__ twg, int nzb, int ni, int nf, int nruns, int nxh,
                 const int *__restrict__ jpos, const int *__restrict__ jneg, int rb, int rbo, PipeCtl ctl) {
  extern __shared__ unsigned char smem_raw[];
  ywarp_body<R, N, E, BZ, S>(blockIdx.x, gridDim.x, 0, align1024(smem_raw), maps, omaps, twg, nzb, ni, nf, nruns, nxh, jpos,
                             jneg, rb, rbo, ctl);
}

}  // namespace gb
