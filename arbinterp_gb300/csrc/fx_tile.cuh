// Bin-staged float64 evaluation in fixed point (included by sorted.cu).
//
// One CTA takes one bin (8^3 cells in 3D, 4^4 in 4D): its footprint of the
// float64 grid is read once, converted to the words of fx.cuh in units of the
// footprint's largest sample per field, and kept in shared memory, so the
// conversion (~20 operations a sample) is paid per tile point and not per query
// point (64 or 256), and the gather is shared-memory loads in the bin's bank
// schedule (placement writes the records of 16 bank classes round robin, see
// eval_binc_kernel) and not one L1 wavefront per lane.
//
// Scale.  Against the footprint's largest sample a result is off by 0.02 (3D)
// to 0.04 (4D) of 2^-53 before its rounding, a float64 evaluation by about 1 of
// 2^-53 of its own block's largest.  So the footprint's scale serves its bin
// where every cell has a corner within 2^-5 of the footprint's largest sample
// (a linear field through zero: 1/22 of it, 4D 1/14).  In the other bins
// (steep fields far from their peak) the tile keeps the float64 samples and
// every query sets the scale from its own cell's corners, converting as it
// reads.  A query that this does not hold either (FX_HEAD), and bins with
// samples outside the scaling, go to eval_otf3_slow / eval_otf4_slow; a query on a
// grid point takes its samples as they are (eval_node3, eval_otf4_slow).
#pragma once

namespace arb {

// Bound by the IMAD.WIDE pipe (4 cycles a warp instruction and scheduler; 'both'
// takes 1332 of them a query, half of its cycles at 305 queries a bin) and by the
// dependent issue of its chains at 12 to 16 warps per SM.  Three CTAs of 128
// threads and 168 registers for 'both' (four of 128 with spills 3222 against 3097 us
// for the binned pass of 1e7 on 256^3; 96, 160, 192 or 256 threads were 5-11 % slower).
constexpr int FX_THREADS = 128;
constexpr int FX_EVEN3 = 5, FX_EVEN4 = 5;

template <int F>
struct FxTile3;
template <>
struct FxTile3<4> {  // words (h, l) of fields 0, 1 and of fields 2, 3: 16-byte loads
  int4 a[TILE_PTS], b[TILE_PTS];
};
template <>
struct FxTile3<3> {
  int4 a[TILE_PTS];
  int2 c[TILE_PTS];
};
template <>
struct FxTile3<1> {
  int2 c[TILE_PTS];
};

// Point e of a tile as F pairs of words (raw: high and low word of the float64).
template <int F>
__device__ __forceinline__ void fx_tile_put(FxTile3<F> &t, int e, const int h[F], const int l[F]) {
  if constexpr (F >= 3) t.a[e] = make_int4(h[0], l[0], h[1 % F], l[1 % F]);
  if constexpr (F == 4) t.b[e] = make_int4(h[2], l[2], h[3], l[3]);
  if constexpr (F == 3) t.c[e] = make_int2(h[2], l[2]);
  if constexpr (F == 1) t.c[e] = make_int2(h[0], l[0]);
}
template <int F>
__device__ __forceinline__ void fx_tile_get(const FxTile3<F> &t, int e, int h[F], int l[F]) {
  if constexpr (F >= 3) {
    const int4 a = t.a[e];
    h[0] = a.x;
    l[0] = a.y;
    h[1 % F] = a.z;
    l[1 % F] = a.w;
  }
  if constexpr (F == 4) {
    const int4 b = t.b[e];
    h[2 % F] = b.x;
    l[2 % F] = b.y;
    h[3 % F] = b.z;
    l[3 % F] = b.w;
  }
  if constexpr (F == 3) {
    const int2 c = t.c[e];
    h[2 % F] = c.x;
    l[2 % F] = c.y;
  }
  if constexpr (F == 1) {
    const int2 c = t.c[e];
    h[0] = c.x;
    l[0] = c.y;
  }
}

template <int F>
struct FxTileSrc3 {
  const FxTile3<F> *t;
  int base;  // tile index of the block corner
  __device__ __forceinline__ void point(int i, int j, int k, int h[F], int l[F]) const {
    fx_tile_get<F>(*t, base + (k * TILE_EDGE + j) * TILE_EDGE + i, h, l);
  }
};

// The same tile holding float64 words (h high, l low), scaled per query.
template <int F>
struct FxRawSrc3 {
  const FxTile3<F> *t;
  int base;
  int emax[F];
  mutable uint32_t over[F];
  __device__ __forceinline__ void raw(int i, int j, int k, int hi[F], int lo[F]) const {
    fx_tile_get<F>(*t, base + (k * TILE_EDGE + j) * TILE_EDGE + i, hi, lo);
  }
  __device__ __forceinline__ void point(int i, int j, int k, int h[F], int l[F]) const {
    int hi[F], lo[F];
    raw(i, j, k, hi, lo);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      over[f] = max(over[f], (uint32_t)hi[f] & 0x7fffffffu);
      fx_sample(fx_pair((uint32_t)lo[f], (uint32_t)hi[f]), emax[f], h[f], l[f]);
    }
  }
  __device__ __forceinline__ bool fit() const {
    bool ok = true;
#pragma unroll
    for (int f = 0; f < F; ++f) ok &= fx_fits(over[f], emax[f]);
    return ok;
  }
  __device__ __forceinline__ bool scale() {
    FxMax m[F];
#pragma unroll 1
    for (int k = 1; k < 3; ++k)
#pragma unroll
      for (int j = 1; j < 3; ++j)
#pragma unroll
        for (int i = 1; i < 3; ++i) {
          int hi[F], lo[F];
          raw(i, j, k, hi, lo);
#pragma unroll
          for (int f = 0; f < F; ++f) m[f].add((uint32_t)hi[f], (uint32_t)lo[f]);
        }
    bool ok = true;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      ok &= m[f].corners(emax[f]);
      over[f] = 0;
    }
    return ok;
  }
};

// Largest samples of the tile, per field, gathered by the CTA.
template <int F>
struct FxTileMax {
  uint32_t m[F], z[F];
};

template <int F>
__device__ __forceinline__ void fx_merge_max(FxTileMax<F> &s, const FxMax v[F]) {
#pragma unroll
  for (int f = 0; f < F; ++f) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, v[f].m), z = __reduce_or_sync(0xffffffffu, v[f].z);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&s.m[f], m);
      atomicOr(&s.z[f], z);
    }
  }
}

// Exponents of the tile's fields; false where one is outside the scaling.
template <int F>
__device__ __forceinline__ bool fx_tile_exponents(const FxTileMax<F> &s, int emax[F]) {
  bool ok = true;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    FxMax v;
    v.m = s.m[f];
    v.z = s.z[f];
    ok &= v.exponent(emax[f]);
  }
  return ok;
}

// Bit o .. o + 31 of a bit string.
__device__ __forceinline__ uint32_t fx_bits_at(const uint32_t *w, int o) {
  return __funnelshift_r(w[o >> 5], w[(o >> 5) + 1], o & 31);
}

template <int F>
__global__ void __launch_bounds__(FX_THREADS, F == 4 ? 3 : 4) eval_fx3_kernel(arb_grid g, KParams kp, BinGeom bg,
                                                                              int64_t nq, arb_query_out o,
                                                                              SortedWork w, uint32_t share) {
  extern __shared__ __align__(16) unsigned char fx_smem[];
  FxTile3<F> &tile = *reinterpret_cast<FxTile3<F> *>(fx_smem);
  __shared__ FxTileMax<F> smax;
  __shared__ uint32_t large_bits[F][(TILE_PTS + FX_THREADS) / 32 + 1];
  const QRec64<3> *recs = reinterpret_cast<const QRec64<3> *>(w.rec);
  const int64_t nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const BinItems items(w, bg, share);
  for (uint32_t it = blockIdx.x; it < items.n; it += gridDim.x) {
    uint32_t t0, t1;
    const uint32_t b = (uint32_t)items.get(it, t0, t1), nb0 = (uint32_t)bg.nb[0], nb1 = (uint32_t)bg.nb[1],
                   r = b / nb0;
    if (t0 == t1) continue;
    const int og[3] = {(int)((b % nb0) * BIN_EDGE), (int)((r % nb1) * BIN_EDGE), (int)((r / nb1) * BIN_EDGE)};
    if (threadIdx.x < F) smax.m[threadIdx.x] = smax.z[threadIdx.x] = 0;
    // the footprint in registers (all loads in flight at once), its largest
    // samples, then its words in shared memory
    const double *corner = g.grid64 + ((og[2] * ny + og[1]) * nx + og[0]) * F;
    const int mx = (int)min((int64_t)TILE_EDGE, nx - og[0]), my = (int)min((int64_t)TILE_EDGE, ny - og[1]),
              mz = (int)min((int64_t)TILE_EDGE, nz - og[2]);
    const int64_t sy = nx * F, sz = nx * ny * F;
    constexpr int PER = (TILE_PTS + FX_THREADS - 1) / FX_THREADS;
    uint32_t lo[PER][F], hi[PER][F];
    bool in[PER];
    FxMax vm[F];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int e = threadIdx.x + m * FX_THREADS;
      const int lx = e % TILE_EDGE, rr = e / TILE_EDGE, ly = rr % TILE_EDGE, lz = rr / TILE_EDGE;
      in[m] = lx < mx && ly < my && lz < mz;
      if (in[m]) {  // points outside the grid: no cell of the bin reads them
        fx_read<F>(corner + lz * sz + ly * sy + lx * F, lo[m], hi[m]);
      } else {
#pragma unroll
        for (int f = 0; f < F; ++f) lo[m][f] = hi[m][f] = 0;
      }
    }
#pragma unroll
    for (int m = 0; m < PER; ++m)
#pragma unroll
      for (int f = 0; f < F; ++f) vm[f].add(hi[m][f], lo[m][f]);
    __syncthreads();  // smax is clear; the previous bin's queries are done with the tile
    fx_merge_max<F>(smax, vm);
    __syncthreads();
    int emax[F];
    const bool ok = fx_tile_exponents<F>(smax, emax);
    // which points are within 2^-FX_EVEN3 of the largest: one bit each, in tile
    // order (a warp holds 32 consecutive points), then every cell's corners
    bool bad = false;
    if (ok) {
      uint32_t least[F];  // of a large point: its high word without the sign, times 2
#pragma unroll
      for (int f = 0; f < F; ++f) least[f] = (smax.m[f] | smax.z[f]) ? (uint32_t)(emax[f] - FX_EVEN3 + 1) << 21 : 0u;
#pragma unroll
      for (int m = 0; m < PER; ++m)
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const bool large = hi[m][f] << 1 >= least[f] || !in[m];
          const uint32_t v = __ballot_sync(0xffffffffu, large);
          if ((threadIdx.x & 31) == 0) large_bits[f][m * (FX_THREADS / 32) + threadIdx.x / 32] = v;
        }
      __syncthreads();
      if (threadIdx.x < BIN_EDGE * BIN_EDGE) {
        const int r = (threadIdx.x / BIN_EDGE + 1) * TILE_EDGE + threadIdx.x % BIN_EDGE + 1;  // row y + 1, z + 1
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const uint32_t v = fx_bits_at(large_bits[f], r * TILE_EDGE) | fx_bits_at(large_bits[f], (r + 1) * TILE_EDGE) |
                             fx_bits_at(large_bits[f], (r + TILE_EDGE) * TILE_EDGE) |
                             fx_bits_at(large_bits[f], (r + TILE_EDGE + 1) * TILE_EDGE);
          bad |= (((v | v >> 1) >> 1) & 0xffu) != 0xffu;
        }
      }
    }
    const bool uneven = __syncthreads_or(bad);
    if (ok) {
#pragma unroll
      for (int m = 0; m < PER; ++m) {
        const int e = threadIdx.x + m * FX_THREADS;
        int h[F], l[F];
#pragma unroll
        for (int f = 0; f < F; ++f) {
          if (uneven) {
            h[f] = (int)hi[m][f];
            l[f] = (int)lo[m][f];
          } else {
            fx_sample(fx_pair(lo[m][f], hi[m][f]), emax[f], h[f], l[f]);
          }
        }
        if (e < TILE_PTS) fx_tile_put<F>(tile, e, h, l);
      }
    }
    __syncthreads();
    // the next record is loaded while this one is evaluated
    QRec64<3> next;
    const uint32_t first = t0 + threadIdx.x;
    if (first < t1) next = recs[first];
    for (uint32_t t = first; t < t1; t += FX_THREADS) {
      const QRec64<3> q = next;
      if (t + FX_THREADS < t1) next = recs[t + FX_THREADS];
      int64_t c[3];
      cell_coords<3>((int64_t)rec64_cell<3>(q), g, c);
      const double fr[3] = {rec64_frac<3>(q, 0), rec64_frac<3>(q, 1), rec64_frac<3>(q, 2)};
      double val[F], grad[3] = {0.0, 0.0, 0.0};
      const int base = (((int)c[2] - og[2]) * TILE_EDGE + ((int)c[1] - og[1])) * TILE_EDGE + ((int)c[0] - og[0]);
      bool fine = ok && !at_node<3>(fr);
      if (fine) {
        FxW wx, wy, wz;
        fx_axis<1>(fx_bits(fr[0]), wx);
        fx_axis<1>(fx_bits(fr[1]), wy);
        fx_axis<1>(fx_bits(fr[2]), wz);
        auto eval = [&](const auto &src, long long R[F], long long G[3]) {
          // z weights from shared memory: 'both' 3215 -> 3097 us (with y's too 3092), scalar 1e6 on
          // 101 x 87 x 93 154 -> 147; three components 818 -> 835, so those keep registers
          if constexpr (F != 3)
            fx_eval3<F>(src, wx, wy, FxZ(), R, G);
          else
            fx_eval3<F>(src, wx, wy, wz, R, G);
        };
        if constexpr (F != 3) FxZ::set(0, wz);
        long long R[F], G[3];
        if (!uneven) {
          FxTileSrc3<F> src;
          src.t = &tile;
          src.base = base;
          eval(src, R, G);
          fx_finish3<F>(R, G, emax, kp.inv_h, val, grad);
        } else {
          FxRawSrc3<F> src;
          src.t = &tile;
          src.base = base;
          fine = src.scale();
          if (fine) {
            eval(src, R, G);
            fx_finish3<F>(R, G, src.emax, kp.inv_h, val, grad);
            fine = src.fit();
          }
        }
      }
      if (!fine) {
        if (ok && at_node<3>(fr))  // the tile is finite: no scan of the block
          eval_node3<F>(g, c, kp.inv_h, val, grad);
        else
          eval_otf3_slow<F>(g, kp, c, fr, val, grad);
      }
      write_vals<3, F>(o, q.row, val, grad);
    }
  }
  // records that need no evaluation (out of volume, NaN, sentinel column)
  for (int64_t t = items.special(bg, nq) + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nq;
       t += (int64_t)gridDim.x * blockDim.x) {
    const QRec64<3> q = recs[t];
    write_const<3, F>(o, q.row, rec64_cell<3>(q) != NAN_CELL<3> && !g.sentinel_nan ? 0.0 : qnan());
  }
}

// 4D: a plane of words per field.
template <int F>
struct FxTile4 {
  int2 v[F][TILE4_PTS];
};

struct FxTileSrc4 {
  static constexpr int UNROLL = 4;
  const int2 *v;
  int base;
  __device__ __forceinline__ int at(int j, int k, int t) const {
    return base + ((t * TILE4_EDGE + k) * TILE4_EDGE + j) * TILE4_EDGE;
  }
  __device__ __forceinline__ void point(int i, int j, int k, int t, int *h, int *l) const {
    const int2 u = v[at(j, k, t) + i];
    *h = u.x;
    *l = u.y;
  }
};

struct FxRawSrc4 {
  static constexpr int UNROLL = 1;
  const int2 *v;
  int base;
  int emax;
  mutable uint32_t over;
  __device__ __forceinline__ int at(int j, int k, int t) const {
    return base + ((t * TILE4_EDGE + k) * TILE4_EDGE + j) * TILE4_EDGE;
  }
  __device__ __forceinline__ void point(int i, int j, int k, int t, int *h, int *l) const {
    const int2 u = v[at(j, k, t) + i];
    over = max(over, (uint32_t)u.x & 0x7fffffffu);
    fx_sample(fx_pair((uint32_t)u.y, (uint32_t)u.x), emax, *h, *l);
  }
  __device__ __forceinline__ bool fit() const { return fx_fits(over, emax); }
  __device__ __forceinline__ bool scale() {
    FxMax m;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int2 u = v[at(1 + ((c >> 1) & 1), 1 + ((c >> 2) & 1), 1 + (c >> 3)) + 1 + (c & 1)];
      m.add((uint32_t)u.x, (uint32_t)u.y);
    }
    over = 0;
    return m.corners(emax);
  }
};

// Two CTAs of up to 255 registers: three of 168 spill (1.5e6 scalar queries at 925
// a bin 1124 against 1069 us).
template <int F>
__global__ void __launch_bounds__(FX_THREADS, 2) eval_fx4_kernel(arb_grid g, KParams kp, BinGeom bg, int64_t nq,
                                                                 arb_query_out o, SortedWork w, uint32_t share) {
  extern __shared__ __align__(16) unsigned char fx_smem[];
  FxTile4<F> &tile = *reinterpret_cast<FxTile4<F> *>(fx_smem);
  __shared__ FxTileMax<F> smax;
  __shared__ uint32_t large_bits[F][(TILE4_PTS + 31) / 32 + 1];
  const QRec64<4> *recs = reinterpret_cast<const QRec64<4> *>(w.rec);
  const int64_t nx = g.n[0], ny = g.n[1], nz = g.n[2], nt = g.n[3];
  const BinItems items(w, bg, share);
  for (int64_t it = blockIdx.x; it < items.n; it += gridDim.x) {
    uint32_t t0, t1;
    const int64_t b = items.get(it, t0, t1);
    if (t0 == t1) continue;
    int64_t og[4];
    bin_origin4(b, bg, og);
    if (threadIdx.x < F) smax.m[threadIdx.x] = smax.z[threadIdx.x] = 0;
    __syncthreads();
    FxMax vm[F];
    for (int e = threadIdx.x; e < TILE4_PTS; e += FX_THREADS) {
      int r = e;
      const int64_t x = og[0] + r % TILE4_EDGE;
      r /= TILE4_EDGE;
      const int64_t y = og[1] + r % TILE4_EDGE;
      r /= TILE4_EDGE;
      const int64_t z = og[2] + r % TILE4_EDGE, t = og[3] + r / TILE4_EDGE;
      const bool in = x < nx && y < ny && z < nz && t < nt;
      const uint2 *p = reinterpret_cast<const uint2 *>(g.grid64 + (((t * nz + z) * ny + y) * nx + x) * F);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const uint2 u = in ? __ldg(p + f) : make_uint2(0, 0);
        vm[f].add(u.y, u.x);
        tile.v[f][e] = make_int2((int)u.y, (int)u.x);
      }
    }
    fx_merge_max<F>(smax, vm);
    __syncthreads();
    int emax[F];
    const bool ok = fx_tile_exponents<F>(smax, emax);
    bool bad = false;
    if (ok) {
      for (int e = threadIdx.x; e < (TILE4_PTS + 31) / 32 * 32; e += FX_THREADS)
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const uint32_t hi = e < TILE4_PTS ? (uint32_t)tile.v[f][e].x : 0u;
          const bool large = (int)(hi >> 20 & 0x7ff) > emax[f] - FX_EVEN4 || !(smax.m[f] | smax.z[f]);
          const uint32_t v = __ballot_sync(0xffffffffu, large);
          if ((threadIdx.x & 31) == 0) large_bits[f][e / 32] = v;
        }
      __syncthreads();
      if (threadIdx.x < BIN4_EDGE * BIN4_EDGE * BIN4_EDGE) {
        const int cy = threadIdx.x % BIN4_EDGE, cz = threadIdx.x / BIN4_EDGE % BIN4_EDGE,
                  ct = threadIdx.x / (BIN4_EDGE * BIN4_EDGE);
        // cells past the grid's last do not count
        const int cells = (int)min((int64_t)BIN4_EDGE, nx - 3 - og[0]);
        const bool there = og[1] + cy < ny - 3 && og[2] + cz < nz - 3 && og[3] + ct < nt - 3;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          uint32_t v = 0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int r = ((ct + 1 + (c >> 2)) * TILE4_EDGE + cz + 1 + (c >> 1 & 1)) * TILE4_EDGE + cy + 1 + (c & 1);
            v |= fx_bits_at(large_bits[f], r * TILE4_EDGE);
          }
          const uint32_t want = (1u << cells) - 1u;
          bad |= there && (((v | v >> 1) >> 1) & want) != want;
        }
      }
    }
    const bool uneven = __syncthreads_or(bad);
    if (ok && !uneven) {
      for (int e = threadIdx.x; e < TILE4_PTS; e += FX_THREADS)
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const int2 u = tile.v[f][e];
          int2 v;
          fx_sample(fx_pair((uint32_t)u.y, (uint32_t)u.x), emax[f], v.x, v.y);
          tile.v[f][e] = v;
        }
    }
    __syncthreads();
    const uint32_t first = t0 + threadIdx.x;
    for (uint32_t t = first; t < t1; t += FX_THREADS) {
      const QRec64<4> q = recs[t];
      int64_t c[4];
      cell_coords<4>((int64_t)rec64_cell<4>(q), g, c);
      const double fr[4] = {rec64_frac<4>(q, 0), rec64_frac<4>(q, 1), rec64_frac<4>(q, 2), rec64_frac<4>(q, 3)};
      double val[F], grad[4] = {0.0, 0.0, 0.0, 0.0};
      const bool node = at_node<4>(fr);
      FxW wt[2];
      fx_weights4(fr, wt);
      const int base = (int)((((c[3] - og[3]) * TILE4_EDGE + (c[2] - og[2])) * TILE4_EDGE + (c[1] - og[1])) * TILE4_EDGE +
                             (c[0] - og[0]));
      // field f in the tile's scale or its own; false: neither holds it
      auto contract = [&](auto gradf, int f, double &v, double gr[4]) {
        constexpr bool GRADF = decltype(gradf)::value;
        if (!ok || node) return false;
        long long R, G[4];
        int e = emax[0];
        bool fine = true;
        if (!uneven) {
#pragma unroll
          for (int m = 1; m < F; ++m) e = m == f ? emax[m] : e;
          FxTileSrc4 src;
          src.v = tile.v[f];
          src.base = base;
          fx_eval4<GRADF>(src, wt, FxZT(), R, G);
        } else {
          FxRawSrc4 src;
          src.v = tile.v[f];
          src.base = base;
          if (!src.scale()) return false;
          fx_eval4<GRADF>(src, wt, FxZT(), R, G);
          fine = src.fit();
          e = src.emax;
        }
        v = fx_to_double(R, e);
        if (GRADF) {
#pragma unroll
          for (int a = 0; a < 4; ++a) gr[a] = fx_to_double(G[a], e + 2) * kp.inv_h[a];
        }
        return fine;
      };
      constexpr int NV = F == 3 ? 3 : F - 1;  // value-only fields come first
#pragma unroll 1
      for (int f = 0; f < NV; ++f) {
        double v = 0.0, none[4];
        if (!contract(std::false_type(), f, v, none)) eval_otf4_slow<false>(g, kp, F, f, c, fr, v, none, ok);
#pragma unroll
        for (int m = 0; m < NV; ++m)
          if (m == f) val[m] = v;
      }
      if constexpr (F != 3) {
        if (!contract(std::true_type(), F - 1, val[F - 1], grad))
          eval_otf4_slow<true>(g, kp, F, F - 1, c, fr, val[F - 1], grad, ok);
      }
      write_vals<4, F>(o, q.row, val, grad);
    }
    __syncthreads();
  }
  for (int64_t t = items.special(bg, nq) + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nq;
       t += (int64_t)gridDim.x * blockDim.x) {
    const QRec64<4> q = recs[t];
    write_const<4, F>(o, q.row, rec64_cell<4>(q) != NAN_CELL<4> && !g.sentinel_nan ? 0.0 : qnan());
  }
}

// Resident grid of a persistent kernel (cached per device); 0 when it cannot run.
template <class K>
static int64_t fx_grid(K kernel, size_t smem, int per_sm[MAX_DEVICES]) {
  const int dev = current_device();
  if (dev < 0) return 0;
  if (!per_sm[dev]) {
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, FX_THREADS, smem) != cudaSuccess || n < 1)
      return 0;
    per_sm[dev] = n;
  }
  return (int64_t)device_sms() * per_sm[dev];
}

template <int DIM, int F>
static bool launch_eval_fx_f(const arb_grid *g, const KParams &kp, const BinGeom &bg, int64_t nq,
                             const arb_query_out *out, const SortedWork &w, cudaStream_t s) {
  static int per_sm[MAX_DEVICES] = {};
  const uint32_t share = bin_share(bg.nbins, nq);
  const int64_t items = bg.nbins + nq / share;  // at most
  if constexpr (DIM == 3) {
    int64_t grid = fx_grid(eval_fx3_kernel<F>, sizeof(FxTile3<F>), per_sm);
    if (!grid) return false;
    if (grid > items) grid = items;
    eval_fx3_kernel<F><<<(unsigned)grid, FX_THREADS, sizeof(FxTile3<F>), s>>>(*g, kp, bg, nq, *out, w, share);
  } else {
    int64_t grid = fx_grid(eval_fx4_kernel<F>, sizeof(FxTile4<F>), per_sm);
    if (!grid) return false;
    if (grid > items) grid = items;
    eval_fx4_kernel<F><<<(unsigned)grid, FX_THREADS, sizeof(FxTile4<F>), s>>>(*g, kp, bg, nq, *out, w, share);
  }
  return true;
}

// Launches the bin-staged float64 kernel when it applies (bins of the tile's
// shape with bank classes, and enough queries); returns false otherwise.
// A tile costs its bin 5.4e3 (F = 4) conversions however many queries it has;
// below the line (fx_dense) the queries are evaluated in bin order from the
// grid (eval_sorted_kernel).  Whole passes, tile against that: 'both' 256^3 at 30
// queries a bin 1308 : 590 us and at 305 3276 : 4613 us; norm 128^3 at 244 219 : 236
// and at 122 145 : 134; vector 128^3 at 49 125 : 115 and at 244 252 : 377; 4D
// scalar at 89 294 : 272 and at 670 1130 : 1701.
template <int DIM>
static bool launch_eval_fx(const arb_grid *g, const KParams &kp, const BinGeom &bg, int64_t nq,
                           const arb_query_out *out, const SortedWork &w, cudaStream_t s) {
  if (bg.cls != 4) return false;
  switch (g->nfield) {
    case 1: return launch_eval_fx_f<DIM, 1>(g, kp, bg, nq, out, w, s);
    case 3: return launch_eval_fx_f<DIM, 3>(g, kp, bg, nq, out, w, s);
    default: return launch_eval_fx_f<DIM, 4>(g, kp, bg, nq, out, w, s);
  }
}

}  // namespace arb
