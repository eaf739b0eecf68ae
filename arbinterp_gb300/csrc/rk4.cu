// Particle trajectories through a 3D interpolated field, fused on the device.
//
// The reference was written to simulate particle motion in magnetic fields
// and planned numerical integrators for it (CHANGELOG.md, v1.0.0); its users
// call Query in a Python loop, one round trip per stage.  Here one thread
// carries one particle through every step: classical fourth-order
// Runge-Kutta on
//     x' = v,   v' = coef * grad f(x) + gravity
// with f the interpolated scalar (scalar and norm modes) or |B| (both mode),
// e.g. coef = -mu/m for a weak-field seeker in a magnetic trap.  Each stage
// evaluates the interpolant on the fly (float64 or the float32 mixed path,
// as the interpolant's queries do).  A stage outside the interpolation
// volume, or on a cell index at or past nc (the upper faces), ends the
// particle: its state becomes NaN and it is counted in lost[0].
#include "eval.cuh"

namespace arb {

// |B| of a mixed 'both' grid as (hi, lo) pairs: the only field an integration
// reads, 8 bytes a point where the grid's rows take 16 and 4.
__global__ void __launch_bounds__(256) norm_pairs_kernel(const float *g32, int64_t npts, float2 *pairs) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p < npts) pairs[p] = make_float2(__ldg(g32 + 4 * p + 3), __ldg(g32 + 4 * npts + p));
}

// Sort key of each position (30 bits): particles of one warp then gather
// neighbouring grid points.  Non-finite rows sort last.  float32 is enough: the
// key orders the work, not the result.
// CELLS: 16-cell cubes in Z-order, inside a cube the x-rows of cells in Z-order
// over (y, z), inside a row x.  A load costs one L1 wavefront per line that its
// lanes touch, and a line is 16 points of one x-row: plain Z-order leaves 9.5
// lines a load at 7 particles a cell.  Whole calls, Z-order against this: 2e5 x 25
// steps on 128^3 1606 : 1350 us, 1e6 x 10 on 256^3 3364 : 2830.  A cloud that ends
// just past a row of cubes has a few warps with one cell of every row, though,
// and where an SM holds few warps the slowest one counts: 2e4 x 20 on 64^3 467 : 427
// or 449 : 559 us, 4e4 516 : 646.  So Z-order over the box (10 bits an axis)
// below CELLS_FROM particles: 77,824 are the 16 warps of every SM, and from 1.4e5 the
// x-rows win at most densities (10 steps, uniform in 0.6 of the box: 64^3 628 : 575,
// 128^3 673 : 590, 256^3 1313 : 1273; 1e6 2419 : 2316, 3025 : 2321, 3185 : 2588; a tight
// cloud 64^3 562 : 554, 128^3 652 : 588, 256^3 1022 : 917) and lose at most 6 % in
// the densest (1e6 in a cloud of 16 cells' width on 64^3: 2206 : 2341).
constexpr int64_t CELLS_FROM = 1 << 17;
__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v = (v | v << 16) & 0x030000ffu;
  v = (v | v << 8) & 0x0300f00fu;
  v = (v | v << 4) & 0x030c30c3u;
  return (v | v << 2) & 0x09249249u;
}
__device__ __forceinline__ uint32_t spread4(uint32_t v) {
  v = (v | v << 2) & 0x33u;
  return (v | v << 1) & 0x55u;
}
template <bool CELLS>
__global__ void __launch_bounds__(256) zorder_kernel(const double *state, int64_t n, double l0, double l1, double l2,
                                                     float s0, float s1, float s2, int32_t *keys) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double lo[3] = {l0, l1, l2};
  const float sc[3] = {s0, s1, s2};
  uint32_t c[3], key = 0;
  bool finite = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float d = (float)(state[i * 6 + a] - lo[a]) * sc[a];
    finite &= fabsf(d) < 1e30f;
    c[a] = (uint32_t)fminf(fmaxf(d, 0.f), 1023.f);
    key |= spread10(CELLS ? c[a] >> 4 : c[a]) << a;
  }
  if (CELLS) key = key << 12 | (spread4(c[1] & 15) | spread4(c[2] & 15) << 1) << 4 | (c[0] & 15);
  keys[i] = finite ? (int32_t)key : 1 << 30;
}

// Acceleration at x; false when x is outside the interpolation volume.  Only
// the last field (the scalar, or |B|) and its gradient are evaluated.
template <int F, bool MIXED, bool PAIRS>
__device__ __forceinline__ bool rk4_accel(const arb_grid &g, const KParams &kp, const float2 *pairs, const double x[3],
                                          double coef, const double grav[3], double a[3]) {
  using T = typename std::conditional<MIXED, float, double>::type;
  T fr[3];
  CoordStep s;
  if constexpr (MIXED)
    s = coord_step_fast<3>(x, kp.ax, g, fr);
  else
    s = coord_step_fx<3>(x, kp.ax, g, fr);
  if (s.oob || s.nan || s.idx >= g.nc) return false;
  int64_t c[3];
  cell_from_step<3>(s, g, c);
  double val[F], grad[3] = {0.0, 0.0, 0.0};
  if constexpr (MIXED && PAIRS) {
    NormBlock3 blk;
    blk.v = pairs;
    blk.sy = g.n[0];
    blk.sz = g.n[0] * g.n[1];
    blk.base = (c[2] * g.n[1] + c[1]) * g.n[0] + c[0];
    eval_otf3_both_block(blk, kp, fr, val, grad);
  } else if constexpr (MIXED) {
    eval_otf3<F, MIXED>(g, kp, c, fr, val, grad);
  } else {
    eval_otf3_fx<1, F>(g, kp, c, fr, val, grad);
  }
#pragma unroll
  for (int a_ = 0; a_ < 3; ++a_) a[a_] = coef * grad[a_] + grav[a_];
  return true;
}

// Bound by L1 gathers and latency: |B| pairs take 8 bytes a point where the
// 'both' grid takes 20, and 16 warps per SM (128 registers, a few spills) hide more
// than 8 (2e5 particles x 25 steps on 128^3 'both', whole call: 3.87 ms; keys in
// one kernel and no state copies, with pairs, 1.95; 16 warps 1.63).  float64: 13.7 ->
// 3.7 ms with |B| alone in fixed point.
template <int F, bool MIXED, bool PAIRS>
__global__ void __launch_bounds__(128, MIXED ? 4 : 3) rk4_kernel(arb_grid g, KParams kp, const float2 *pairs,
                                                                  const int64_t *order, double *state, int64_t n, double dt,
                                                  int64_t nsteps, double coef, double g0, double g1, double g2,
                                                  double *path, int64_t rec_every, unsigned long long *lost) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t i = order ? order[t] : t;  // the particle
  double *st = state + i * 6;
  double x[3] = {st[0], st[1], st[2]}, v[3] = {st[3], st[4], st[5]};
  const double grav[3] = {g0, g1, g2};
  const double h2 = 0.5 * dt, h6 = dt / 6.0;
  bool alive = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) alive &= (x[a] == x[a]) && (v[a] == v[a]);
  int64_t rec = 0;
  for (int64_t s = 0; s < nsteps && alive; ++s) {
    double k1v[3], k2v[3], k3v[3], k4v[3];
    // the four stages share one copy of the field evaluation (a rolled loop:
    // four inlined copies made instruction fetch the kernel's first stall)
#pragma unroll 1
    for (int stg = 0; stg < 4 && alive; ++stg) {
      double xs[3], k[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (stg == 0)
          xs[a] = x[a];
        else if (stg == 1)
          xs[a] = x[a] + h2 * v[a];
        else if (stg == 2)
          xs[a] = x[a] + h2 * (v[a] + h2 * k1v[a]);
        else
          xs[a] = x[a] + dt * (v[a] + h2 * k2v[a]);
      }
      alive = rk4_accel<F, MIXED, PAIRS>(g, kp, pairs, xs, coef, grav, k);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (stg == 0)
          k1v[a] = k[a];
        else if (stg == 1)
          k2v[a] = k[a];
        else if (stg == 2)
          k3v[a] = k[a];
        else
          k4v[a] = k[a];
      }
    }
    if (!alive) break;
    // position stages are v + dt/2 k1v, v + dt/2 k2v, v + dt k3v
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double dx = v[a] + (v[a] + h2 * k1v[a]) * 2.0 + (v[a] + h2 * k2v[a]) * 2.0 + (v[a] + dt * k3v[a]);
      x[a] += h6 * dx;
      v[a] += h6 * (k1v[a] + 2.0 * k2v[a] + 2.0 * k3v[a] + k4v[a]);
    }
    if (path && rec_every > 0 && (s + 1) % rec_every == 0) {
      double *r = path + (rec * n + i) * 6;
      for (int a = 0; a < 3; ++a) {
        r[a] = x[a];
        r[3 + a] = v[a];
      }
      ++rec;
    }
  }
  if (!alive) {
    const double nan = qnan();
    for (int a = 0; a < 3; ++a) x[a] = v[a] = nan;
    atomicAdd(lost, 1ULL);
    // the remaining recorded states of a lost particle are NaN as well
    if (path && rec_every > 0)
      for (int64_t r = rec; r < nsteps / rec_every; ++r)
        for (int a = 0; a < 6; ++a) path[(r * n + i) * 6 + a] = nan;
  }
  for (int a = 0; a < 3; ++a) {
    st[a] = x[a];
    st[3 + a] = v[a];
  }
}

}  // namespace arb

using namespace arb;

extern "C" int arb_rk4_trajectories_ordered(const arb_grid *g, int32_t precision, const float *pairs,
                                            const int64_t *order, double *state, int64_t n, double dt,
                                            int64_t nsteps, double coef, const double *gravity, double *path,
                                            int64_t record_every, unsigned long long *lost, arb_stream_t stream) {
  if (!g || !state || !lost || n < 0 || nsteps < 0 || g->dim != 3) return ARB_ERR_INVALID;
  if (g->nfield == 3) return ARB_ERR_UNSUPPORTED;  // vector mode carries no gradient
  if (path && record_every <= 0) return ARB_ERR_INVALID;
  const bool mixed = precision == ARB_PREC_MIXED;
  if (mixed ? !g->grid32 : !g->grid64) return ARB_ERR_INVALID;
  if (pairs && (!mixed || g->nfield != 4)) return ARB_ERR_INVALID;
  if (n == 0 || nsteps == 0) return ARB_OK;
  const double gr[3] = {gravity ? gravity[0] : 0.0, gravity ? gravity[1] : 0.0, gravity ? gravity[2] : 0.0};
  const KParams kp = make_kparams(g);
  cudaStream_t s = (cudaStream_t)stream;
  const int T = 128;
  const unsigned B = (unsigned)((n + T - 1) / T);
#define RK(FF, MX, PR)                                                                                          \
  rk4_kernel<FF, MX, PR><<<B, T, 0, s>>>(*g, kp, (const float2 *)pairs, order, state, n, dt, nsteps, coef, gr[0], \
                                         gr[1], gr[2], path, record_every, lost)
  if (g->nfield == 1) {
    if (mixed) RK(1, true, false); else RK(1, false, false);
  } else if (mixed) {
    if (pairs) RK(4, true, true); else RK(4, true, false);
  } else {
    RK(4, false, false);
  }
#undef RK
  return launch_status();
}

extern "C" int arb_rk4_trajectories(const arb_grid *g, int32_t precision, double *state, int64_t n, double dt,
                                    int64_t nsteps, double coef, const double *gravity, double *path,
                                    int64_t record_every, unsigned long long *lost, arb_stream_t stream) {
  return arb_rk4_trajectories_ordered(g, precision, nullptr, nullptr, state, n, dt, nsteps, coef, gravity, path,
                                      record_every, lost, stream);
}

extern "C" int arb_norm_pairs(const arb_grid *g, float *pairs, arb_stream_t stream) {
  if (!g || !g->grid32 || !pairs || g->nfield != 4 || g->dim != 3) return ARB_ERR_INVALID;
  const int64_t npts = g->n[0] * g->n[1] * g->n[2];
  norm_pairs_kernel<<<(unsigned)((npts + 255) / 256), 256, 0, (cudaStream_t)stream>>>(g->grid32, npts,
                                                                                     (float2 *)pairs);
  return launch_status();
}

extern "C" int arb_zorder_keys(const arb_grid *g, const double *state, int64_t n, int32_t *keys, arb_stream_t stream) {
  if (!g || g->dim != 3 || n < 0 || (n > 0 && (!state || !keys))) return ARB_ERR_INVALID;
  if (n == 0) return ARB_OK;
  const bool cells = n >= CELLS_FROM;
  float sc[3];
  for (int a = 0; a < 3; ++a) {  // cells where an axis has at most 1023 of them, else 1023 steps
    const double span = g->hi[a] - g->lo[a];
    sc[a] = (float)(cells && span <= 1023.0 * g->h[a] ? 1.0 / g->h[a] : 1023.0 / span);
  }
  const unsigned b = (unsigned)((n + 255) / 256);
  cudaStream_t s = (cudaStream_t)stream;
  if (cells)
    zorder_kernel<true><<<b, 256, 0, s>>>(state, n, g->lo[0], g->lo[1], g->lo[2], sc[0], sc[1], sc[2], keys);
  else
    zorder_kernel<false><<<b, 256, 0, s>>>(state, n, g->lo[0], g->lo[1], g->lo[2], sc[0], sc[1], sc[2], keys);
  return launch_status();
}
