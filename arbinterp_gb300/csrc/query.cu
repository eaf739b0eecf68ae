// Query evaluation kernels: replace rQuery1/2/3 and sQuery1/2/3
// (src/ARBInterp/ARBInterp.py:213-521, 916-1258).
//
// Two strategies, both one thread per query row:
//   * on-the-fly (otf_*): gathers the 4^dim grid block of the query's cell
//     and contracts it with tensor-product Catmull-Rom weights.  This is the
//     reference's  p(x) . (A f)  regrouped as  (A^T p(x)) . f , exact in real
//     arithmetic because A = kron(A1, A1, A1) in 3D; in 4D the reference's A
//     carries an extra rank-16 term from its row-240 D-matrix off-by-one,
//     evaluated here from 16 mixed fourth-difference stencils.
//   * table (tab_*): gathers the cell's coefficient row(s) and evaluates the
//     monomial sum by Horner's rule.
//
// Precision: FP64 forms cell index and fraction as the IEEE quotient gives
// them and contracts the float64 grid in block fixed point (fx.cuh; the table
// in float64 arithmetic).  MIXED reads the (hi, lo) float32 split of the grid
// (or a float32 table) and evaluates in float32; the cell index is that of the
// float64 step, so indices and NaN masks are bit-exact.
#include "eval.cuh"

namespace arb {

template <int F, bool MIXED>
__global__ void __launch_bounds__(256, MIXED && F != 1 ? 0 : 2) otf3_kernel(arb_grid g, KParams kp, double *q, int64_t nq,
                                                   int64_t qs, int wb, arb_query_out o,
                                                   int32_t *status) {
  using T = typename std::conditional<MIXED, float, double>::type;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  T frac_[3];
  int64_t idx;
  if (!query_prologue<3, F, !MIXED>(g, kp, q, i, qs, wb, o, status, frac_, idx)) return;
  const T fr[3] = {frac_[0], frac_[1], frac_[2]};
  double val[F], grad[3];
  int64_t c[3];
  cell_coords<3>(idx, g, c);
  eval_otf3<F, MIXED>(g, kp, c, fr, val, grad);
  write_vals<3, F>(o, i, val, grad);
}

template <int F, bool MIXED>
__global__ void __launch_bounds__(128, MIXED ? 0 : 3) otf4_kernel(arb_grid g, KParams kp, double *q, int64_t nq,
                                                   int64_t qs, int wb, arb_query_out o,
                                                   int32_t *status) {
  using T = typename std::conditional<MIXED, float, double>::type;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  T frac_[4];
  int64_t idx;
  if (!query_prologue<4, F, !MIXED>(g, kp, q, i, qs, wb, o, status, frac_, idx)) return;
  const T fr[4] = {frac_[0], frac_[1], frac_[2], frac_[3]};
  double val[F], grad[4] = {0, 0, 0, 0};
  int64_t c[4];
  cell_coords<4>(idx, g, c);
  eval_otf4<F, MIXED>(g, kp, c, fr, val, grad);
  write_vals<4, F>(o, i, val, grad);
}

template <int DIM, int F, bool MIXED>
__global__ void __launch_bounds__(256) tab_kernel(arb_grid g, KParams kp, double *q, int64_t nq,
                                                  int64_t qs, int wb, arb_query_out o,
                                                  int32_t *status) {
  using T = typename std::conditional<MIXED, float, double>::type;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  T x[DIM];
  int64_t idx;
  if (!query_prologue<DIM, F, !MIXED>(g, kp, q, i, qs, wb, o, status, x, idx)) return;
  double val[F], grad[DIM];
  int64_t c[DIM];
  cell_coords<DIM>(idx, g, c);
  eval_tab<DIM, F, MIXED>(g, kp, c, x, val, grad);
  write_vals<DIM, F>(o, i, val, grad);
}

// One point, as the row kernels evaluate it: the coordinates arrive with the
// launch and the results go straight to pinned host memory, so a call is one
// launch and one wait.  res: components [0..2], value [3], gradient [4..7], flat
// cell index [8] and the status word [9] (taken and cleared) as integers.
struct PointArg {
  double q[4];
};
template <int DIM, int F, bool MIXED, bool TABLE>
__global__ void __launch_bounds__(32) point_kernel(arb_grid g, KParams kp, PointArg p, double *res, int32_t *status) {
  using T = typename std::conditional<MIXED, float, double>::type;
  if (threadIdx.x) return;
  arb_query_out o{};
  o.comps = F >= 3 ? res : nullptr;
  o.norms = F != 3 ? res + 3 : nullptr;
  o.grads = F != 3 ? res + 4 : nullptr;
  o.inds = reinterpret_cast<int64_t *>(res + 8);
  o.comps_stride = 3;
  o.norms_stride = 1;
  o.grads_stride = DIM;
  T x[DIM];
  int64_t idx;
  if (query_prologue<DIM, F, !MIXED>(g, kp, (const double *)p.q, 0, DIM, 0, o, status, x, idx)) {
    int64_t c[DIM];
    cell_coords<DIM>(idx, g, c);
    double val[F], grad[DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) grad[a] = 0.0;
    if constexpr (TABLE)
      eval_tab<DIM, F, MIXED>(g, kp, c, x, val, grad);
    else if constexpr (DIM == 3)
      eval_otf3<F, MIXED>(g, kp, c, x, val, grad);
    else
      eval_otf4<F, MIXED>(g, kp, c, x, val, grad);
    write_vals<DIM, F>(o, 0, val, grad);
  }
  reinterpret_cast<int64_t *>(res)[9] = atomicExch(status, 0);
}

}  // namespace arb

using namespace arb;

extern "C" int arb_query_point(const arb_grid *g, int32_t precision, int32_t use_table, const double *q,
                               double *result, int32_t *status, arb_stream_t stream) {
  if (!g || !q || !result || !status || (g->dim != 3 && g->dim != 4)) return ARB_ERR_INVALID;
  if (g->nfield != 1 && g->nfield != 3 && g->nfield != 4) return ARB_ERR_INVALID;
  const bool mixed = use_table ? g->table_prec == ARB_PREC_MIXED : precision == ARB_PREC_MIXED;
  if (use_table ? !g->table : mixed ? !g->grid32 : !g->grid64) return ARB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  const KParams kp = make_kparams(g);
  PointArg p{};
  for (int a = 0; a < g->dim; ++a) p.q[a] = q[a];
#define PT(D, FF, MX, TB) point_kernel<D, FF, MX, TB><<<1, 32, 0, s>>>(*g, kp, p, result, status)
#define PTF(D, MX, TB) switch (g->nfield) { case 1: PT(D, 1, MX, TB); break; case 3: PT(D, 3, MX, TB); break; default: PT(D, 4, MX, TB); break; }
#define PTD(MX, TB) if (g->dim == 3) { PTF(3, MX, TB) } else { PTF(4, MX, TB) }
  if (use_table) {
    if (mixed) { PTD(true, true) } else { PTD(false, true) }
  } else {
    if (mixed) { PTD(true, false) } else { PTD(false, false) }
  }
#undef PTD
#undef PTF
#undef PT
  if (cudaGetLastError() != cudaSuccess) return ARB_ERR_CUDA;
  return cudaStreamSynchronize(s) == cudaSuccess ? ARB_OK : ARB_ERR_CUDA;
}

#define ARB_DISPATCH_F(KER, ...)                                \
  switch (g->nfield) {                                          \
    case 1: KER<1, __VA_ARGS__>; break;                         \
    case 3: KER<3, __VA_ARGS__>; break;                         \
    case 4: KER<4, __VA_ARGS__>; break;                         \
    default: return ARB_ERR_INVALID;                            \
  }

extern "C" int arb_query_eval_otf(const arb_grid *g, int32_t precision, double *q, int64_t nq,
                                  int64_t q_stride, int32_t q_writeback, const arb_query_out *out,
                                  int32_t *status, arb_stream_t stream) {
  int rc = check_query_args(g, q, nq, q_stride, out);
  if (rc) return rc;
  if (nq == 0) return ARB_OK;
  const bool mixed = precision == ARB_PREC_MIXED;
  if (mixed ? !g->grid32 : !g->grid64) return ARB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  const arb_query_out out_norm = normalize_out(*out, g->dim);
  out = &out_norm;
  const KParams kp = make_kparams(g);
  if (g->dim == 3) {
    const int T = 256;
    const unsigned B = (unsigned)((nq + T - 1) / T);
#define L3(FF, MX) otf3_kernel<FF, MX><<<B, T, 0, s>>>(*g, kp, q, nq, q_stride, q_writeback, *out, status)
    if (mixed) {
      switch (g->nfield) { case 1: L3(1, true); break; case 3: L3(3, true); break; case 4: L3(4, true); break; }
    } else {
      switch (g->nfield) { case 1: L3(1, false); break; case 3: L3(3, false); break; case 4: L3(4, false); break; }
    }
#undef L3
  } else {
    const int T = 128;
    const unsigned B = (unsigned)((nq + T - 1) / T);
#define L4(FF, MX) otf4_kernel<FF, MX><<<B, T, 0, s>>>(*g, kp, q, nq, q_stride, q_writeback, *out, status)
    if (mixed) {
      switch (g->nfield) { case 1: L4(1, true); break; case 3: L4(3, true); break; case 4: L4(4, true); break; }
    } else {
      switch (g->nfield) { case 1: L4(1, false); break; case 3: L4(3, false); break; case 4: L4(4, false); break; }
    }
#undef L4
  }
  return launch_status();
}

extern "C" int arb_query_eval(const arb_grid *g, double *q, int64_t nq, int64_t q_stride,
                              int32_t q_writeback, const arb_query_out *out, int32_t *status,
                              arb_stream_t stream) {
  int rc = check_query_args(g, q, nq, q_stride, out);
  if (rc) return rc;
  if (!g->table) return ARB_ERR_INVALID;
  if (nq == 0) return ARB_OK;
  const bool mixed = g->table_prec == ARB_PREC_MIXED;
  cudaStream_t s = (cudaStream_t)stream;
  const arb_query_out out_norm = normalize_out(*out, g->dim);
  out = &out_norm;
  const KParams kp = make_kparams(g);
  const int T = 256;
  const unsigned B = (unsigned)((nq + T - 1) / T);
#define LT(D, FF, MX) tab_kernel<D, FF, MX><<<B, T, 0, s>>>(*g, kp, q, nq, q_stride, q_writeback, *out, status)
#define LTF(D, MX) switch (g->nfield) { case 1: LT(D, 1, MX); break; case 3: LT(D, 3, MX); break; case 4: LT(D, 4, MX); break; }
  if (g->dim == 3) {
    if (mixed) { LTF(3, true) } else { LTF(3, false) }
  } else {
    if (mixed) { LTF(4, true) } else { LTF(4, false) }
  }
#undef LTF
#undef LT
  return launch_status();
}
