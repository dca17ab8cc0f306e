// General sparse solves for the reference's second plugin point,
// matrix_solver(A, b, **opts) -> x (meanas/fdfd/solvers.py:97-103,134), where A is the
// assembled CSR operator (the symmetrised e_full of generic(), or any other operator a
// caller builds, e.g. from eh_full / h_full).  Complex128 CSR, 32-bit column indices,
// 64-bit row pointers.
//
// SpMV: a group of LPR lanes per row walks the row's nonzeros, CSR_UNROLL steps at a time
// with all their loads in flight together, and reduces with warp shuffles; every warp
// handles 32 / LPR consecutive rows per step, so all lanes of a warp run the same number of
// steps (the shuffles need whole warps).
//
// BiCGSTAB (complex, hashed shadow vector as in the stencil solver), three kernels per
// iteration; s = r - alpha v is formed where it is needed and never stored:
//   CA: v = A p, sigma = (rh, v)                                        -> alpha
//   CB: t = A (r - alpha v) with s formed at the columns, (t, s), |t|^2, |s|^2, (rh, s),
//       (rh, t)                                                         -> omega, beta
//   CC: x += alpha p + omega s, r = s - omega t, p = r + beta (p - omega v), |r|^2
// Forming p and s in the gathers instead cost CA three gathers per nonzero.  Reductions are
// the deterministic grid reductions of the stencil engine; the scalars (rho, alpha, omega,
// beta) stay in FP64 device state.
//
// What bounds it: the latency of index load and gather, then L2 (a matrix of 20 bytes per
// nonzero that stays there), and the reductions' tails.  Per iteration on the wave operator of
// 40x36x32 cells (138 thousand rows, 12.9 nonzeros each): CA 33 -> 11.5 us, CB 26 -> 20, CC (one
// lane in four worked) 20 -> 10.6, and 2 us between each two; launched so that a pass's CTAs
// come up during the one before (pass_begin), 86 -> 43 us in all.  Four lanes per row: two are
// as fast, eight 30 % slower; three CTAs per SM leave the registers for the unrolled loads.
#pragma once
#include "fdfd_ops.cuh"

namespace fdfd {

struct CsrView {
  int n;
  const long long* indptr;
  const int* indices;
  const cx<double>* data;
};

constexpr int CSR_LPR = 4;    // lanes per row
constexpr int CSR_NT = 256;   // threads per CTA

// Row loop shared by the CSR kernels: calls f(row, lane_in_group, valid) for each step.
template <class F>
__device__ __forceinline__ void csr_rows(int n, F&& f) {
  constexpr int RPW = 32 / CSR_LPR;  // rows per warp per step
  const int lane = threadIdx.x & 31, g = lane / CSR_LPR, l = lane % CSR_LPR;
  const int warp = (blockIdx.x * CSR_NT + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * CSR_NT) >> 5;
  for (long long base = (long long)warp * RPW; base < n; base += (long long)nwarps * RPW) {
    const long long row = base + g;
    f((int)row, l, row < n);
  }
}

// sum over the row of A[row, j] * xf(j), reduced over the lane group (valid in every lane)
constexpr int CSR_UNROLL = 4;
template <class XF>
__device__ __forceinline__ cx<double> csr_row(const CsrView& A, int row, int l, bool valid, XF&& xf) {
  cx<double> acc = czero<double>();
  if (valid) {
    const long long e1 = A.indptr[row + 1];
    for (long long e = A.indptr[row] + l; e < e1; e += CSR_LPR * CSR_UNROLL) {
      int j[CSR_UNROLL];
      cx<double> a[CSR_UNROLL], v[CSR_UNROLL];
#pragma unroll
      for (int u = 0; u < CSR_UNROLL; ++u) {
        const bool in = e + u * CSR_LPR < e1;
        j[u] = in ? A.indices[e + u * CSR_LPR] : -1;
        a[u] = in ? A.data[e + u * CSR_LPR] : czero<double>();
      }
#pragma unroll
      for (int u = 0; u < CSR_UNROLL; ++u) v[u] = j[u] >= 0 ? xf(j[u]) : czero<double>();
#pragma unroll
      for (int u = 0; u < CSR_UNROLL; ++u)
        if (j[u] >= 0) acc = acc + a[u] * v[u];
    }
  }
#pragma unroll
  for (int o = 1; o < CSR_LPR; o <<= 1) {
    acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o);
    acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o);
  }
  return acc;
}

// y = A x
__global__ void __launch_bounds__(CSR_NT) k_csr_spmv(CsrView A, const cx<double>* __restrict__ x,
                                                    cx<double>* __restrict__ y) {
  csr_rows(A.n, [&](int row, int l, bool valid) {
    const cx<double> v = csr_row(A, row, l, valid, [&](int j) { return x[j]; });
    if (valid && l == 0) y[row] = v;
  });
}

struct CsrBufs {
  cx<double>* p;
  cx<double>* v;
  cx<double>* r;
  cx<double>* t;
  cx<double>* x;
  const cx<double>* b;
};

template <int NRED, class Body, class Fin>
__device__ __forceinline__ void csr_pass(const CsrView& A, RedBuf rb, Body&& body, Fin&& fin) {
  __shared__ double shred[64];
  double acc[NRED];
#pragma unroll
  for (int r = 0; r < NRED; ++r) acc[r] = 0.0;
  csr_rows(A.n, [&](int row, int l, bool valid) { body(row, l, valid, acc); });
  double sums[NRED];
  if (grid_reduce<CSR_NT, NRED>(acc, rb, shred, sums)) fin(sums);
}

// Start: r = b - A x (x = 0 unless a guess is given), p = r, rho = (rh, r), |r|^2, |b|^2.
__global__ void __launch_bounds__(CSR_NT) k_csr_init(CsrView A, CsrBufs B, int guess, unsigned seed, KState* st,
                                                    RedBuf rb) {
  csr_pass<4>(A, rb, [&](int row, int l, bool valid, double* acc) {
    cx<double> ax = czero<double>();
    if (guess) ax = csr_row(A, row, l, valid, [&](int j) { return B.x[j]; });
    if (valid && l == 0) {
      const cx<double> bv = B.b[row];
      const cx<double> r = bv - ax;
      B.r[row] = r;
      B.p[row] = r;
      if (!guess) B.x[row] = czero<double>();
      acc_cdot<double>(acc, shadow<double>(row, seed), r);
      acc[2] += cabs2(r);
      acc[3] += cabs2(bv);
    }
  }, [&](const double* s) {
    st->rho = {s[0], s[1]};
    st->rr = s[2];
    st->bb = s[3];
    const double tol2 = fmax(st->rtol * st->rtol * s[3], st->atol * st->atol);
    st->tol2 = tol2;
    st->alpha = {0.0, 0.0};
    st->omega = {0.0, 0.0};
    st->beta = {0.0, 0.0};
    st->iter = 0;
    st->pending = 0;
    if (!isfinite(s[2]) || !isfinite(s[3])) st->status = ST_NONFINITE;
    else if (s[2] <= tol2) st->status = ST_CONVERGED;
    else st->status = ST_RUNNING;
  });
}

__global__ void __launch_bounds__(CSR_NT, 3) k_csr_a(CsrView A, CsrBufs B, unsigned seed, KState* st, RedBuf rb) {
  pass_begin();
  if (ld_status(st) != ST_RUNNING) return;
  csr_pass<2>(A, rb, [&](int row, int l, bool valid, double* acc) {
    const cx<double> v = csr_row(A, row, l, valid, [&](int j) { return B.p[j]; });
    if (valid && l == 0) {
      B.v[row] = v;
      acc_cdot<double>(acc, shadow<double>(row, seed), v);
    }
  }, [&](const double* s) {
    const dcx sigma = {s[0], s[1]};
    if (!dfinite(sigma)) { st->status = ST_NONFINITE; return; }
    if (sigma.re == 0.0 && sigma.im == 0.0) { st->status = ST_BREAKDOWN; return; }
    st->alpha = ddiv(st->rho, sigma);
  });
}

__global__ void __launch_bounds__(CSR_NT, 3) k_csr_b(CsrView A, CsrBufs B, unsigned seed, KState* st, RedBuf rb) {
  pass_begin();
  if (ld_status(st) != ST_RUNNING) return;
  const dcx ad = ld_dcx(&st->alpha);
  const cx<double> malpha = mkc<double>(-ad.re, -ad.im);
  auto snew = [&](int j) { return caxpy(malpha, B.v[j], B.r[j]); };
  csr_pass<8>(A, rb, [&](int row, int l, bool valid, double* acc) {
    const cx<double> t = csr_row(A, row, l, valid, snew);
    if (valid && l == 0) {
      const cx<double> s = snew(row), h = shadow<double>(row, seed);
      B.t[row] = t;
      acc_cdot<double>(acc, t, s);
      acc[2] += cabs2(t);
      acc[3] += cabs2(s);
      acc_cdot<double>(acc + 4, h, s);
      acc_cdot<double>(acc + 6, h, t);
    }
  }, [&](const double* s) {
    bool ok = true;
    for (int q = 0; q < 8; ++q) ok = ok && isfinite(s[q]);
    if (!ok) {
      st->status = ST_NONFINITE;
      return;
    }
    st->beta = {0.0, 0.0};
    if (s[3] <= st->tol2 || s[2] <= 0.0) {
      // s is small enough (or t vanished): finish this iteration with omega = 0
      st->omega = {0.0, 0.0};
      st->pending = s[3] <= st->tol2 ? 2 : 3;
      return;
    }
    const dcx om = {s[0] / s[2], s[1] / s[2]}, w = dmul(om, {s[6], s[7]});
    const dcx rho_new = {s[4] - w.re, s[5] - w.im};  // (rh, s - omega t)
    st->omega = om;
    if ((rho_new.re == 0.0 && rho_new.im == 0.0) || (om.re == 0.0 && om.im == 0.0)) {
      st->pending = 4;  // a breakdown, unless this iteration converges
      return;
    }
    st->beta = dmul(ddiv(rho_new, st->rho), ddiv(st->alpha, om));
    st->rho = rho_new;
  });
}

// (elementwise: every lane a row)
__global__ void __launch_bounds__(CSR_NT) k_csr_c(CsrView A, CsrBufs B, KState* st, RedBuf rb) {
  pass_begin();
  if (ld_status(st) != ST_RUNNING) return;
  const cx<double> alpha = from_d<double>(ld_dcx(&st->alpha)), beta = from_d<double>(ld_dcx(&st->beta));
  const cx<double> omega = from_d<double>(ld_dcx(&st->omega));
  const cx<double> malpha = mkc<double>(-alpha.re, -alpha.im), momega = mkc<double>(-omega.re, -omega.im);
  __shared__ double shred[64];
  double acc[1] = {0.0};
  for (long long row = blockIdx.x * (long long)CSR_NT + threadIdx.x; row < A.n; row += (long long)gridDim.x * CSR_NT) {
    const cx<double> p = B.p[row], v = B.v[row], s = caxpy(malpha, v, B.r[row]);
    B.x[row] = caxpy(omega, s, caxpy(alpha, p, B.x[row]));
    const cx<double> r = caxpy(momega, B.t[row], s);
    B.r[row] = r;
    B.p[row] = caxpy(beta, caxpy(momega, v, p), r);
    acc[0] += cabs2(r);
  }
  double sums[1];
  if (grid_reduce<CSR_NT, 1>(acc, rb, shred, sums)) {
    st->iter += 1;
    st->rr = sums[0];
    if (!isfinite(sums[0])) st->status = ST_NONFINITE;
    else if (st->pending == 2 || sums[0] <= st->tol2) st->status = ST_CONVERGED;
    else if (st->pending == 3) st->status = ST_BREAKDOWN;
    else if (st->iter >= st->maxiter) st->status = ST_MAXITER;
    else if (st->pending == 4) st->status = ST_BREAKDOWN;
  }
}

// |b - A x|^2 and |b|^2 (the true residual of the final iterate)
__global__ void __launch_bounds__(CSR_NT) k_csr_residual(CsrView A, const cx<double>* __restrict__ x,
                                                        const cx<double>* __restrict__ b, double* out, RedBuf rb) {
  csr_pass<2>(A, rb, [&](int row, int l, bool valid, double* acc) {
    const cx<double> ax = csr_row(A, row, l, valid, [&](int j) { return x[j]; });
    if (valid && l == 0) {
      acc[0] += cabs2(b[row] - ax);
      acc[1] += cabs2(b[row]);
    }
  }, [&](const double* s) {
    out[0] = s[0];
    out[1] = s[1];
  });
}

}  // namespace fdfd
