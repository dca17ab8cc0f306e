// FDTD Yee updates with CPML: the time-domain stencil loop of the reference
// (meanas/fdtd/base.py:13-125, meanas/fdtd/pml.py:96-230).
//
//   H step:  H -= dt / mu * (curl_f(E) + psi terms)      (forward differences)
//   E step:  E += dt / eps * (curl_b(H) + psi terms)     (backward differences)
//
// Two forms, matching the reference's two update builders:
//   PLAIN (maxwell_h / maxwell_e): H -= dt * curl_f(E) [/ mu];  E += dt * curl_b(H) / eps,
//          forward differences over dxes[0], backward over dxes[1];
//   CPML  (updates_with_cpml):     H -= dt / mu * (curl_f(E) + pH);  E += dt / eps * (curl_b(H) + pE),
//          both difference kinds over dxes[1] (the reference builds deriv_forward(dxes[1])),
//          and on the PML slab of each face the differences along that axis are scaled by
//          p2 = 1/kappa and feed the psi recurrences  psi = p0 psi + p1 d  whose sums form pE/pH.
// Arithmetic follows the reference's numpy evaluation step by step: a difference of two
// field values in the field type, everything after it in FP64 with explicit
// round-to-nearest operations (no contraction), psi and the PML sums rounded to the psi
// type at every in-place step, the result rounded to the field type.  So the GPU
// trajectories equal the reference's bit for bit.
#pragma once
#include "fdfd_device.cuh"

namespace fdfd {

struct CpmlFace {
  int th;                 // layers (0: no PML on this face)
  const double* p;        // [3][th]: p0, p1, p2 per layer
  void* psi_u;            // psi of the first transverse component, region shape
  void* psi_v;
};

struct FdtdGeo {
  int X, Y, Z;
  // The cells in two lists: those outside the layers along z (all, without layers) and those
  // inside them; nz cells of every (x, y) row are in the first.  by_*[list]: number -> row, plane.
  int nz, slab_blocks;    // CTAs of the second list (the first in the grid)
  FastDiv by_row[2], by_y;
  int table;              // cell widths and reciprocals fit the shared-memory table
  const double* dxf[3];   // widths dividing the forward differences
  const double* dxb[3];   // widths dividing the backward differences
  const double* mat;      // epsilon (E step) or mu (H step, may be null: 1), [3N]
  double dt;
  int cpml;               // 0: PLAIN form, 1: CPML form
  CpmlFace face[3][2];    // [axis][0: low face, 1: high face]
};

__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmulr(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddivr(double a, double b) { return __ddiv_rn(a, b); }

template <typename T>
__device__ __forceinline__ T tsub(T a, T b);
template <>
__device__ __forceinline__ float tsub<float>(float a, float b) { return __fsub_rn(a, b); }
template <>
__device__ __forceinline__ double tsub<double>(double a, double b) { return __dsub_rn(a, b); }
template <typename T>
__device__ __forceinline__ T tadd(T a, T b);
template <>
__device__ __forceinline__ float tadd<float>(float a, float b) { return __fadd_rn(a, b); }
template <>
__device__ __forceinline__ double tadd<double>(double a, double b) { return __dadd_rn(a, b); }

template <typename T>
__device__ __forceinline__ T tmul(T a, T b);
template <>
__device__ __forceinline__ float tmul<float>(float a, float b) { return __fmul_rn(a, b); }
template <>
__device__ __forceinline__ double tmul<double>(double a, double b) { return __dmul_rn(a, b); }

// psi in place:  psi = P(psi * p0);  psi = P(psi + p1 * d)   (FP64 products, as numpy does
// for a psi array and FP64 parameters)
template <typename P>
__device__ __forceinline__ P psi_step(P psi, double p0, double p1, double d) {
  const P a = (P)dmulr((double)psi, p0);
  return (P)dadd((double)a, dmulr(p1, d));
}

// a / w rounded to nearest, from r = 1 / w rounded to nearest: Markstein's correction (the
// residual a - q w is exact in a fused multiply-add), applied twice so that the quotient it
// finally corrects is within one ulp.  Outside the exponents where the residual is exact
// (and for infinities and NaN) the plain division runs; a zero's quotient is a r.  r = 0
// marks a width the correction does not cover (see width_entry).
__device__ __forceinline__ double div_by(double a, double2 wr) {
  const double w = wr.x, r = wr.y;
  double q = dmulr(a, r);
  const unsigned e = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  if (e - 200u < 1600u && r != 0.0) {
    q = fma(fma(-q, w, a), r, q);
    q = fma(fma(-q, w, a), r, q);
  } else if (a != 0.0 || r == 0.0) {
    q = ddivr(a, w);
  }
  return q;
}
// A width and its rounded reciprocal; widths beyond 2^+-100, NaN, or with a mantissa of ones
// (the one case Markstein's theorem leaves out) get reciprocal 0.
__device__ __forceinline__ double2 width_entry(double w) {
  const unsigned hi = (unsigned)__double2hiint(w), lo = (unsigned)__double2loint(w);
  const unsigned e = (hi >> 20) & 0x7ffu;
  const bool ok = e - 923u < 200u && !((hi & 0xfffffu) == 0xfffffu && lo == 0xffffffffu);
  return make_double2(w, ok ? ddivr(1.0, w) : 0.0);
}

constexpr int FDTD_NT = 256;
constexpr int FDTD_TABLE = 2048;  // widths of the three axes together (32 KB)

// FACES: 0 PLAIN or no layers, 1 at most one layer per axis holds a cell, 2 any.  ZL: the
// cells of the second list (inside the layers along z), otherwise the first.
//
// One half step on cells first, first + stride, ... of a list: ESTEP updates E from H,
// otherwise H from E.
template <typename R, typename P, bool ESTEP, int FACES, bool TABLE, bool ZL>
__device__ __forceinline__ void fdtd_cells(const FdtdGeo& g, const double2* tab, R* __restrict__ e, R* __restrict__ h,
                                           int first, int stride) {
  const int YZ = g.Y * g.Z, N = g.X * YZ;
  const R* const src = ESTEP ? h : e;
  R* const dst = ESTEP ? e : h;
  const int row = ZL ? g.Z - g.nz : g.nz, count = g.X * g.Y * row;
  for (int base = first; base < count; base += stride) {
    R here[3], there[3][3], old[3];  // there[a][c]: component c one cell along a
    double mat[3];
    const int r = (int)g.by_row[ZL]((unsigned)base), s = base - r * row;
    const int i = (int)g.by_y((unsigned)r), j = r - i * g.Y;
    const int lo = FACES == 1 ? g.face[2][0].th : 0;  // (one list otherwise)
    const int k = ZL ? (s < lo ? s : s + g.nz) : s + lo;
    const int n = r * g.Z + k;
    const int idx[3] = {i, j, k};
    // neighbour cells: -1 (E step) or +1 (H step) along each axis, periodic
    int nb[3];
    if (ESTEP) {
      nb[0] = i == 0 ? n + (g.X - 1) * YZ : n - YZ;
      nb[1] = j == 0 ? n + (g.Y - 1) * g.Z : n - g.Z;
      nb[2] = k == 0 ? n + (g.Z - 1) : n - 1;
    } else {
      nb[0] = i + 1 == g.X ? n - i * YZ : n + YZ;
      nb[1] = j + 1 == g.Y ? n - j * g.Z : n + g.Z;
      nb[2] = k + 1 == g.Z ? n - k : n + 1;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      here[c] = src[c * N + n];
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (a != c) there[a][c] = src[c * N + nb[a]];
      old[c] = dst[c * N + n];
      mat[c] = g.mat ? g.mat[c * N + n] : 1.0;
    }
    // the layer, if any, that holds the cell on each axis, and what it needs
    P pu[3], pv[3];
    double q0[3], q1[3], q2[3];
    P *psi_u[3], *psi_v[3];
    bool in[3];
    if (FACES == 1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int na = a == 0 ? g.X : (a == 1 ? g.Y : g.Z);
        const int lo = g.face[a][0].th, hi = g.face[a][1].th;
        const bool low = idx[a] < lo;
        in[a] = a == 2 ? ZL : low || idx[a] >= na - hi;
        if (!in[a]) continue;
        // (selects: a face picked by index would be a divergent constant load)
        const int th = low ? lo : hi, l = low ? idx[a] : idx[a] - (na - hi);
        const double* const fp = low ? g.face[a][0].p : g.face[a][1].p;
        const int ri = a == 0 ? (l * g.Y + j) * g.Z + k : (a == 1 ? (i * th + l) * g.Z + k : (i * g.Y + j) * th + l);
        psi_u[a] = (P*)(low ? g.face[a][0].psi_u : g.face[a][1].psi_u) + ri;
        psi_v[a] = (P*)(low ? g.face[a][0].psi_v : g.face[a][1].psi_v) + ri;
        pu[a] = *psi_u[a];
        pv[a] = *psi_v[a];
        q0[a] = fp[l];
        q1[a] = fp[th + l];
        q2[a] = fp[2 * th + l];
      }
    }
    // d[a][c]: difference along axis a of component c (only c != a is used)
    double d[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double2 wr;
      if (TABLE) wr = tab[idx[a] + (a > 0 ? g.X : 0) + (a > 1 ? g.Y : 0)];
      else wr = make_double2(ESTEP ? g.dxb[a][idx[a]] : g.dxf[a][idx[a]], 0.0);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (c == a) continue;
        const R diff = ESTEP ? tsub<R>(here[c], there[a][c]) : tsub<R>(there[a][c], here[c]);
        d[a][c] = TABLE ? div_by((double)diff, wr) : ddivr((double)diff, wr.x);
      }
    }
    P pc[3] = {P(0), P(0), P(0)};
    if (FACES == 1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (!in[a]) continue;
        const int uu = a == 0 ? 1 : 0, vv = a == 2 ? 1 : 2;
        d[a][uu] = dmulr(d[a][uu], q2[a]);
        d[a][vv] = dmulr(d[a][vv], q2[a]);
        const P su = psi_step<P>(pu[a], q0[a], q1[a], d[a][vv]);  // reversed u, v, as in the reference
        const P sv = psi_step<P>(pv[a], q0[a], q1[a], d[a][uu]);
        *psi_u[a] = su;
        *psi_v[a] = sv;
        pc[uu] = tadd<P>(pc[uu], a == 1 ? su : -su);
        pc[vv] = tadd<P>(pc[vv], a == 1 ? -sv : sv);
      }
    } else if (FACES == 2) {
      const int dims[3] = {g.X, g.Y, g.Z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int uu = a == 0 ? 1 : 0, vv = a == 2 ? 1 : 2;
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          const CpmlFace& f = g.face[a][pp];
          if (f.th == 0) continue;
          const int l = pp == 0 ? idx[a] : idx[a] - (dims[a] - f.th);
          if (l < 0 || l >= f.th) continue;
          const double p0 = f.p[l], p1 = f.p[f.th + l], p2 = f.p[2 * f.th + l];
          d[a][uu] = dmulr(d[a][uu], p2);
          d[a][vv] = dmulr(d[a][vv], p2);
          // region index of this cell (region shape: th along a, full along the others)
          const int rc = a == 0 ? (l * g.Y + j) * g.Z + k : (a == 1 ? (i * f.th + l) * g.Z + k : (i * g.Y + j) * f.th + l);
          P* fu = (P*)f.psi_u;
          P* fv = (P*)f.psi_v;
          const P su = psi_step<P>(fu[rc], p0, p1, d[a][vv]);
          const P sv = psi_step<P>(fv[rc], p0, p1, d[a][uu]);
          fu[rc] = su;
          fv[rc] = sv;
          pc[uu] = tadd<P>(pc[uu], a == 1 ? su : -su);
          pc[vv] = tadd<P>(pc[vv], a == 1 ? -sv : sv);
        }
      }
    }
    // curl components: x: d_y(.z) - d_z(.y); y: d_z(.x) - d_x(.z); z: d_x(.y) - d_y(.x)
    double curl[3];
    curl[0] = dsub(d[1][2], d[2][1]);
    curl[1] = dsub(d[2][0], d[0][2]);
    curl[2] = dsub(d[0][1], d[1][0]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double mc = mat[c];
      if (g.cpml) {
        const double coef = mc == 1.0 ? g.dt : ddivr(g.dt, mc);
        const double step = dmulr(coef, dadd(curl[c], (double)pc[c]));
        dst[c * N + n] = (R)(ESTEP ? dadd((double)old[c], step) : dsub((double)old[c], step));
      } else {
        // the PLAIN form keeps the curl in an array of the field type and scales it there
        const R st = tmul<R>((R)g.dt, (R)curl[c]);
        if (g.mat) {
          const double step = mc == 1.0 ? (double)st : ddivr((double)st, mc);
          dst[c * N + n] = (R)(ESTEP ? dadd((double)old[c], step) : dsub((double)old[c], step));
        } else {
          dst[c * N + n] = ESTEP ? tadd<R>(old[c], st) : tsub<R>(old[c], st);
        }
      }
    }
  }
}

// What bounds it: the fields mostly stay in L2 between half steps, and an FP64 division is
// some thirty instructions, so it waited for one cell's dependent loads and then for
// instruction issue.  Cells go to threads by number, so every lane works on any shape (lanes
// along z leave one of 32 on a flat grid) and all loads of a cell are in flight together;
// six of the six (H) or nine (E) divisions of a cell are by cell widths and take div_by;
// dt / epsilon is dt where epsilon is 1.  The cells inside the layers along z, a few of every
// row, are a list of their own: in the rows' warps their code ran for half of all warps.
// H / E half step before and now, 160x160x128: float32 51 / 84 -> 35 / 50 us (PLAIN), 78 / 100 ->
// 59 / 65 (CPML on every face); float64 93 / 103 -> 47 / 53, 115 / 124 -> 60 / 64; flat
// 1000x800 float32 454 / 525 -> 19 / 21.  Four CTAs of 64 registers per SM: three or five are 2
// to 15 % slower.  The instances with layers (FACES 1) spill 130 to 240 bytes per thread at
// that cap, the others next to nothing.
template <typename R, typename P, bool ESTEP, int FACES, bool TABLE>
__global__ void __launch_bounds__(FDTD_NT, 4) k_fdtd(const FdtdGeo g, R* __restrict__ e, R* __restrict__ h) {
  __shared__ double2 tab[TABLE ? FDTD_TABLE : 1];
  if (TABLE) {
    for (int t = threadIdx.x; t < g.X + g.Y + g.Z; t += FDTD_NT) {
      const int a = t < g.X ? 0 : (t < g.X + g.Y ? 1 : 2);
      const int i = t - (a > 0 ? g.X : 0) - (a > 1 ? g.Y : 0);
      tab[t] = width_entry(ESTEP ? g.dxb[a][i] : g.dxf[a][i]);
    }
    __syncthreads();
  }
  const int b = (int)blockIdx.x - g.slab_blocks;
  if (FACES == 1 && b < 0) {
    fdtd_cells<R, P, ESTEP, FACES, TABLE, true>(g, tab, e, h, blockIdx.x * FDTD_NT + threadIdx.x,
                                               g.slab_blocks * FDTD_NT);
  } else {
    fdtd_cells<R, P, ESTEP, FACES, TABLE, false>(g, tab, e, h, b * FDTD_NT + threadIdx.x,
                                                (gridDim.x - g.slab_blocks) * FDTD_NT);
  }
}

}  // namespace fdfd
