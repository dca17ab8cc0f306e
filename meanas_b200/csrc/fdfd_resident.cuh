// Resident Krylov iterations for grids whose vectors fit on the SMs.
//
// One cooperative launch holds the whole grid: CTA b owns a brick of cells and keeps the
// Krylov vectors of its brick and of a one-cell shell around it in registers and shared
// memory for many iterations.  The shell is updated redundantly with the same arithmetic as
// its owner, so the only data that cross CTAs are the operator products on brick surfaces
// and the partial sums of the dot products, which travel through L2 with the two grid-wide
// exchanges that an iteration needs anyway.
//
// What bounds it: the latency of those two exchanges plus a few shared-memory passes over
// the brick.  The two-launch form of the same iteration pays instead a launch, a serial
// chain of plane loads per CTA and a last-CTA reduction tail in each of its two kernels,
// all of it latency.
//
// Exchange (the forms measured at 148 CTAs, cycles per exchange of one or two sums, the
// block sum not counted): every CTA polling every CTA's word 6400; release /
// acquire around a counter and plain partial sums 5800 (the fences wait for all stores in
// flight and empty the L1); a counter without fences and tagged words 2000, which is the
// one taken.  A CTA stores a partial sum together with the number of the exchange in one
// 16-byte word and adds one to a counter; one lane per sum polls the counter, then a warp
// reads the words of all CTAs and adds them in a fixed order, so the sums are the same in
// every CTA and from run to run.  The counter only says when to look: a word counts when
// its tag is right and is read again until it is.  Surface values carry their tag in the
// same way.  Nothing relies on fences.
//
// Reuse of words: a CTA writes its words of the next exchange of a kind only after the
// other exchange in between has completed, which all readers entered after reading.
// Every wait is bounded: after `limit` reads (SPIN_LIMIT, or the caller's; SPIN_LIMIT in the
// first exchange of a launch, which waits for the launch itself) a CTA gives up, sets
// KState::timed_out and returns (the launch is cooperative, so its CTAs do run at the same
// time).  The others may have got past that exchange, converged even, so the flag and not the
// status that CTA 0 writes says whether the vectors belong together; launches that find it set
// do nothing.
#pragma once
#include "fdfd_ops.cuh"

namespace fdfd {

constexpr int ST_TIMEOUT = 5;
constexpr int SPIN_LIMIT = 1 << 22;  // one to two seconds

// Bricks of the grid: nx x ny x nz of them, at most bx x by x bz cells each (the split of
// an axis is balanced: brick i covers [i n / m, (i + 1) n / m)).
struct Bricks {
  int nx, ny, nz, bx, by, bz;
};

// ------------------------------------------------------------------ tagged words
struct __align__(16) Word {  // a value and the number of the exchange it belongs to
  unsigned long long v, tag;
};

__device__ __forceinline__ void word_store(Word* p, unsigned long long v, unsigned long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p), "l"(v),
               "l"(tag)
               : "memory");
}
__device__ __forceinline__ Word word_load(const Word* p) {
  Word w;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(w.v), "=l"(w.tag)
               : "l"(p)
               : "memory");
  return w;
}
__device__ __forceinline__ unsigned long long pack(float a, float b) {
  return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}

// Global scratch of a resident solve: a row of words and a counter (on a line of its own)
// per sum.  Counters are zeroed before every launch; the words' tags never repeat within a
// solve.
constexpr int RES_CTAS = 160;  // CTAs at most
constexpr int RES_SUMS = 8;    // sums of the two exchanges together
struct ResidentScratch {
  unsigned int counter[RES_SUMS][64];
  Word word[RES_SUMS][RES_CTAS];
};

// Sum NRED per-thread values over the grid, sums number FIRST ... of the scratch.  The
// first half stores and arrives; the second waits for exchange `tag`, the `round`-th of
// this launch (from 1), and leaves the totals in `out` (shared memory).  Warp r looks after
// value r throughout.  Every thread must call both.
//
// Block sum: two shuffle rounds, then the quarter lanes' sums through shared memory
// (`red`, NRED rows of RED_ROW), where warp r adds up row r.  Shuffling all the way is 10
// shuffles per value and warp, and the SM has one shuffle unit for them.
template <int NT>
struct RedRow {
  static constexpr int value = NT / 4;
};
template <int NT, int FIRST, int NRED>
__device__ __forceinline__ void sums_begin(double (&v)[NRED], double* red, ResidentScratch* gs,
                                           unsigned long long tag) {
  constexpr int ROW = RedRow<NT>::value;
  static_assert(NRED <= NT / 32 && FIRST + NRED <= RES_SUMS && ROW % 32 == 0, "");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 4; o >>= 1) {
#pragma unroll
    for (int r = 0; r < NRED; ++r) v[r] += __shfl_down_sync(0xffffffffu, v[r], o);
  }
  if (lane < 8) {
#pragma unroll
    for (int r = 0; r < NRED; ++r) red[r * ROW + warp * 8 + lane] = v[r];
  }
  __syncthreads();
  if (warp < NRED) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < ROW; q += 32) s += red[warp * ROW + q + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
      word_store(&gs->word[FIRST + warp][blockIdx.x], (unsigned long long)__double_as_longlong(s), tag);
      asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&gs->counter[FIRST + warp][0]) : "memory");
    }
  }
}

template <int FIRST, int NRED>
__device__ __forceinline__ bool sums_end(double* out, int* gave_up, ResidentScratch* gs, unsigned long long tag,
                                         unsigned int round, int limit) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < NRED) {
    bool ok = true;
    if (lane == 0) {
      const unsigned int all = gridDim.x * round;
      unsigned int n = 0;
      int spin = 0;
      do {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&gs->counter[FIRST + warp][0]) : "memory");
      } while (n < all && ++spin < limit);
      ok = n >= all;
    }
    __syncwarp();
    constexpr int M = RES_CTAS / 32;
    const Word* w = gs->word[FIRST + warp];
    const int last = (int)gridDim.x - 1;
    Word got[M];
    bool here = false;
    int spin = 0;
    do {
#pragma unroll
      for (int m = 0; m < M; ++m) got[m] = word_load(w + min(lane + 32 * m, last));
      here = true;
#pragma unroll
      for (int m = 0; m < M; ++m) here = here && got[m].tag == tag;
    } while (!here && ++spin < limit);
    double s = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (lane + 32 * m <= last) s += __longlong_as_double((long long)got[m].v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (!(ok && here)) *gave_up = 1;
    if (lane == 0) out[warp] = s;
  }
  __syncthreads();
  return *gave_up == 0;
}

// x / d for normal d, from the hardware's approximate reciprocal (better than 2^-20), two
// Newton steps, whose errors square (2^-40, then rounding: within an ulp), and the residual of
// the quotient, which rounds it as a division does but for rare last bits.  A division is some
// 400 cycles of latency, an iteration's scalar work had six to nine of them.
__device__ __forceinline__ double newton_reciprocal(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  y = fma(y, fma(-d, y, 1.0), y);
  return fma(y, fma(-d, y, 1.0), y);
}
__device__ __forceinline__ double quotient(double x, double d, double inv_d) {
  const double q = x * inv_d;
  return fma(fma(-q, d, x), inv_d, q);
}

// a / b by Smith's algorithm as in ddiv, with quotients of that kind, where the exponents keep
// them far from overflow and underflow (|a| and |b| within 2^+-450); ddiv elsewhere.  Largest
// and root mean square error over random pairs, in units of 2^-53 |a / b|: 2.9 and 0.75, as
// ddiv's (a conj(b) / |b|^2 with the same reciprocals: 4.6 and 0.95).
__device__ __forceinline__ bool mid_range(dcx z) {
  const int e = (__double2hiint(fmax(fabs(z.re), fabs(z.im))) >> 20) & 0x7ff;
  return (unsigned)(e - 573) <= 900u;
}
__device__ __forceinline__ dcx cdiv(dcx a, dcx b) {
  if (!mid_range(a) || !mid_range(b)) return ddiv(a, b);
  const bool swap = fabs(b.re) < fabs(b.im);
  const double p = swap ? b.im : b.re, o = swap ? b.re : b.im;
  const double r = quotient(o, p, newton_reciprocal(p)), d = fma(o, r, p), inv_d = newton_reciprocal(d);
  const double re = swap ? fma(a.re, r, a.im) : fma(a.im, r, a.re);
  const double im = swap ? fma(a.im, r, -a.re) : fma(-a.re, r, a.im);
  return {quotient(re, d, inv_d), quotient(im, d, inv_d)};
}

// The three components at a surface cell, rows of n words (complex128: one row per real
// part, complex64: one per component).
template <typename R>
struct SurfaceRows {
  static constexpr int value = sizeof(R) == 8 ? 6 : 3;
};
__device__ __forceinline__ void surface_store(Word* w, size_t n, int cell, const cx<double> v[3],
                                              unsigned long long tag) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    word_store(w + (2 * c) * n + cell, (unsigned long long)__double_as_longlong(v[c].re), tag);
    word_store(w + (2 * c + 1) * n + cell, (unsigned long long)__double_as_longlong(v[c].im), tag);
  }
}
__device__ __forceinline__ void surface_store(Word* w, size_t n, int cell, const cx<float> v[3],
                                              unsigned long long tag) {
#pragma unroll
  for (int c = 0; c < 3; ++c) word_store(w + c * n + cell, pack(v[c].re, v[c].im), tag);
}
template <typename R>
__device__ __forceinline__ bool surface_load(const Word* w, size_t n, int cell, cx<R> v[3], unsigned long long tag,
                                             int limit) {
  constexpr int NR = SurfaceRows<R>::value;
  Word a[NR];
  bool ok = false;
  int spin = 0;
  do {
#pragma unroll
    for (int q = 0; q < NR; ++q) a[q] = word_load(w + q * n + cell);
    ok = true;
#pragma unroll
    for (int q = 0; q < NR; ++q) ok = ok && a[q].tag == tag;
  } while (!ok && ++spin < limit);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if constexpr (sizeof(R) == 8) {
      v[c] = mkc<R>(__longlong_as_double((long long)a[2 * c].v), __longlong_as_double((long long)a[2 * c + 1].v));
    } else {
      v[c] = mkc<R>(__uint_as_float((unsigned)a[c].v), __uint_as_float((unsigned)(a[c].v >> 32)));
    }
  }
  return ok;
}

// Which entries of the shell list a thread reads while NRED warps wait for sums: where those
// are less than half of the CTA they read none, otherwise they come last (32^3 with 256
// threads, none / last: COCG 8.2 / 7.6 us per iteration, BiCGSTAB 9.3 / 8.6).
template <int NT, int NRED>
struct ShellReaders {
  static constexpr int waiting = 32 * NRED;
  static constexpr bool all = 2 * waiting > NT;
  static constexpr int step = all ? NT : NT - waiting;
  static __device__ __forceinline__ int first(int tid) {  // (negative: none)
    return all && tid < waiting ? tid - waiting + NT : tid - waiting;
  }
};

// Whether a launch has work.  One thread looks and the CTA follows: a CTA may start while
// others give up already.
__device__ __forceinline__ bool resident_begin(KState* st) {
  bool go = true;
  if (threadIdx.x == 0) {
    const bool lost = *(volatile const int*)&st->timed_out != 0;
    go = ld_status(st) == ST_RUNNING && !lost;
    if (lost && blockIdx.x == 0) st->status = ST_TIMEOUT;  // the host looks here between launches
  }
  return __syncthreads_and(go) != 0;
}

// ------------------------------------------------------------------ bricks
// n / d for n, d < 2^16 by a multiplication with inv = ceil(2^32 / d)
struct SmallDiv {
  unsigned inv;
  int d;
  __device__ __forceinline__ void init(int div) {
    d = div;
    inv = div > 1 ? 0xffffffffu / (unsigned)div + 1u : 0u;
  }
  __device__ __forceinline__ int div(int n) const { return d > 1 ? (int)__umulhi((unsigned)n, inv) : n; }
};

// The brick of one CTA.  Box = brick plus a one-cell shell (no shell along z on flat
// grids, where nothing varies along z), positions z fastest; H region = box without its
// high faces.
template <typename R, bool FLAT>
struct Brick {
  static constexpr int KZ = FLAT ? 0 : 1;
  int i0, j0, k0, lx, ly, lz;  // first cell, sizes
  int sz, sy;                  // box strides of z rows and y-z planes
  int own, box, hbox;
  int hz, hy;                  // H region strides
  SmallDiv by_hy, by_hz;

  __device__ __forceinline__ void init(const Geo<R>& g, const Bricks& bk) {
    int b = blockIdx.x;
    const int iz = b % bk.nz;
    b /= bk.nz;
    const int iy = b % bk.ny, ix = b / bk.ny;
    i0 = (int)((long long)ix * g.X / bk.nx);
    j0 = (int)((long long)iy * g.Y / bk.ny);
    k0 = (int)((long long)iz * g.Z / bk.nz);
    lx = (int)((long long)(ix + 1) * g.X / bk.nx) - i0;
    ly = (int)((long long)(iy + 1) * g.Y / bk.ny) - j0;
    lz = (int)((long long)(iz + 1) * g.Z / bk.nz) - k0;
    sz = lz + 2 * KZ;
    sy = (ly + 2) * sz;
    own = lx * ly * lz;
    box = (lx + 2) * sy;
    hz = lz + KZ;
    hy = (ly + 1) * hz;
    hbox = (lx + 1) * hy;
    by_hy.init(hy);
    by_hz.init(hz);
  }
};

// 1D tables of a brick's box coordinates in shared memory (x, y, z after one another)
template <typename R>
struct BrickTables {
  cx<R>* idxe[3];
  cx<R>* idxh[3];
  cx<R>* dxe[3];
  cx<R>* dxh[3];
  R* adxe[3];
  R* adxh[3];
  static __host__ __device__ size_t bytes(int bx, int by, int bz) {
    return (size_t)(bx + by + bz + 6) * (4 * sizeof(cx<R>) + 2 * sizeof(R));
  }
  __device__ __forceinline__ void carve(unsigned char* base, int bx, int by, int bz) {
    const int len[3] = {bx + 2, by + 2, bz + 2};
    const int n = len[0] + len[1] + len[2];
    cx<R>* c = reinterpret_cast<cx<R>*>(base);
    R* s = reinterpret_cast<R*>(c + 4 * n);
    int off = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      idxe[a] = c + off;
      idxh[a] = c + n + off;
      dxe[a] = c + 2 * n + off;
      dxh[a] = c + 3 * n + off;
      adxe[a] = s + off;
      adxh[a] = s + n + off;
      off += len[a];
    }
  }
  // entry t of axis a: cell (first + t) wrapped
  __device__ __forceinline__ void load(const Geo<R>& g, int a, int first, int n, int total, int tid, int nt) {
    for (int t = tid; t < n; t += nt) {
      const int i = wrapi(first + t, total);
      idxe[a][t] = g.idxe[a][i];
      idxh[a][t] = g.idxh[a][i];
      dxe[a][t] = g.dxe[a][i];
      dxh[a][t] = g.dxh[a][i];
      adxe[a][t] = g.adxe[a][i];
      adxh[a][t] = g.adxh[a][i];
    }
  }
  template <bool FLAT>
  __device__ __forceinline__ void load_all(const Geo<R>& g, const Brick<R, FLAT>& B, int nt) {
    load(g, 0, B.i0 - 1, B.lx + 2, g.X, threadIdx.x, nt);
    load(g, 1, B.j0 - 1, B.ly + 2, g.Y, threadIdx.x, nt);
    load(g, 2, B.k0 - Brick<R, FLAT>::KZ, B.lz + 2 * Brick<R, FLAT>::KZ, g.Z, threadIdx.x, nt);
  }
};

// H = pm mu^-1 ce(U) on the H region of a brick, U and Hs in shared memory (component
// stride box / hbox).  An item is two cells adjacent in x, which share a third of their
// loads: the pass is bound by shared-memory bandwidth.
template <typename R, int NT, bool FLAT, bool MAT>
__device__ __forceinline__ void brick_curl_e(const Geo<R>& g, const Brick<R, FLAT>& B, const BrickTables<R>& T,
                                             const cx<R>* U, cx<R>* Hs) {
  const cx<R>* Ux = U;
  const cx<R>* Uy = U + B.box;
  const cx<R>* Uz = U + 2 * B.box;
  const int items = ((B.lx + 2) >> 1) * B.hy;
  for (int n = threadIdx.x; n < items; n += NT) {
    const int ii = B.by_hy.div(n), rem = n - ii * B.hy, j = B.by_hz.div(rem), k = rem - j * B.hz;
    int i = 2 * ii, p = i * B.sy + j * B.sz + k;
    const cx<R> idy = T.idxe[1][j], idz = FLAT ? czero<R>() : T.idxe[2][k];
    cx<R> ux = Ux[p], uy = Uy[p], uz = Uz[p];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if (i > B.lx) break;
      const cx<R> idx = T.idxe[0][i];
      const cx<R> uyn = Uy[p + B.sy], uzn = Uz[p + B.sy];
      const cx<R> dyuz = (Uz[p + B.sz] - uz) * idy;
      const cx<R> dyux = (Ux[p + B.sz] - ux) * idy;
      const cx<R> dxuz = (uzn - uz) * idx;
      const cx<R> dxuy = (uyn - uy) * idx;
      cx<R> hx, hy, hz;
      if (FLAT) {
        hx = dyuz;
        hy = czero<R>() - dxuz;
        hz = dxuy - dyux;
      } else {
        const cx<R> dzuy = (Uy[p + 1] - uy) * idz;
        const cx<R> dzux = (Ux[p + 1] - ux) * idz;
        hx = dyuz - dzuy;
        hy = dzux - dxuz;
        hz = dxuy - dyux;
      }
      if (MAT) {
        int ci = B.i0 + i - 1, cj = B.j0 + j - 1, ck = B.k0 + k - Brick<R, FLAT>::KZ;
        ci = ci < 0 ? g.X - 1 : ci;
        cj = cj < 0 ? g.Y - 1 : cj;
        ck = ck < 0 ? g.Z - 1 : ck;
        const int cell = (ci * g.Y + cj) * g.Z + ck;
        if (g.muinv) {
          hx = __ldg(g.muinv + cell) * hx;
          hy = __ldg(g.muinv + g.N + cell) * hy;
          hz = __ldg(g.muinv + 2 * g.N + cell) * hz;
        }
        if (g.mask) {
          const uint8_t mk = __ldg(g.mask + cell);
          if (mk & 8u) hx = czero<R>();
          if (mk & 16u) hy = czero<R>();
          if (mk & 32u) hz = czero<R>();
        }
      }
      const int h = i * B.hy + rem;
      Hs[h] = hx;
      Hs[B.hbox + h] = hy;
      Hs[2 * B.hbox + h] = hz;
      if (m == 0) {
        ++i;
        p += B.sy;
        ux = Ux[p];
        uy = uyn;
        uz = uzn;
      }
    }
  }
}

// Own cells of a thread: K cells adjacent in x, the first at brick coordinates (i, j, k).
template <int K>
struct OwnCells {
  int pos, cell, n;  // box position and cell number of the first, how many there are
  int i, j, k;
  bool edge;         // the row of cells lies on a y or z face of the brick
};
template <int K, typename R, bool FLAT>
__device__ __forceinline__ OwnCells<K> own_cells(const Geo<R>& g, const Brick<R, FLAT>& B) {
  OwnCells<K> o;
  const int rows = B.ly * B.lz, ii = (int)threadIdx.x / rows, rem = (int)threadIdx.x - ii * rows;
  o.i = K * ii;
  o.j = rem / B.lz;
  o.k = rem - o.j * B.lz;
  o.n = max(0, min(K, B.lx - o.i));
  if (o.n == 0) o.i = o.j = o.k = 0;
  o.pos = (o.i + 1) * B.sy + (o.j + 1) * B.sz + o.k + Brick<R, FLAT>::KZ;
  o.cell = ((B.i0 + o.i) * g.Y + B.j0 + o.j) * g.Z + B.k0 + o.k;
  o.edge = o.j == 0 || o.j == B.ly - 1 || (!FLAT && (o.k == 0 || o.k == B.lz - 1));
  return o;
}

// y = A0 u on a thread's own cells; cells on the brick's surface also go to their words.
template <typename R, int K, bool FLAT, bool MAT>
__device__ __forceinline__ void brick_curl_h(const Geo<R>& g, const Brick<R, FLAT>& B, const BrickTables<R>& T,
                                             const cx<R>* U, const cx<R>* Hs, cx<R> w2, const OwnCells<K>& o,
                                             cx<R> (&y)[K][3], Word* surface, unsigned long long tag) {
  if (o.n == 0) return;
  const cx<R>* Hx = Hs;
  const cx<R>* Hy = Hs + B.hbox;
  const cx<R>* Hz = Hs + 2 * B.hbox;
  int h = (o.i + 1) * B.hy + (o.j + 1) * B.hz + (o.k + Brick<R, FLAT>::KZ);
  const cx<R> idyh = T.idxh[1][o.j + 1], idzh = FLAT ? czero<R>() : T.idxh[2][o.k + 1];
  cx<R> hy_prev = Hy[h - B.hy], hz_prev = Hz[h - B.hy];
  int cell = o.cell;
#pragma unroll
  for (int m = 0; m < K; ++m) {
    if (m >= o.n) break;
    const cx<R> idxh = T.idxh[0][o.i + m + 1];
    const cx<R> hx = Hx[h], hy = Hy[h], hz = Hz[h];
    if (FLAT) {
      y[m][0] = (hz - Hz[h - B.hz]) * idyh;
      y[m][1] = czero<R>() - (hz - hz_prev) * idxh;
    } else {
      y[m][0] = (hz - Hz[h - B.hz]) * idyh - (hy - Hy[h - 1]) * idzh;
      y[m][1] = (hx - Hx[h - 1]) * idzh - (hz - hz_prev) * idxh;
    }
    y[m][2] = (hy - hy_prev) * idxh - (hx - Hx[h - B.hz]) * idyh;
    const uint8_t mk = MAT && g.mask ? __ldg(g.mask + cell) : (uint8_t)0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const cx<R> v = y[m][c] - (__ldg(g.eps + c * g.N + cell) * w2) * U[c * B.box + o.pos + m * B.sy];
      y[m][c] = (mk & (1u << c)) ? czero<R>() : v;
    }
    const int i = o.i + m;
    if (o.edge || i == 0 || i == B.lx - 1) surface_store(surface, (size_t)g.N, cell, y[m], tag);
    hy_prev = hy;
    hz_prev = hz;
    h += B.hy;
    cell += g.Y * g.Z;
  }
}

// Symmetriser weights (WeightYZ of fdfd_device.cuh) from a brick's tables
template <typename R, bool FLAT, int K>
__device__ __forceinline__ void weights_yz(const BrickTables<R>& T, const OwnCells<K>& o, WeightYZ<R>& w) {
  const int j = o.j + 1, k = o.k + (FLAT ? 0 : 1);
  const cx<R> ey = T.dxe[1][j], hy = T.dxh[1][j], ez = T.dxe[2][k], hz = T.dxh[2][k];
  w.yz[0] = hy * hz;
  w.yz[1] = ey * hz;
  w.yz[2] = hy * ez;
  const R aey = T.adxe[1][j], ahy = T.adxh[1][j], aez = T.adxe[2][k], ahz = T.adxh[2][k];
  w.ayz[0] = ahy * ahz;
  w.ayz[1] = aey * ahz;
  w.ayz[2] = ahy * aez;
}

// The shell's box positions and cells, listed once per launch (the order in the list does
// not matter: each entry is updated on its own).
template <typename R, int NT, bool FLAT>
__device__ __forceinline__ void list_shell(const Geo<R>& g, const Brick<R, FLAT>& B, int2* shell, int* count) {
  for (int p = threadIdx.x; p < B.box; p += NT) {
    const int i = p / B.sy, rem = p - i * B.sy, j = rem / B.sz, k = rem - j * B.sz;
    const bool in = i >= 1 && i <= B.lx && j >= 1 && j <= B.ly && (FLAT || (k >= 1 && k <= B.lz));
    if (in) continue;
    const int ci = wrapi(B.i0 + i - 1, g.X), cj = wrapi(B.j0 + j - 1, g.Y);
    const int ck = FLAT ? B.k0 + k : wrapi(B.k0 + k - 1, g.Z);
    shell[atomicAdd(count, 1)] = make_int2(p, (ci * g.Y + cj) * g.Z + ck);
  }
}

// Shared memory of a resident solve: the box vector U, `nshell` vectors on the shell, the H
// region, the shell list, the tables and the exchange scratch (of at
// most `nred` sums at once).
struct ResidentLayout {
  size_t shell_vec, h, shell, tables, red, total;
};
// Threads of a CTA, of 128 registers each: a whole SM's (576 to 768 spill more and are slower),
// or half of them, so that two solves can share the SMs (see plan_resident).
constexpr int RES_NT = 512, RES_NT_HALF = 256;
template <typename R>
__host__ __device__ inline ResidentLayout resident_layout(int nshell, int nred, bool flat, int bx, int by, int bz,
                                                          int nt) {
  const size_t kz = flat ? 0 : 1;
  const size_t box = (size_t)(bx + 2) * (by + 2) * (bz + 2 * kz), own = (size_t)bx * by * bz;
  const size_t hbox = (size_t)(bx + 1) * (by + 1) * (bz + kz);
  ResidentLayout L;
  L.shell_vec = sizeof(cx<R>) * 3 * box;
  L.h = L.shell_vec + sizeof(cx<R>) * 3 * (box - own) * nshell;
  L.shell = (L.h + sizeof(cx<R>) * 3 * hbox + 15) & ~(size_t)15;
  L.tables = L.shell + ((sizeof(int2) * (box - own) + 15) & ~(size_t)15);
  L.red = L.tables + ((BrickTables<R>::bytes(bx, by, bz) + 15) & ~(size_t)15);
  L.total = L.red + ((size_t)nred * (nt / 4) + 2 * RES_SUMS + 2) * sizeof(double);
  return L;
}

// ------------------------------------------------------------------ COCG
// `nit` iterations of the COCG of fdfd_ops.cuh (OpCocgA / OpCocgB: the same recurrences,
// the same tests in the same order) on resident r and p:
//   p = r + beta p          own cells and shell   (x += alpha p of the step before, own)
//   q = A0 p                own cells; surface cells also to their words   -> p^T W q
//   r -= alpha q            own cells and shell (q of the shell from the words)
//                                                 -> r^T W r and the three norms
// p of the box and r of the shell are in shared memory, r and q of the K own cells of a
// thread in registers.  `surface`: two buffers (even and odd tags) of 6 N words, since the
// shell is read while the second exchange is under way.
//
// Measured per iteration, two launches / resident: 16^3 20.8 / 5.6 us, 32^3 21.9 / 7.3, 40^3
// 23.0 / 10.2, 52^3 (the largest cube that fits) 32.5 / 17.4; flat 128^2 20.0 / 5.5, 380^2 31.5 / 11.3.  It is
// bound by the exchanges (about 3 us of each iteration) and, on full bricks, by shared-memory
// bandwidth in the two curl passes.  Dividing by reciprocals (cdiv), block sums through shared
// memory and material code by template gave 0.4 to 0.7 us of it.
constexpr int COCG_SUMS = 5;
template <int NT, int K, bool FLAT, bool MAT>
__global__ void __launch_bounds__(NT, RES_NT / NT)
    k_cocg_resident(const Geo<double> g, const Bricks bk, cx<double>* r, cx<double>* p, cx<double>* x, Word* surface,
                    KState* st, ResidentScratch* gs, unsigned long long tag0, int nit, int limit) {
  using R = double;
  using C = cx<R>;
  if (!resident_begin(st)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ResidentLayout L = resident_layout<R>(1, COCG_SUMS, FLAT, bk.bx, bk.by, bk.bz, NT);
  Brick<R, FLAT> B;
  B.init(g, bk);
  C* P = reinterpret_cast<C*>(smem_raw);
  C* Rs = reinterpret_cast<C*>(smem_raw + L.shell_vec);
  C* Hs = reinterpret_cast<C*>(smem_raw + L.h);
  int2* shell = reinterpret_cast<int2*>(smem_raw + L.shell);
  BrickTables<R> T;
  T.carve(smem_raw + L.tables, bk.bx, bk.by, bk.bz);
  double* red = reinterpret_cast<double*>(smem_raw + L.red);
  double* sums = red + COCG_SUMS * RedRow<NT>::value;
  int* flags = reinterpret_cast<int*>(sums + 2 * RES_SUMS);  // [0] shell count, [1] gave up
  const int tid = threadIdx.x, N = g.N, YZ = g.Y * g.Z;
  if (tid == 0) flags[0] = flags[1] = 0;
  __syncthreads();
  list_shell<R, NT, FLAT>(g, B, shell, &flags[0]);
  T.load_all(g, B, NT);
  const OwnCells<K> o = own_cells<K>(g, B);
  __syncthreads();
  const int nshell = B.box - B.own;
  C rv[K][3];  // r of the own cells
  C t[K][3];   // q between the two exchanges, x from there to the p update
#pragma unroll
  for (int m = 0; m < K; ++m) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int idx = c * N + o.cell + m * YZ;
      if (m < o.n) P[c * B.box + o.pos + m * B.sy] = p[idx];
      rv[m][c] = m < o.n ? r[idx] : czero<R>();
      t[m][c] = czero<R>();
    }
  }
  for (int e = tid; e < nshell; e += NT) {
    const int2 sh = shell[e];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      P[c * B.box + sh.x] = p[c * N + sh.y];
      Rs[c * nshell + e] = r[c * N + sh.y];
    }
  }
  __syncthreads();  // other threads update these shell entries
  const C w2 = *g.w2p;
  // The scalar recurrences run in every thread (the sums are in shared memory, so this
  // needs no further exchange); one thread keeps the state that the host reads.
  const bool scribe = blockIdx.x == 0 && tid == 0;
  const double tol2 = st->tol2;
  const int crit = st->crit, maxiter = st->maxiter;
  double* const hist = scribe ? st->hist : nullptr;
  const double bbm = monitored_bb(st);
  const int iter0 = st->iter;
  int iter = iter0, status = ST_RUNNING;
  dcx rho = st->rho;
  double rr_pc = st->rr_pc;
  C alpha = czero<R>(), beta = from_d<R>(st->beta);
  bool owed = false;
  // shell entries go round from the first thread without own cells
  const int rows = B.ly * B.lz, items = ((B.lx + K - 1) / K) * rows;
  const int spare = tid >= items ? tid - items : tid - items + NT;
  constexpr int NRHO = COCG_SUMS;
  for (int it = 0; it < nit; ++it) {
    const unsigned long long tag = tag0 + (unsigned long long)it + 1;
    Word* const sw = surface + (tag & 1) * SurfaceRows<R>::value * (size_t)N;
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (m >= o.n) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int at = c * B.box + o.pos + m * B.sy;
        const C pv = P[at];
        if (owed) x[c * N + o.cell + m * YZ] = caxpy(alpha, pv, t[m][c]);
        P[at] = caxpy(beta, pv, rv[m][c]);
      }
    }
    for (int e = spare; e < nshell; e += NT) {
      const int pos = shell[e].x;
#pragma unroll
      for (int c = 0; c < 3; ++c) P[c * B.box + pos] = caxpy(beta, P[c * B.box + pos], Rs[c * nshell + e]);
    }
    owed = false;
    __syncthreads();
    brick_curl_e<R, NT, FLAT, MAT>(g, B, T, P, Hs);
    __syncthreads();
    brick_curl_h<R, K, FLAT, MAT>(g, B, T, P, Hs, w2, o, t, sw, tag);
    {
      double acc[2] = {0.0, 0.0};
      WeightYZ<R> wyz;
      weights_yz<R, FLAT>(T, o, wyz);
#pragma unroll
      for (int m = 0; m < K; ++m) {
        if (m >= o.n) break;
        C W[3];
        R aW[3];
        wyz.at(T.dxe[0][o.i + m + 1], T.dxh[0][o.i + m + 1], R(0), R(0), W, aW);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C wp = W[c] * P[c * B.box + o.pos + m * B.sy];
          acc[0] += wp.re * t[m][c].re - wp.im * t[m][c].im;
          acc[1] += wp.re * t[m][c].im + wp.im * t[m][c].re;
        }
      }
      sums_begin<NT, 0, 2>(acc, red, gs, tag);
    }
    if (!sums_end<0, 2>(sums, &flags[1], gs, tag, it + 1, it > 0 ? limit : SPIN_LIMIT)) { status = ST_TIMEOUT; break; }
    const dcx sigma = {sums[0], sums[1]};
    if (!dfinite(sigma)) { status = ST_NONFINITE; break; }
    if (sigma.re == 0.0 && sigma.im == 0.0) { status = ST_BREAKDOWN; break; }
    alpha = from_d<R>(cdiv(rho, sigma));
    const C malpha = mkc<R>(-alpha.re, -alpha.im);
    {
      double acc[NRHO] = {0.0, 0.0, 0.0, 0.0, 0.0};
      WeightYZ<R> wyz;
      weights_yz<R, FLAT>(T, o, wyz);
#pragma unroll
      for (int m = 0; m < K; ++m) {
        if (m >= o.n) break;
        C W[3];
        R aW[3];
        wyz.at(T.dxe[0][o.i + m + 1], T.dxh[0][o.i + m + 1], T.adxe[0][o.i + m + 1], T.adxh[0][o.i + m + 1], W, aW);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C v = caxpy(malpha, t[m][c], rv[m][c]);
          rv[m][c] = v;
          const C wr = W[c] * v;
          acc[0] += wr.re * v.re - wr.im * v.im;
          acc[1] += wr.re * v.im + wr.im * v.re;
          const double r2 = cabs2(v);
          acc[2] += r2;
          acc[3] += aW[c] * r2;
          acc[4] += aW[c] * aW[c] * r2;
        }
      }
      sums_begin<NT, 2, NRHO>(acc, red, gs, tag);
    }
    // while the sums travel: the loads of x, and the shell's r
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (m >= o.n) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) t[m][c] = x[c * N + o.cell + m * YZ];
    }
    using Readers = ShellReaders<NT, NRHO>;
    for (int e = Readers::first(tid); e >= 0 && e < nshell; e += Readers::step) {
      C qv[3];
      if (!surface_load<R>(sw, (size_t)N, shell[e].y, qv, tag, limit)) flags[1] = 1;
#pragma unroll
      for (int c = 0; c < 3; ++c) Rs[c * nshell + e] = caxpy(malpha, qv[c], Rs[c * nshell + e]);
    }
    if (!sums_end<2, NRHO>(sums + RES_SUMS, &flags[1], gs, tag, it + 1, limit)) { status = ST_TIMEOUT; break; }
    const double* sr = sums + RES_SUMS;
    const dcx rho_new = {sr[0], sr[1]};
    const double monitored = sr[2 + crit], pc = sr[3];
    const bool ok = dfinite(rho_new);
    iter += 1;
    owed = ok;
    if (ok && pc > 1e16 * rr_pc) {  // a near-zero p^T W q: the step is discarded
      owed = false;
      status = ST_BREAKDOWN;
      break;
    }
    rr_pc = pc;
    if (hist) hist[iter] = bbm > 0 ? sqrt(monitored / bbm) : 0.0;
    if (!ok || !isfinite(monitored)) status = ST_NONFINITE;
    else if (monitored <= tol2) status = ST_CONVERGED;
    else if (iter >= maxiter) status = ST_MAXITER;
    if (status != ST_RUNNING) {
      rho = rho_new;
      break;
    }
    // |rho_new| >= its larger part: the square root is needed only close to a breakdown
    const double floor_rho = BREAKDOWN_RATIO * pc;
    if (fmax(fabs(rho_new.re), fabs(rho_new.im)) <= floor_rho && dabs(rho_new) <= floor_rho) {
      status = ST_BREAKDOWN;
      break;
    }
    beta = from_d<R>(cdiv(rho_new, rho));
    rho = rho_new;
  }
#pragma unroll
  for (int m = 0; m < K; ++m) {
    if (m >= o.n) break;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int idx = c * N + o.cell + m * YZ;
      const C pv = P[c * B.box + o.pos + m * B.sy];
      if (owed) x[idx] = caxpy(alpha, pv, t[m][c]);
      p[idx] = pv;
      r[idx] = rv[m][c];
    }
  }
  if (status == ST_TIMEOUT && tid == 0) *(volatile int*)&st->timed_out = 1;
  if (scribe) {
    if (iter > iter0) {
      st->rr = sums[RES_SUMS + 2];
      st->rr_pc = sums[RES_SUMS + 3];
      st->rr_w2 = sums[RES_SUMS + 4];
    }
    st->sigma = {sums[0], sums[1]};
    st->alpha = {alpha.re, alpha.im};
    st->rho = rho;
    st->beta = {beta.re, beta.im};
    st->iter = iter;
    st->pending = 0;
    st->status = status;
  }
}

// ------------------------------------------------------------------ BiCGSTAB
// `nit` iterations of the complex64 BiCGSTAB of fdfd_ops.cuh (OpBsP / OpBsS: the same
// recurrences and tests) with r, p, v, t and x of a thread's K own cells in registers, r, p,
// v and t of the shell and the operator's input U in shared memory:
//   v = A0 p                own cells; surface cells also to their words   -> (rh, v)
//   s = r - alpha v         own cells and shell (v of the shell from the words)
//   t = A0 s                own cells, words                -> (t, s), |t|^2, (rh, t), |s|^2
//   x += alpha p + omega s, r = s - omega t, p = r + beta (p - omega v)
// A state with pending = 2 goes on from r and p in memory; otherwise p starts as r.  Both
// shells are read before the sums that their writers wait for, so each product has one
// buffer of 3 N words.
//
// Measured per iteration, two launches / resident: 16^3 26.8 / 6.3 us, 32^3 28.6 / 8.4, 40^3
// 30.1 / 9.8, 52^3 (the largest cube that fits) 39.5 / 14.4; flat 128^2 25.6 / 6.2, 380^2 35.6 / 10.2.
// Bound as COCG is: two exchanges, then shared-memory bandwidth on full bricks.
constexpr int BS_SUMS = 6;
template <int NT, int K, bool FLAT, bool MAT>
__global__ void __launch_bounds__(NT, RES_NT / NT)
    k_bicgstab_resident(const Geo<float> g, const Bricks bk, cx<float>* r, cx<float>* p, cx<float>* x, Word* surface,
                        unsigned seed, KState* st, ResidentScratch* gs, unsigned long long tag0, int nit,
                        int limit) {
  using R = float;
  using C = cx<R>;
  if (!resident_begin(st)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ResidentLayout L = resident_layout<R>(4, BS_SUMS, FLAT, bk.bx, bk.by, bk.bz, NT);
  Brick<R, FLAT> B;
  B.init(g, bk);
  C* U = reinterpret_cast<C*>(smem_raw);
  const int nshell = B.box - B.own;
  C* Rs = reinterpret_cast<C*>(smem_raw + L.shell_vec);
  C* Ps = Rs + 3 * nshell;
  C* Vs = Ps + 3 * nshell;
  C* Ts = Vs + 3 * nshell;
  C* Hs = reinterpret_cast<C*>(smem_raw + L.h);
  int2* shell = reinterpret_cast<int2*>(smem_raw + L.shell);
  BrickTables<R> T;
  T.carve(smem_raw + L.tables, bk.bx, bk.by, bk.bz);
  double* red = reinterpret_cast<double*>(smem_raw + L.red);
  double* sums = red + BS_SUMS * RedRow<NT>::value;
  int* flags = reinterpret_cast<int*>(sums + 2 * RES_SUMS);
  const int tid = threadIdx.x, N = g.N, YZ = g.Y * g.Z;
  if (tid == 0) flags[0] = flags[1] = 0;
  __syncthreads();
  list_shell<R, NT, FLAT>(g, B, shell, &flags[0]);
  T.load_all(g, B, NT);
  const OwnCells<K> o = own_cells<K>(g, B);
  __syncthreads();
  const bool resume = st->pending == 2;
  C rv[K][3], pv[K][3], vv[K][3], tv[K][3], xv[K][3], hv[K][3];
#pragma unroll
  for (int m = 0; m < K; ++m) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      rv[m][c] = pv[m][c] = vv[m][c] = tv[m][c] = xv[m][c] = hv[m][c] = czero<R>();
      if (m >= o.n) continue;
      const int idx = c * N + o.cell + m * YZ;
      rv[m][c] = r[idx];
      pv[m][c] = resume ? p[idx] : rv[m][c];
      xv[m][c] = x[idx];
      hv[m][c] = shadow<R>(idx, seed);
    }
  }
  for (int e = tid; e < nshell; e += NT) {
    const int cell = shell[e].y;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const C v = r[c * N + cell];
      Rs[c * nshell + e] = v;
      Ps[c * nshell + e] = resume ? p[c * N + cell] : v;
    }
  }
  __syncthreads();  // other threads update these shell entries
  const C w2 = *g.w2p;
  const bool scribe = blockIdx.x == 0 && tid == 0;
  const double tol2 = st->tol2;
  const int maxiter = st->maxiter, stall_limit = st->stall_limit;
  int iter = st->iter, status = ST_RUNNING, best_iter = st->best_iter;
  double best_rr = st->best_rr, rr = st->rr;
  dcx rho = st->rho;
  const size_t nw = (size_t)N;
  // shell entries go round from the first thread without own cells
  const int items = ((B.lx + K - 1) / K) * B.ly * B.lz;
  const int spare = tid >= items ? tid - items : tid - items + NT;
  constexpr int NS = 2, NT6 = BS_SUMS;
  for (int it = 0; it < nit; ++it) {
    const unsigned long long tag = tag0 + (unsigned long long)it + 1;
    C alpha, omega, beta;
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (m >= o.n) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) U[c * B.box + o.pos + m * B.sy] = pv[m][c];
    }
    for (int e = spare; e < nshell; e += NT) {
      const int pos = shell[e].x;
#pragma unroll
      for (int c = 0; c < 3; ++c) U[c * B.box + pos] = Ps[c * nshell + e];
    }
    __syncthreads();
    brick_curl_e<R, NT, FLAT, MAT>(g, B, T, U, Hs);
    __syncthreads();
    brick_curl_h<R, K, FLAT, MAT>(g, B, T, U, Hs, w2, o, vv, surface, tag);
    {
      R a[2] = {R(0), R(0)};
#pragma unroll
      for (int m = 0; m < K; ++m) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc_cdot<R>(a, hv[m][c], vv[m][c]);
      }
      double acc[NS] = {(double)a[0], (double)a[1]};
      sums_begin<NT, 0, NS>(acc, red, gs, tag);
    }
    // while the sums travel: v of the shell
    for (int e = ShellReaders<NT, NS>::first(tid); e >= 0 && e < nshell; e += ShellReaders<NT, NS>::step) {
      C q[3];
      if (!surface_load<R>(surface, nw, shell[e].y, q, tag, it > 0 ? limit : SPIN_LIMIT)) flags[1] = 1;
#pragma unroll
      for (int c = 0; c < 3; ++c) Vs[c * nshell + e] = q[c];
    }
    if (!sums_end<0, NS>(sums, &flags[1], gs, tag, it + 1, it > 0 ? limit : SPIN_LIMIT)) { status = ST_TIMEOUT; break; }
    const dcx sigma = {sums[0], sums[1]};
    if (!dfinite(sigma)) { status = ST_NONFINITE; break; }
    if ((fmax(fabs(sigma.re), fabs(sigma.im)) <= 1e-300 && dabs(sigma) <= 1e-300) ||
        (fmax(fabs(rho.re), fabs(rho.im)) <= 1e-300 && dabs(rho) <= 1e-300)) {
      status = ST_BREAKDOWN;
      break;
    }
    const dcx alpha_d = cdiv(rho, sigma);
    alpha = from_d<R>(alpha_d);
    const C malpha = mkc<R>(-alpha.re, -alpha.im);
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (m >= o.n) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        rv[m][c] = caxpy(malpha, vv[m][c], rv[m][c]);
        U[c * B.box + o.pos + m * B.sy] = rv[m][c];
      }
    }
    for (int e = spare; e < nshell; e += NT) {
      const int pos = shell[e].x;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const C s = caxpy(malpha, Vs[c * nshell + e], Rs[c * nshell + e]);
        Rs[c * nshell + e] = s;
        U[c * B.box + pos] = s;
      }
    }
    __syncthreads();
    brick_curl_e<R, NT, FLAT, MAT>(g, B, T, U, Hs);
    __syncthreads();
    brick_curl_h<R, K, FLAT, MAT>(g, B, T, U, Hs, w2, o, tv, surface + SurfaceRows<R>::value * nw, tag);
    {
      R a[NT6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
#pragma unroll
      for (int m = 0; m < K; ++m) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc_cdot<R>(a, tv[m][c], rv[m][c]);
          a[2] += cabs2(tv[m][c]);
          acc_cdot<R>(a + 3, hv[m][c], tv[m][c]);
          a[5] += cabs2(rv[m][c]);
        }
      }
      double acc[NT6];
#pragma unroll
      for (int q = 0; q < NT6; ++q) acc[q] = (double)a[q];
      sums_begin<NT, NS, NT6>(acc, red, gs, tag);
    }
    for (int e = ShellReaders<NT, NT6>::first(tid); e >= 0 && e < nshell; e += ShellReaders<NT, NT6>::step) {
      C q[3];
      if (!surface_load<R>(surface + SurfaceRows<R>::value * nw, nw, shell[e].y, q, tag, limit)) flags[1] = 1;
#pragma unroll
      for (int c = 0; c < 3; ++c) Ts[c * nshell + e] = q[c];
    }
    if (!sums_end<NS, NT6>(sums + RES_SUMS, &flags[1], gs, tag, it + 1, limit)) { status = ST_TIMEOUT; break; }
    const double* q = sums + RES_SUMS;
    const dcx ts = {q[0], q[1]}, rht = {q[3], q[4]};
    const double tt = q[2], ss = q[5];
    iter += 1;
    if (!dfinite(ts) || !isfinite(tt) || !dfinite(rht) || !isfinite(ss)) {
      status = ST_NONFINITE;
      break;
    }
    const bool small_s = ss <= tol2 || tt <= 0.0;  // s small enough (or t vanished): finish with omega = 0
    dcx om = {0.0, 0.0};
    rr = ss;
    if (!small_s) {
      const double tstt = ts.re * ts.re + ts.im * ts.im;
      double off;  // |(t, s)|^2 / |t|^2
      if (mid_range(ts) && mid_range({tt, 0.0})) {
        const double itt = newton_reciprocal(tt);
        om = {quotient(ts.re, tt, itt), quotient(ts.im, tt, itt)};
        off = quotient(tstt, tt, itt);
      } else {
        om = {ts.re / tt, ts.im / tt};
        off = tstt / tt;
      }
      rr = fmax(ss - off, 0.0);
    }
    omega = from_d<R>(om);
    if (rr <= tol2) status = ST_CONVERGED;
    else if (iter >= maxiter) status = ST_MAXITER;
    if (status == ST_RUNNING && small_s) status = ST_BREAKDOWN;
    if (status == ST_RUNNING) {
      // stagnation: no 1 % improvement on the best residual for stall_limit iterations
      if (rr < 0.98 * best_rr || iter == 1) {
        best_rr = rr;
        best_iter = iter;
      } else if (stall_limit > 0 && iter - best_iter >= stall_limit) {
        status = ST_BREAKDOWN;
      }
    }
    beta = czero<R>();
    if (status == ST_RUNNING) {
      const dcx rho_new = {-(om.re * rht.re - om.im * rht.im), -(om.re * rht.im + om.im * rht.re)};
      if ((fmax(fabs(om.re), fabs(om.im)) <= 1e-300 && dabs(om) <= 1e-300) ||
          (fmax(fabs(rho_new.re), fabs(rho_new.im)) <= 1e-300 && dabs(rho_new) <= 1e-300)) {
        status = ST_BREAKDOWN;
      } else {
        // beta = (rho_new / rho) (alpha / omega)
        beta = from_d<R>(dmul(cdiv(rho_new, rho), cdiv(alpha_d, om)));
        rho = rho_new;
      }
    }
    const C momega = mkc<R>(-omega.re, -omega.im);
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (m >= o.n) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        xv[m][c] = caxpy(omega, rv[m][c], caxpy(alpha, pv[m][c], xv[m][c]));
        rv[m][c] = caxpy(momega, tv[m][c], rv[m][c]);
        pv[m][c] = caxpy(beta, caxpy(momega, vv[m][c], pv[m][c]), rv[m][c]);
      }
    }
    if (status != ST_RUNNING) break;
    for (int e = spare; e < nshell; e += NT) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int at = c * nshell + e;
        const C rn = caxpy(momega, Ts[at], Rs[at]);
        Rs[at] = rn;
        Ps[at] = caxpy(beta, caxpy(momega, Vs[at], Ps[at]), rn);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < K; ++m) {
    if (m >= o.n) break;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int idx = c * N + o.cell + m * YZ;
      x[idx] = xv[m][c];
      p[idx] = pv[m][c];
      r[idx] = rv[m][c];
    }
  }
  if (status == ST_TIMEOUT && tid == 0) *(volatile int*)&st->timed_out = 1;
  if (scribe) {
    st->rho = rho;
    st->rr = rr;
    st->best_rr = best_rr;
    st->best_iter = best_iter;
    st->iter = iter;
    st->pending = 2;
    st->status = status;
  }
}

}  // namespace fdfd
