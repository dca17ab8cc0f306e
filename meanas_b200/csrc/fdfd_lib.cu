// Host side of libmeanas_fdfd.so: plans, solver drivers and the C ABI of
// include/meanas_fdfd.h.  All device memory comes from the caller (workspaces);
// the only allocations here are a host plan object, a private capture stream,
// two events and a few bytes of pinned host memory for convergence polling.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/meanas_fdfd.h"
#include "fdfd_csr.cuh"
#include "fdfd_fdtd.cuh"
#include "fdfd_ops.cuh"
#include "fdfd_resident.cuh"

using namespace fdfd;

// ------------------------------------------------------------------ errors
static thread_local std::string g_err;

static int set_err(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define CK(call)                                                                           \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess) return set_err(FDFD_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

#define CKL()                                                                              \
  do {                                                                                     \
    cudaError_t e_ = cudaGetLastError();                                                   \
    if (e_ != cudaSuccess) return set_err(FDFD_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e_)); \
  } while (0)

// ------------------------------------------------------------------ set-up kernels
__global__ void k_mask_bits(const double* pec, const double* pmc, uint8_t* mask, long long N) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x) {
    uint8_t m = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (pec && pec[a * N + c] != 0.0) m |= (uint8_t)(1u << a);
      if (pmc && pmc[a * N + c] != 0.0) m |= (uint8_t)(8u << a);
    }
    mask[c] = m;
  }
}

__global__ void k_recip_real(const double* src, double* dst64, float* dst32, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double v = 1.0 / src[i];
    dst64[i] = v;
    if (dst32) dst32[i] = (float)v;
  }
}

__global__ void k_set_w2(cx<double>* w64, cx<float>* w32, double re, double im) {
  *w64 = mkc<double>(re, im);
  *w32 = mkc<float>((float)re, (float)im);
}

__global__ void k_to_f32(const double* src, float* dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

// 1D tables: copies of dx, |dx|, and 1/dx (given, or computed with a scaled complex division)
__global__ void k_tables(const double2* dx, const double2* inv_given, double2* dx64, double2* inv64, double* abs64,
                         float2* dx32, float2* inv32, float* abs32, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double2 d = dx[i];
    double2 r;
    if (inv_given) {
      r = inv_given[i];
    } else {
      const dcx q = ddiv({1.0, 0.0}, {d.x, d.y});
      r = make_double2(q.re, q.im);
    }
    dx64[i] = d;
    inv64[i] = r;
    abs64[i] = hypot(d.x, d.y);
    if (dx32) {
      dx32[i] = make_float2((float)d.x, (float)d.y);
      inv32[i] = make_float2((float)r.x, (float)r.y);
      abs32[i] = (float)abs64[i];
    }
  }
}

// ------------------------------------------------------------------ plan
struct Tiling {
  int XC, ntz, nty, nxc;
  long long nblocks;
};

// Resident solve of one precision: brick split, cells per thread, launch shape (grid 0: the
// grid does not fit).
struct ResidentPlan {
  Bricks bk;
  int k, grid, nt;
  size_t smem;
};

struct GraphEntry {
  int kind;
  const void* a;
  const void* b;
  int chunk;
  cudaGraphExec_t exec;
};

struct fdfd_plan {
  int X, Y, Z;
  long long N;
  int flags;
  char* ws;                // plan workspace (caller's)
  bool has_mu, has_mask;
  cx<double> w2;           // omega^2 (host copy)
  double om_re, om_im;
  bool flat;
  bool has32;
  int nsm;
  int rb_shift;            // reductions over blocks of 2^rb_shift x planes (a grid property)
  int xc_override[2];
  int xc128;               // x planes per CTA of the complex128 passes (default_xchunk)
  CellDiv cells;
  Geo<double> g64;
  Geo<float> g32;
  cudaStream_t cap;        // private stream for graph capture
  cudaEvent_t ev[2];
  int* h_poll;             // pinned: 2 x 4 ints (crit, iter, maxiter, status)
  KState* h_state;         // pinned
  std::vector<GraphEntry> graphs;
  int launches;            // kernel launches counter for the current call
  ResidentPlan res_cocg;   // complex128 COCG
  ResidentPlan res_bs;     // complex64 BiCGSTAB
  size_t smem_optin;       // shared memory a CTA may ask for
  // optional per-kernel timing (fdfd_solve_opts.profile)
  bool profiling;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<int, std::pair<int, int>>> ev_marks;  // kind, (start idx, stop idx)
  int ev_used;
};

// Bracket one launch with timing events when profiling (kind indexes kernel_ms).
struct ProfScope {
  fdfd_plan* P;
  int kind, i0;
  cudaStream_t s;
  ProfScope(fdfd_plan* P_, int kind_, cudaStream_t s_) : P(P_), kind(kind_), i0(-1), s(s_) {
    if (!P->profiling) return;
    if (P->ev_used + 2 > (int)P->ev_pool.size()) {
      for (int k = 0; k < 256; ++k) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) return;
        P->ev_pool.push_back(e);
      }
    }
    i0 = P->ev_used;
    P->ev_used += 2;
    cudaEventRecord(P->ev_pool[i0], s);
  }
  ~ProfScope() {
    if (i0 < 0) return;
    cudaEventRecord(P->ev_pool[i0 + 1], s);
    P->ev_marks.push_back({kind, {i0, i0 + 1}});
  }
};

// Sum the recorded intervals into info (called after a stream synchronize).
static void prof_collect(fdfd_plan* P, double* ms, int* cnt) {
  for (auto& m : P->ev_marks) {
    float t = 0.f;
    if (cudaEventElapsedTime(&t, P->ev_pool[m.second.first], P->ev_pool[m.second.second]) == cudaSuccess) {
      ms[m.first] += t;
      cnt[m.first] += 1;
    }
  }
  P->ev_marks.clear();
  P->ev_used = 0;
}

static constexpr int FLAT_TY = 256;

// Resident CTAs per SM the stencil kernels are compiled for (register cap 65536 /
// (256 threads x value)): complex64 passes carry less state than complex128 ones, and those
// with one or two inputs less than the others (product 65.7 -> 61.6 us at 160x160x128, with
// mu and masks at 121x97x109 56.9 -> 43.9).  Complex128 products at three CTAs spill: 104.7 ->
// 134.0 us.
template <typename R, class Op>
struct MinBlocks {
  static constexpr int value = sizeof(R) == 8 ? 2 : (Op::NB <= 2 ? 4 : 3);
};
static constexpr int TZ3 = 32, TY3 = 8;

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// x planes per CTA for the complex128 passes: the choice (whole reduction blocks) whose CTAs,
// taken in order by the resident slots, finish first.  A CTA costs its planes and a prologue
// of about 2.5; the last chunk may be short.  The results do not depend on it (the sums run
// over a fixed partition).  COCG stencil pass, the earlier rule of about eight CTAs per SM /
// this one: 160x160x128 (16 / 48 planes) 208 / 198 us, 128^3 (8 / 32) 153 / 135, 121x97x109 with
// masks (8 / 24) 153 / 143, flat 700x613 (4 / 8) 48 / 42.  (Complex64 passes, throughput-bound at three or four CTAs per SM,
// do not follow this model and keep that rule.)
static int default_xchunk(const fdfd_plan* P) {
  const int TZ = P->flat ? 1 : TZ3, TY = P->flat ? FLAT_TY : TY3, rbp = 1 << P->rb_shift;
  const long long tiles = (long long)((P->Z + TZ - 1) / TZ) * ((P->Y + TY - 1) / TY), slots = 2LL * P->nsm;
  int best = rbp;
  double best_t = -1.0;
  for (int xc = rbp; xc <= XC_MAX; xc += rbp) {
    const double full = xc + 2.5, part = P->X % xc + 2.5;
    const long long nf = tiles * (P->X / xc);
    // full chunks first: `busy` slots end with the last round, the others one round earlier
    const long long rounds = (nf + slots - 1) / slots, busy = nf - std::max(0LL, rounds - 1) * slots;
    double t = rounds * full;
    if (P->X % xc) {
      // then the short ones, on whichever slots are free first
      double early = std::max(0.0, (rounds - 1) * full), late = rounds * full;
      long long ne = slots - busy, left = tiles;
      while (left > 0) {
        const bool on_early = ne > 0 && early <= late;
        const long long n = std::min(left, on_early ? ne : std::max(1LL, busy));
        (on_early ? early : late) += part;
        left -= n;
        t = std::max(t, on_early ? early : late);
      }
    }
    if (best_t < 0 || t < best_t) {
      best_t = t;
      best = xc;
    }
    if (xc >= P->X) break;
  }
  return best;
}

static Tiling make_tiling(const fdfd_plan* P, int precision) {
  Tiling t;
  const int TZ = P->flat ? 1 : TZ3, TY = P->flat ? FLAT_TY : TY3;
  t.ntz = (P->Z + TZ - 1) / TZ;
  t.nty = (P->Y + TY - 1) / TY;
  const long long tiles = (long long)t.ntz * t.nty;
  int xc = P->xc_override[precision];
  if (xc <= 0 && precision == 0) xc = P->xc128;
  if (xc <= 0) {
    // aim for about 8 CTAs per SM in total (two waves at 4 resident CTAs per SM)
    const long long target = 8LL * P->nsm;
    long long need = (P->X * tiles + target - 1) / target;
    xc = (int)std::max(4LL, std::min(64LL, need));
  }
  // complex128: whole blocks of the reductions' fixed plane partition per CTA (the last
  // may be short)
  if (precision == 0) {
    const int rbp = 1 << P->rb_shift;
    xc = (xc + rbp - 1) / rbp * rbp;
  }
  xc = std::min(std::min(xc, P->X), XC_MAX);
  t.XC = xc;
  t.nxc = (P->X + xc - 1) / xc;
  t.nblocks = tiles * t.nxc;
  return t;
}

template <typename R>
static Geo<R> geo_with(const Geo<R>& g, const Tiling& t) {
  Geo<R> r = g;
  r.XC = t.XC;
  r.ntz = t.ntz;
  r.nty = t.nty;
  r.nxc = t.nxc;
  return r;
}

// Partial sums of one stencil reduction: one per (block of 2^rb_shift x planes, tile).
static long long stencil_parts(const fdfd_plan* P, const Tiling& t) {
  const int rbp = 1 << P->rb_shift;
  return (long long)((P->X + rbp - 1) / rbp) * t.ntz * t.nty;
}

static long long max_blocks(const fdfd_plan* P) {
  long long m = make_tiling(P, 0).nblocks;
  m = std::max(m, make_tiling(P, 1).nblocks);
  // worst case over all x-chunk choices (the autotuner may pick XC = 1..)
  const int TZ = P->flat ? 1 : TZ3, TY = P->flat ? FLAT_TY : TY3;
  const long long tiles = (long long)((P->Z + TZ - 1) / TZ) * ((P->Y + TY - 1) / TY);
  return std::max(m, tiles * P->X);
}

// ------------------------------------------------------------------ launches
static std::mutex g_smem_mutex;

template <typename K>
static int ensure_smem(K kern, size_t bytes) {
  // Only needed above the 48 KB default.  The attribute belongs to the current
  // device, so it is remembered per (device, kernel); plans may run on several
  // host threads at once.
  static std::vector<std::pair<int, const void*>> done;
  if (bytes <= 48 * 1024) return 0;
  int dev = -1;
  CK(cudaGetDevice(&dev));
  const std::pair<int, const void*> key(dev, (const void*)kern);
  std::lock_guard<std::mutex> lock(g_smem_mutex);
  if (std::find(done.begin(), done.end(), key) != done.end()) return 0;
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  done.push_back(key);
  return 0;
}

// Launch a pass whose kernel calls pass_begin(): its CTAs may come up before the pass in
// front of it on the stream has finished.
template <class... KArgs, class... Args>
static cudaError_t launch_pass(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

template <typename R, bool FLAT, bool MAT, class Op>
static int launch_stencil_as(fdfd_plan* P, const Tiling& t, const Geo<R>& g, const Op& op, RedBuf rb, cudaStream_t s) {
  constexpr int TZ = FLAT ? 1 : TZ3, TY = FLAT ? FLAT_TY : TY3;
  using Sh = StencilShape<R, TZ, TY, FLAT, Op::NB, Op::NO>;
  auto kern = k_stencil<R, TZ, TY, FLAT, MAT, MinBlocks<R, Op>::value, Op>;
  if (int rc = ensure_smem(kern, Sh::smem_bytes(Op::NRED))) return rc;
  kern<<<(unsigned)t.nblocks, dim3(TZ, TY), Sh::smem_bytes(Op::NRED), s>>>(g, op, rb);
  P->launches++;
  CKL();
  return 0;
}

template <typename R, class Op>
static int launch_stencil(fdfd_plan* P, const Geo<R>& g0, int precision, const Op& op, RedBuf rb,
                          cudaStream_t s) {
  const Tiling t = make_tiling(P, precision);
  const Geo<R> g = geo_with(g0, t);
  const bool mat = g.muinv || g.mask;
  if (P->flat)
    return mat ? launch_stencil_as<R, true, true>(P, t, g, op, rb, s) : launch_stencil_as<R, true, false>(P, t, g, op, rb, s);
  return mat ? launch_stencil_as<R, false, true>(P, t, g, op, rb, s) : launch_stencil_as<R, false, false>(P, t, g, op, rb, s);
}

template <typename K>
static int occupancy(K kern, int threads) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, 0) != cudaSuccess || n < 1) n = 1;
  return n;
}

// CTAs for a kernel over the plan's cells: one per resident slot (`occ` per SM) at most
static unsigned point_blocks(const fdfd_plan* P, int occ) {
  return (unsigned)std::min((P->N + POINT_NT - 1) / POINT_NT, (long long)occ * P->nsm);
}

template <typename R, class Op>
static int launch_point(fdfd_plan* P, const Geo<R>& g, const Op& op, RedBuf rb, cudaStream_t s) {
  auto kern = k_point<R, Op>;
  static const int occ = occupancy(kern, POINT_NT);  // queried once
  kern<<<point_blocks(P, occ), POINT_NT, 0, s>>>(g, P->cells, op, rb);
  P->launches++;
  CKL();
  return 0;
}

// ------------------------------------------------------------------ resident solves
// Iterations per launch.  A launch of whole-SM CTAs and the kernels of a solve on another stream
// take turns, so it ends before a millisecond; half-SM CTAs run beside such kernels.  Per
// iteration of 48^3 alone, and of a 160x160x128 solve on another stream meanwhile: 256 iterations
// 12.7 and 1990 us, 64 12.9 and 1450, 32 13.4 and 1000, 16 14.4 and 700 (one more launch costs 27
// us).  The same of 128x128 with 256: 6.6 and 440 us.
static constexpr int RES_CHUNK = 64, RES_CHUNK_HALF = 256;
static constexpr int RES_CHUNK_MAX = 1 << 16;  // counters are 32 bits: CTAs x iterations of a launch
static constexpr int RES_REFUSED = 1;  // the device does not take the cooperative launch; nothing ran

// The brick split with the least work on the largest brick among those of at most one CTA of
// `nt` threads per SM that fit the shared memory with `nshell` shell vectors, at most `kmax`
// (1 or 2) own cells per thread.  Work: an own cell takes part in every pass, a shell cell and
// an H cell in one or two.
template <typename R>
static ResidentPlan split_bricks(const fdfd_plan* P, int nshell, int nred, int nt, int kmax, size_t smem_max) {
  ResidentPlan best{};
  long long best_cost = -1;
  const int most = std::min(P->nsm, RES_CTAS);
  for (int nx = 1; nx <= std::min(P->X, most); ++nx) {
    for (int ny = 1; ny <= std::min(P->Y, most / nx); ++ny) {
      for (int nz = 1; nz <= (P->flat ? 1 : std::min(P->Z, most / (nx * ny))); ++nz) {
        const int bx = (P->X + nx - 1) / nx, by = (P->Y + ny - 1) / ny, bz = (P->Z + nz - 1) / nz;
        const long long own = (long long)bx * by * bz;
        const int k = own > nt ? 2 : 1;
        if (k > kmax || (long long)((bx + k - 1) / k) * by * bz > nt) continue;
        const int kz = P->flat ? 0 : 1;
        const long long box = (long long)(bx + 2) * (by + 2) * (bz + 2 * kz);
        const long long hbox = (long long)(bx + 1) * (by + 1) * (bz + kz);
        const size_t smem = resident_layout<R>(nshell, nred, P->flat, bx, by, bz, nt).total;
        if (smem > smem_max) continue;
        const long long cost = own + box + hbox;
        if (best_cost < 0 || cost < best_cost) {
          best_cost = cost;
          best = ResidentPlan{Bricks{nx, ny, nz, bx, by, bz}, k, nx * ny * nz, nt, smem};
        }
      }
    }
  }
  return best;
}

// CTAs of half an SM where bricks of one cell per thread (two on flat grids) cover the grid,
// otherwise of a whole SM.  A launch of the latter has the GPU to itself, so solves on other
// streams take turns with it, while two of the former share the SMs.  Alone / eight at once, us per iteration of the two-launch form before, whole SM, half:
// BiCGSTAB 128x128 30 / 4.7, 6.6 / 6.3, 6.4 / 3.4; 256x256 32 / 6.6, 7.6 / 7.3, 8.1 / 5.0; COCG 24^3
// 26 / 3.9, 6.3 / 6.0, 6.1 / 3.4; 32^3 27 / 4.7, 7.7 / 7.4, 7.5 / 5.0.  Larger 3D grids gain on whole SMs
// either way: 36^3 29 / 9.2, 8.2 / 7.9, 11.3 / 6.9 (two cells per thread); 48^3 31 / 16, 12.4 / 12.2, does
// not fit.
template <typename R>
static ResidentPlan plan_resident(const fdfd_plan* P, int nshell, int nred, size_t smem_max, size_t smem_half) {
  const ResidentPlan half = split_bricks<R>(P, nshell, nred, RES_NT_HALF, P->flat ? 2 : 1, smem_half);
  return half.grid > 0 ? half : split_bricks<R>(P, nshell, nred, RES_NT, 2, smem_max);
}

template <class... KArgs, class... Args>
static int launch_resident(fdfd_plan* P, void (*kern)(KArgs...), const ResidentPlan& rp, cudaStream_t s,
                           Args... args) {
  // (the attribute is set once per kernel: to the most any plan may ask for)
  if (int rc = ensure_smem(kern, P->smem_optin)) return rc;
  std::tuple<KArgs...> a(args...);
  const cudaError_t e = std::apply(
      [&](auto&... v) {
        void* ptr[] = {(void*)&v...};
        return cudaLaunchCooperativeKernel((const void*)kern, dim3(rp.grid), dim3(rp.nt), ptr, rp.smem, s);
      },
      a);
  // a context may have fewer SMs than the device (an MPS share, a green context)
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported ||
      e == cudaErrorInvalidConfiguration) {
    cudaGetLastError();
    return RES_REFUSED;
  }
  P->launches++;
  CK(e);
  CKL();
  return 0;
}

// The instance of a resident kernel for a plan: threads, cells per thread, flat, materials (of
// the combinations that plan_resident makes).
#define RES_MAT(name, nt, k, flat, mat) ((mat) ? name<nt, k, flat, true> : name<nt, k, flat, false>)
#define RES_PICK(name, rp, flat, mat)                                                                      \
  ((rp).nt == RES_NT_HALF                                                                                  \
       ? ((flat) ? ((rp).k == 1 ? RES_MAT(name, RES_NT_HALF, 1, true, mat) : RES_MAT(name, RES_NT_HALF, 2, true, mat)) \
                 : RES_MAT(name, RES_NT_HALF, 1, false, mat))                                              \
       : ((flat) ? RES_MAT(name, RES_NT, 2, true, mat)                                                     \
                 : ((rp).k == 1 ? RES_MAT(name, RES_NT, 1, false, mat) : RES_MAT(name, RES_NT, 2, false, mat))))

static int launch_cocg_resident(fdfd_plan* P, cx<double>* r, cx<double>* p, cx<double>* x, Word* surface, KState* st,
                                ResidentScratch* gs, unsigned long long tag, int nit, int limit, cudaStream_t s) {
  const ResidentPlan& rp = P->res_cocg;
  CK(cudaMemsetAsync(gs->counter, 0, sizeof(gs->counter), s));
  return launch_resident(P, RES_PICK(k_cocg_resident, rp, P->flat, P->has_mu || P->has_mask), rp, s, P->g64, rp.bk, r,
                         p, x, surface, st, gs, tag, nit, limit);
}

static int launch_bicgstab_resident(fdfd_plan* P, cx<float>* r, cx<float>* p, cx<float>* x, Word* surface,
                                    unsigned seed, KState* st, ResidentScratch* gs, unsigned long long tag, int nit,
                                    int limit, cudaStream_t s) {
  const ResidentPlan& rp = P->res_bs;
  CK(cudaMemsetAsync(gs->counter, 0, sizeof(gs->counter), s));
  return launch_resident(P, RES_PICK(k_bicgstab_resident, rp, P->flat, P->has_mu || P->has_mask), rp, s, P->g32, rp.bk,
                         r, p, x, surface, seed, st, gs, tag, nit, limit);
}

#define TRY(x)                 \
  do {                         \
    int rc_ = (x);             \
    if (rc_ != 0) return rc_;  \
  } while (0)

// ------------------------------------------------------------------ C ABI: plan
extern "C" int fdfd_abi_version(void) { return FDFD_ABI_VERSION; }

extern "C" const char* fdfd_last_error(void) { return g_err.c_str(); }

struct PlanLayout {
  size_t consts, muinv64, muinv32, eps32, mask, tab64, tab32, total;
};

static int plan_layout(const fdfd_grid_desc* d, PlanLayout* L) {
  if (!d) return set_err(FDFD_ERR_ARG, "desc is NULL");
  for (int a = 0; a < 3; ++a)
    if (d->shape[a] < 1) return set_err(FDFD_ERR_ARG, "shape[%d] = %d must be >= 1", a, d->shape[a]);
  const long long N = (long long)d->shape[0] * d->shape[1] * d->shape[2];
  // kernels index field elements with 32-bit integers (3N < 2^31: 34 GB per complex128
  // vector, beyond what a solve's ten vectors can hold on one GPU anyway)
  if (3 * N > 2147483647LL)
    return set_err(FDFD_ERR_ARG, "grid of %lld cells is too large: 3*X*Y*Z must be < 2^31", N);
  const long long S = (long long)d->shape[0] + d->shape[1] + d->shape[2];
  const bool f32 = (d->flags & FDFD_GRID_FP32) != 0;
  size_t off = 0;
  L->consts = off;  // omega^2 (complex128, complex64)
  off += 256;
  L->muinv64 = off;
  if (d->mu) off += align256(3 * N * sizeof(double));
  L->muinv32 = off;
  if (d->mu && f32) off += align256(3 * N * sizeof(float));
  L->eps32 = off;
  if (f32) off += align256(3 * N * sizeof(float));
  L->mask = off;
  if (d->pec || d->pmc) off += align256((size_t)N);
  L->tab64 = off;
  off += align256(4 * S * sizeof(double2) + 2 * S * sizeof(double));
  L->tab32 = off;
  if (f32) off += align256(4 * S * sizeof(float2) + 2 * S * sizeof(float));
  L->total = off;
  return 0;
}

// (Re)compute everything the plan derives from a grid description into its workspace.
static void plan_fill(fdfd_plan* P, const fdfd_grid_desc* d, const PlanLayout& L, cudaStream_t s) {
  char* base = P->ws;
  const long long N = P->N;
  const int sh[3] = {P->X, P->Y, P->Z};
  // 1D tables: [dxe | dxh | idxe | idxh], each X+Y+Z long (axis-major)
  double2* t64 = (double2*)(base + L.tab64);
  float2* t32 = P->has32 ? (float2*)(base + L.tab32) : nullptr;
  const long long S = (long long)P->X + P->Y + P->Z;
  long long aoff = 0;
  double* a64 = (double*)(t64 + 4 * S);
  float* a32 = t32 ? (float*)(t32 + 4 * S) : nullptr;
  for (int a = 0; a < 3; ++a) {
    double2* dxe64 = t64 + aoff;
    double2* dxh64 = t64 + S + aoff;
    double2* ie64 = t64 + 2 * S + aoff;
    double2* ih64 = t64 + 3 * S + aoff;
    double* ae64 = a64 + aoff;
    double* ah64 = a64 + S + aoff;
    float2* dxe32 = t32 ? t32 + aoff : nullptr;
    float2* dxh32 = t32 ? t32 + S + aoff : nullptr;
    float2* ie32 = t32 ? t32 + 2 * S + aoff : nullptr;
    float2* ih32 = t32 ? t32 + 3 * S + aoff : nullptr;
    float* ae32 = a32 ? a32 + aoff : nullptr;
    float* ah32 = a32 ? a32 + S + aoff : nullptr;
    k_tables<<<(sh[a] + 255) / 256, 256, 0, s>>>((const double2*)d->dxe[a], (const double2*)d->inv_dxe[a], dxe64,
                                                 ie64, ae64, dxe32, ie32, ae32, sh[a]);
    k_tables<<<(sh[a] + 255) / 256, 256, 0, s>>>((const double2*)d->dxh[a], (const double2*)d->inv_dxh[a], dxh64,
                                                 ih64, ah64, dxh32, ih32, ah32, sh[a]);
    P->g64.dxe[a] = (const cx<double>*)dxe64;
    P->g64.dxh[a] = (const cx<double>*)dxh64;
    P->g64.idxe[a] = (const cx<double>*)ie64;
    P->g64.idxh[a] = (const cx<double>*)ih64;
    P->g64.adxe[a] = ae64;
    P->g64.adxh[a] = ah64;
    P->g32.dxe[a] = (const cx<float>*)dxe32;
    P->g32.dxh[a] = (const cx<float>*)dxh32;
    P->g32.idxe[a] = (const cx<float>*)ie32;
    P->g32.idxh[a] = (const cx<float>*)ih32;
    P->g32.adxe[a] = ae32;
    P->g32.adxh[a] = ah32;
    aoff += sh[a];
  }
  const int nb = (int)std::min<long long>((3 * N + 255) / 256, 148LL * 16);
  P->g64.eps = d->epsilon;
  P->g64.rb_shift = P->g32.rb_shift = P->rb_shift;
  P->g64.muinv = nullptr;
  P->g32.muinv = nullptr;
  P->g32.eps = nullptr;
  if (d->mu) {
    double* mi64 = (double*)(base + L.muinv64);
    float* mi32 = P->has32 ? (float*)(base + L.muinv32) : nullptr;
    k_recip_real<<<nb, 256, 0, s>>>(d->mu, mi64, mi32, 3 * N);
    P->g64.muinv = mi64;
    P->g32.muinv = mi32;
  }
  if (P->has32) {
    float* e32 = (float*)(base + L.eps32);
    k_to_f32<<<nb, 256, 0, s>>>(d->epsilon, e32, 3 * N);
    P->g32.eps = e32;
  }
  uint8_t* mask = nullptr;
  if (d->pec || d->pmc) {
    mask = (uint8_t*)(base + L.mask);
    k_mask_bits<<<nb, 256, 0, s>>>(d->pec, d->pmc, mask, N);
  }
  P->g64.mask = mask;
  P->g32.mask = mask;
  P->om_re = d->omega[0];
  P->om_im = d->omega[1];
  const double w2re = P->om_re * P->om_re - P->om_im * P->om_im;
  const double w2im = 2.0 * P->om_re * P->om_im;
  P->w2 = mkc<double>(w2re, w2im);
  cx<double>* c64p = (cx<double>*)(base + L.consts);
  cx<float>* c32p = (cx<float>*)(base + L.consts + 64);
  k_set_w2<<<1, 1, 0, s>>>(c64p, c32p, w2re, w2im);
  P->g64.w2p = c64p;
  P->g32.w2p = c32p;
  P->g64.X = P->g32.X = P->X;
  P->g64.Y = P->g32.Y = P->Y;
  P->g64.Z = P->g32.Z = P->Z;
  P->g64.N = P->g32.N = N;
}

extern "C" int fdfd_plan_workspace_bytes(const fdfd_grid_desc* desc, size_t* bytes) {
  PlanLayout L;
  TRY(plan_layout(desc, &L));
  if (!bytes) return set_err(FDFD_ERR_ARG, "bytes is NULL");
  *bytes = L.total;
  return 0;
}

extern "C" int fdfd_plan_create(const fdfd_grid_desc* d, void* ws, size_t ws_bytes, void* stream,
                                fdfd_plan** out) {
  PlanLayout L;
  TRY(plan_layout(d, &L));
  if (!out) return set_err(FDFD_ERR_ARG, "out is NULL");
  if (!d->epsilon) return set_err(FDFD_ERR_ARG, "epsilon is NULL");
  for (int a = 0; a < 3; ++a)
    if (!d->dxe[a] || !d->dxh[a]) return set_err(FDFD_ERR_ARG, "dxe/dxh[%d] is NULL", a);
  if (ws_bytes < L.total || (L.total > 0 && !ws))
    return set_err(FDFD_ERR_WORKSPACE, "plan workspace too small: %zu < %zu", ws_bytes, L.total);
  if (((uintptr_t)ws & 255) != 0) return set_err(FDFD_ERR_ARG, "plan workspace must be 256-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  fdfd_plan* P = new fdfd_plan();
  P->X = d->shape[0];
  P->Y = d->shape[1];
  P->Z = d->shape[2];
  P->N = (long long)P->X * P->Y * P->Z;
  P->flags = d->flags;
  P->om_re = d->omega[0];
  P->om_im = d->omega[1];
  P->flat = (P->Z == 1);
  P->has32 = (d->flags & FDFD_GRID_FP32) != 0;
  P->xc_override[0] = P->xc_override[1] = 0;
  // reduction blocks of 8 x planes; 4 below 2M cells, where 4-plane chunks keep more SMs busy
  P->rb_shift = P->N >= (1LL << 21) ? 3 : 2;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&P->nsm, cudaDevAttrMultiProcessorCount, dev);
  if (P->nsm <= 0) P->nsm = 148;
  {
    int coop = 0, optin = 0, per_sm = 0, reserved = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    P->smem_optin = (size_t)optin;
    const size_t half = (size_t)std::max(0, per_sm / 2 - reserved);
    if (coop) {
      P->res_cocg = plan_resident<double>(P, 1, COCG_SUMS, P->smem_optin, half);
      if (P->has32) P->res_bs = plan_resident<float>(P, 4, BS_SUMS, P->smem_optin, half);
    }
  }
  auto cleanup = [&](int rc) {
    delete P;
    return rc;
  };
  if (cudaStreamCreateWithFlags(&P->cap, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&P->ev[0], cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&P->ev[1], cudaEventDisableTiming) != cudaSuccess ||
      cudaMallocHost((void**)&P->h_poll, 8 * sizeof(int)) != cudaSuccess ||
      cudaMallocHost((void**)&P->h_state, sizeof(KState)) != cudaSuccess)
    return cleanup(set_err(FDFD_ERR_CUDA, "plan: stream/event/pinned allocation failed"));

  P->xc128 = default_xchunk(P);
  P->cells.init(P->Y, P->Z);
  P->ws = (char*)ws;
  P->has_mu = d->mu != nullptr;
  P->has_mask = (d->pec != nullptr) || (d->pmc != nullptr);
  plan_fill(P, d, L, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cleanup(set_err(FDFD_ERR_CUDA, "plan set-up kernels: %s", cudaGetErrorString(e)));
  *out = P;
  return 0;
}

extern "C" int fdfd_plan_update(fdfd_plan* P, const fdfd_grid_desc* d, void* stream) {
  if (!P || !d) return set_err(FDFD_ERR_ARG, "fdfd_plan_update: NULL argument");
  if (d->shape[0] != P->X || d->shape[1] != P->Y || d->shape[2] != P->Z || d->flags != P->flags ||
      (d->mu != nullptr) != P->has_mu || ((d->pec != nullptr) || (d->pmc != nullptr)) != P->has_mask)
    return set_err(FDFD_ERR_ARG, "fdfd_plan_update: shape, flags or optional arrays differ from the plan");
  if (!d->epsilon) return set_err(FDFD_ERR_ARG, "epsilon is NULL");
  for (int a = 0; a < 3; ++a)
    if (!d->dxe[a] || !d->dxh[a]) return set_err(FDFD_ERR_ARG, "dxe/dxh[%d] is NULL", a);
  PlanLayout L;
  TRY(plan_layout(d, &L));
  // captured iteration graphs hold the epsilon pointer: drop them if it moves
  if (d->epsilon != P->g64.eps) {
    for (auto& ge : P->graphs) cudaGraphExecDestroy(ge.exec);
    P->graphs.clear();
  }
  plan_fill(P, d, L, (cudaStream_t)stream);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(FDFD_ERR_CUDA, "plan update kernels: %s", cudaGetErrorString(e));
  return 0;
}

extern "C" int fdfd_plan_destroy(fdfd_plan* P) {
  if (!P) return 0;
  for (auto e : P->ev_pool) cudaEventDestroy(e);
  for (auto& ge : P->graphs) cudaGraphExecDestroy(ge.exec);
  if (P->cap) cudaStreamDestroy(P->cap);
  cudaEventDestroy(P->ev[0]);
  cudaEventDestroy(P->ev[1]);
  if (P->h_poll) cudaFreeHost(P->h_poll);
  if (P->h_state) cudaFreeHost(P->h_state);
  delete P;
  return 0;
}

extern "C" int fdfd_plan_set_xchunk(fdfd_plan* P, int32_t precision, int32_t xchunk) {
  if (!P || (precision != FDFD_C128 && precision != FDFD_C64) || xchunk < 0)
    return set_err(FDFD_ERR_ARG, "bad arguments to fdfd_plan_set_xchunk");
  P->xc_override[precision] = xchunk;
  for (auto& ge : P->graphs) cudaGraphExecDestroy(ge.exec);
  P->graphs.clear();
  return 0;
}

extern "C" int fdfd_plan_resident(const fdfd_plan* P, int32_t method) {
  if (!P || method < FDFD_METHOD_COCG || method > FDFD_METHOD_BICGSTAB)
    return set_err(FDFD_ERR_ARG, "bad arguments to fdfd_plan_resident");
  return method == FDFD_METHOD_COCG ? P->res_cocg.grid : (method == FDFD_METHOD_MIXED ? P->res_bs.grid : 0);
}

// ------------------------------------------------------------------ apply
extern "C" int fdfd_apply(fdfd_plan* P, int32_t op, int32_t precision, const void* x, void* y, void* stream) {
  if (!P || !x || !y) return set_err(FDFD_ERR_ARG, "fdfd_apply: NULL argument");
  if (op < FDFD_OP_A0 || op > FDFD_OP_SYM_H) return set_err(FDFD_ERR_ARG, "fdfd_apply: bad op %d", op);
  if (x == y) return set_err(FDFD_ERR_ARG, "fdfd_apply: x and y must not alias");
  cudaStream_t s = (cudaStream_t)stream;
  P->launches = 0;
  RedBuf rb{nullptr, nullptr};
  if (precision == FDFD_C128) {
    if (op == FDFD_OP_A0)
      return launch_stencil<double>(P, P->g64, 0, OpApply<double, false>{(const cx<double>*)x, (cx<double>*)y, op, P->g64}, rb, s);
    return launch_stencil<double>(P, P->g64, 0, OpApply<double, true>{(const cx<double>*)x, (cx<double>*)y, op, P->g64}, rb, s);
  }
  if (precision == FDFD_C64) {
    if (!P->has32) return set_err(FDFD_ERR_ARG, "fdfd_apply: plan built without FDFD_GRID_FP32");
    if (op == FDFD_OP_A0)
      return launch_stencil<float>(P, P->g32, 1, OpApply<float, false>{(const cx<float>*)x, (cx<float>*)y, op, P->g32}, rb, s);
    return launch_stencil<float>(P, P->g32, 1, OpApply<float, true>{(const cx<float>*)x, (cx<float>*)y, op, P->g32}, rb, s);
  }
  return set_err(FDFD_ERR_ARG, "fdfd_apply: bad precision %d", precision);
}

// ------------------------------------------------------------------ workspaces
// Every method keeps b (complex128) and, for its refinement loop, a complex128
// partner of E plus eight vectors of the inner BiCGSTAB (R0 R1 V0 V1 P0 P1 T D) in
// the inner precision.  COCG also needs r, q, P0, P1, which its breakdown
// fallback (complex128 BiCGSTAB) reuses as R0, R1, P0, P1.
struct SolveLayout {
  size_t state, ticket, scratch, partials, resid, b, e2, cocg[4], inner[8], total;
};

static void solve_layout(const fdfd_plan* P, const fdfd_solve_opts* o, SolveLayout* L) {
  const long long N = P->N;
  const size_t c128 = align256(3 * N * sizeof(double2));
  const size_t c64 = align256(3 * N * sizeof(float2));
  size_t off = 0;
  L->state = off;
  off += align256(2 * sizeof(KState));
  L->ticket = off;
  off += 256;
  L->resid = off;
  off += 256;
  L->scratch = off;
  off += align256(sizeof(ResidentScratch));
  L->partials = off;
  off += align256((size_t)max_blocks(P) * 8 * sizeof(double));
  L->b = off;
  off += c128;
  L->e2 = off;
  off += c128;
  if (o->method == FDFD_METHOD_COCG) {
    for (int i = 0; i < 4; ++i) { L->cocg[i] = off; off += c128; }
    const int reuse[8] = {0, 1, -1, -1, 2, 3, -1, -1};
    for (int i = 0; i < 8; ++i) {
      if (reuse[i] >= 0) { L->inner[i] = L->cocg[reuse[i]]; } else { L->inner[i] = off; off += c128; }
    }
  } else {
    const size_t v = (o->method == FDFD_METHOD_MIXED) ? c64 : c128;
    for (int i = 0; i < 4; ++i) L->cocg[i] = 0;
    for (int i = 0; i < 8; ++i) { L->inner[i] = off; off += v; }
  }
  L->total = off;
}

static int check_opts(const fdfd_plan* P, const fdfd_solve_opts* o) {
  if (!P || !o) return set_err(FDFD_ERR_ARG, "NULL plan or opts");
  if (o->method < FDFD_METHOD_COCG || o->method > FDFD_METHOD_BICGSTAB)
    return set_err(FDFD_ERR_ARG, "bad method %d", o->method);
  if (o->criterion != FDFD_CRIT_TRUE && o->criterion != FDFD_CRIT_PRECOND)
    return set_err(FDFD_ERR_ARG, "bad criterion %d", o->criterion);
  if (o->maxiter < 0 || !(o->rtol >= 0) || !(o->atol >= 0)) return set_err(FDFD_ERR_ARG, "bad tolerances/maxiter");
  if (o->method == FDFD_METHOD_MIXED && !P->has32)
    return set_err(FDFD_ERR_ARG, "MIXED needs a plan built with FDFD_GRID_FP32");
  return 0;
}

extern "C" int fdfd_solve_workspace_bytes(const fdfd_plan* P, const fdfd_solve_opts* o, size_t* bytes) {
  TRY(check_opts(P, o));
  if (!bytes) return set_err(FDFD_ERR_ARG, "bytes is NULL");
  SolveLayout L;
  solve_layout(P, o, &L);
  *bytes = L.total;
  return 0;
}

extern "C" int fdfd_residual_workspace_bytes(const fdfd_plan* P, size_t* bytes) {
  if (!P || !bytes) return set_err(FDFD_ERR_ARG, "NULL argument");
  *bytes = 512 + align256((size_t)max_blocks(P) * 8 * sizeof(double));
  return 0;
}

// A reduction buffer before its first pass: ticket zero, `n` partial sums unwritten.  (Every
// pass leaves it like that again.)
static int red_init(RedBuf rb, size_t n, cudaStream_t s) {
  CK(cudaMemsetAsync(rb.ticket, 0, sizeof(unsigned int), s));
  CK(cudaMemsetAsync(rb.partials, 0xff, n * sizeof(double), s));
  return 0;
}

static int residual_into(fdfd_plan* P, const void* E, const void* J, int adjoint, double* d_out, RedBuf rb,
                         cudaStream_t s) {
  OpResidual<double> o{(const cx<double>*)E, (const cx<double>*)J, P->om_re, P->om_im, adjoint, P->g64, d_out};
  return launch_stencil<double>(P, P->g64, 0, o, rb, s);
}

extern "C" int fdfd_residual(fdfd_plan* P, const void* E, const void* J, double out[4], void* ws, size_t ws_bytes,
                             void* stream) {
  size_t need = 0;
  TRY(fdfd_residual_workspace_bytes(P, &need));
  if (!E || !J || !out || !ws) return set_err(FDFD_ERR_ARG, "fdfd_residual: NULL argument");
  if (ws_bytes < need) return set_err(FDFD_ERR_WORKSPACE, "residual workspace too small: %zu < %zu", ws_bytes, need);
  if (((uintptr_t)ws & 255) != 0) return set_err(FDFD_ERR_ARG, "residual workspace must be 256-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  char* base = (char*)ws;
  unsigned int* ticket = (unsigned int*)base;
  double* d_out = (double*)(base + 256);
  RedBuf rb{(double*)(base + 512), ticket};
  P->launches = 0;
  TRY(red_init(rb, (size_t)stencil_parts(P, make_tiling(P, 0)) * OpResidual<double>::NRED, s));
  TRY(residual_into(P, E, J, 0, d_out, rb, s));
  CK(cudaMemcpyAsync(P->h_state, d_out, 4 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const double* h = (const double*)P->h_state;
  for (int i = 0; i < 4; ++i) out[i] = std::sqrt(h[i]);
  return 0;
}

// ------------------------------------------------------------------ iteration driver
// Runs `body` (which enqueues one batch of iterations) until the device state
// leaves ST_RUNNING.  Batches are enqueued one ahead of the convergence check, so
// the GPU never idles while the host polls; kernels of a batch that starts after
// convergence return at once (they test the status first).
template <class Body>
static int drive(fdfd_plan* P, KState* d_st, int chunk, int maxiter, cudaStream_t s, Body body) {
  int* hp = P->h_poll;
  const int max_batches = maxiter / chunk + 3;
  int b = 0;
  for (;;) {
    TRY(body());
    CK(cudaMemcpyAsync(hp + 4 * (b & 1), &d_st->crit, 4 * sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaEventRecord(P->ev[b & 1], s));
    if (b > 0) {
      CK(cudaEventSynchronize(P->ev[(b - 1) & 1]));
      if (hp[4 * ((b - 1) & 1) + 3] != ST_RUNNING) break;
    }
    ++b;
    if (b >= max_batches) break;
  }
  CK(cudaStreamSynchronize(s));
  return 0;
}

// Capture `enqueue` (one batch) as a CUDA graph on the private stream, cached by key
// (at most kMaxGraphs executables per plan).
static constexpr size_t kMaxGraphs = 24;

template <class Enq>
static int graph_batch(fdfd_plan* P, int kind, const void* ka, const void* kb, int chunk, cudaStream_t s,
                       Enq enqueue) {
  for (auto& ge : P->graphs) {
    if (ge.kind == kind && ge.a == ka && ge.b == kb && ge.chunk == chunk) {
      CK(cudaGraphLaunch(ge.exec, s));
      return 0;
    }
  }
  cudaGraph_t g;
  CK(cudaStreamBeginCapture(P->cap, cudaStreamCaptureModeRelaxed));
  const int saved = P->launches;
  int rc = enqueue(P->cap);
  P->launches = saved;
  cudaError_t e = cudaStreamEndCapture(P->cap, &g);
  if (rc != 0) return rc;
  if (e != cudaSuccess) return set_err(FDFD_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
  cudaGraphExec_t ex;
  e = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return set_err(FDFD_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
  // bounded cache: a long-lived plan that solves into fresh output buffers would otherwise
  // keep one executable per buffer address; the oldest entry goes first (its launches
  // were enqueued on `s` earlier, and a graph may be destroyed while it runs)
  if (P->graphs.size() >= kMaxGraphs) {
    cudaGraphExecDestroy(P->graphs.front().exec);
    P->graphs.erase(P->graphs.begin());
  }
  P->graphs.push_back({kind, ka, kb, chunk, ex});
  CK(cudaGraphLaunch(ex, s));
  return 0;
}

static KState make_state(const fdfd_solve_opts* o, int crit, int maxiter, double* hist) {
  KState h;
  memset(&h, 0, sizeof(h));
  h.crit = crit;
  h.maxiter = maxiter;
  h.rtol = o->rtol;
  h.atol = o->atol;
  h.hist = hist;
  h.status = ST_RUNNING;
  return h;
}

struct SolveCtx {
  fdfd_plan* P;
  const fdfd_solve_opts* o;
  cudaStream_t s;
  void* ws;
  KState* st;      // outer state
  KState* st_in;   // inner state
  RedBuf rb;
  ResidentScratch* scratch;  // of resident solves, and the number of their last exchange
  unsigned long long tag;
  Word* surface;   // their surface words (two buffers of all cells), null: no room for them
  int limit;       // reads of a word before a CTA of theirs gives up
  int launches_left;  // resident launches still allowed (negative: any number)
  // One launch of theirs fewer; none once a wait ran out or a launch was refused.
  bool take_launch() { return launches_left < 0 || launches_left-- > 0; }
  cx<double>* b;
  cx<double>* x;   // the caller's E
  cx<double>* e2;  // partner of E for the refinement ping-pong
  int crit, chunk;
  double tol2;     // on the monitored norm^2
  double bnorm;    // |b|
  int iters, outer, status;
  int fallbacks;   // mixed -> complex128 COCG switches
};

// iterations of one resident launch
static int resident_chunk(const ResidentPlan& rp, const fdfd_solve_opts* o) {
  if (o->chunk > 0) return std::min(o->chunk, RES_CHUNK_MAX);
  return rp.nt == RES_NT_HALF ? RES_CHUNK_HALF : RES_CHUNK;
}

static double monitored(const KState& h, int crit) { return crit == 0 ? h.rr : (crit == 1 ? h.rr_pc : h.rr_w2); }

// Refinement loop: r = b - A0 E in complex128 (exact criterion), then an inner
// BiCGSTAB in precision RI on A0 d = r / |b| to a relative reduction eta, and
// E += |b| d; repeated until the criterion holds.  E starts from the current
// content of ctx.x; the result ends in ctx.x.
template <typename RI>
static int refine_loop(SolveCtx& c, const Geo<RI>& gi, int prec, BsBufs B, double eta, int max_outer, int kind) {
  fdfd_plan* P = c.P;
  cudaStream_t s = c.s;
  const int N = (int)P->N;
  const size_t vb = 3 * (size_t)N * sizeof(cx<RI>);
  const double rscale = c.bnorm > 0 ? 1.0 / c.bnorm : 1.0;
  cx<double>* Ecur = c.x;
  cx<double>* Enext = c.e2;
  cx<RI>* D = (cx<RI>*)B.x;
  bool have_d = false;
  int local_outer = 0, no_progress = 0;
  double prev_mon = 0.0;
  for (;;) {
    // the shadow seed is baked into captured graphs, which are keyed by local_outer % 8
    const unsigned seed = 0x5eed5eedU + 0x9e3779b9U * (unsigned)(local_outer % 8);
    OpRefine<RI> rf{Ecur, have_d ? D : nullptr, Enext, c.b, (cx<RI>*)B.R0, c.bnorm, rscale, N, seed, c.st};
    TRY(launch_stencil<double>(P, P->g64, 0, rf, c.rb, s));
    std::swap(Ecur, Enext);
    CK(cudaMemcpyAsync(P->h_state, c.st, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const KState ho = *P->h_state;
    const double mon = monitored(ho, c.crit);
    if (!std::isfinite(mon)) { c.status = ST_NONFINITE; break; }
    if (mon <= c.tol2) { c.status = ST_CONVERGED; break; }
    if (c.iters >= c.o->maxiter) { c.status = ST_MAXITER; break; }
    // a refinement step must at least halve the true residual norm^2 ...
    if (local_outer > 0 && mon > 0.25 * prev_mon) ++no_progress;
    // ... or the inner precision is not enough for this problem: report it as a
    // breakdown so the caller can continue in complex128
    if (no_progress >= 2 || local_outer >= max_outer) { c.status = ST_BREAKDOWN; break; }
    const double mon_before = prev_mon;
    prev_mon = mon;
    ++local_outer;
    ++c.outer;
    KState hi = make_state(c.o, 0, std::max(1, c.o->maxiter - c.iters), nullptr);
    hi.rho = {ho.extra[0], ho.extra[1]};
    hi.rr = ho.extra[2];
    hi.bb = ho.extra[2];
    hi.tol2 = eta * eta * ho.extra[2];
    hi.stall_limit = sizeof(RI) == 4 ? 4000 : 20000;
    hi.best_rr = ho.extra[2];
    *P->h_state = hi;
    CK(cudaMemcpyAsync(c.st_in, P->h_state, sizeof(KState), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(D, 0, vb, s));
    KState* sti = c.st_in;
    RedBuf rb = c.rb;
    const int chunk = c.chunk;
    auto enqueue = [&, seed](cudaStream_t ss) -> int {
      for (int it = 0; it < chunk; ++it) {
        {
          ProfScope ps(P, 2, ss);
          OpBsP<RI> pp{B, N, seed, sti};
          TRY(launch_stencil<RI>(P, gi, prec, pp, rb, ss));
        }
        {
          ProfScope ps(P, 3, ss);
          OpBsS<RI> sp{B, N, seed, sti};
          TRY(launch_stencil<RI>(P, gi, prec, sp, rb, ss));
        }
      }
      return 0;
    };
    bool resident = false;
    int rc = 0;
    if constexpr (sizeof(RI) == 4) {
      // As for COCG, every grid that fits runs resident.  r, t and x keep their vectors (t's
      // holds p between launches); the five between lie one after another and hold the
      // surface words (96 of their 120 bytes per cell).
      resident = P->res_bs.grid > 0 && !P->profiling && c.launches_left != 0;
      if (resident) {
        Word* surface = (Word*)B.R1;
        if (local_outer == 1) CK(cudaMemsetAsync(surface, 0, 5 * vb, s));
        const int nit = resident_chunk(P->res_bs, c.o);
        rc = drive(P, sti, nit, hi.maxiter, s, [&]() -> int {
          if (!c.take_launch()) return RES_REFUSED;
          const unsigned long long tag = c.tag;
          c.tag += (unsigned long long)nit;
          return launch_bicgstab_resident(P, (cx<RI>*)B.R0, (cx<RI>*)B.T, D, surface, seed, sti, c.scratch, tag, nit, c.limit, s);
        });
        if (rc != 0 && rc != RES_REFUSED) return rc;
      }
    }
    // the shadow seed is baked into the batch, so graphs are keyed by it too
    if (!resident) TRY(drive(P, sti, chunk, hi.maxiter, s, [&]() -> int {
      if (c.o->use_graph && !P->profiling) {
        P->launches += 2 * chunk;
        return graph_batch(P, kind + 16 * (local_outer % 8), c.ws, c.x, chunk, s, enqueue);
      }
      return enqueue(s);
    }));
    if (!resident) {
      OpBsFinal<RI> fin{B, N, sti};
      TRY(launch_point<RI>(P, gi, fin, rb, s));
    }
    CK(cudaMemcpyAsync(P->h_state, sti, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (resident && (P->h_state->timed_out || (rc == RES_REFUSED && P->h_state->status == ST_RUNNING))) {
      // what the SMs held is gone or does not belong together: this correction is formed
      // again, from the field, by the two-launch form
      c.launches_left = 0;
      have_d = false;
      prev_mon = mon_before;
      --local_outer;
      --c.outer;
      continue;
    }
    c.iters += P->h_state->iter;
    if (P->h_state->status == ST_NONFINITE) { c.status = ST_NONFINITE; break; }
    have_d = true;
  }
  if (Ecur != c.x) CK(cudaMemcpyAsync(c.x, Ecur, 3 * N * sizeof(double2), cudaMemcpyDeviceToDevice, s));
  return 0;
}

// Complex128 COCG on A0 with the W bilinear form, from the iterate in c.x when
// `from_x` (else from zero), with random-perturbation restarts after a breakdown and
// complex128 BiCGSTAB refinement as the last resort.  `gkind` keys its graphs.
static int cocg_loop(SolveCtx& c, cx<double>* r, cx<double>* q, cx<double>* P0, cx<double>* P1, BsBufs B,
                     bool from_x, int gkind) {
  fdfd_plan* P = c.P;
  const fdfd_solve_opts* o = c.o;
  cudaStream_t s = c.s;
  const int N = (int)P->N;
  const size_t vbytes128 = 3 * (size_t)N * sizeof(double2);
  const int maxiter = o->maxiter;
  CK(cudaMemsetAsync(P0, 0, vbytes128, s));
  {
    OpCocgInit<double> op{c.b, from_x ? c.x : nullptr, r, N, c.st, 0.0, 0U, nullptr};
    TRY(launch_stencil<double>(P, P->g64, 0, op, c.rb, s));
  }
  KState* st = c.st;
  RedBuf rb = c.rb;
  const int chunk = c.chunk;
  cx<double>* x = c.x;
  // x updates two at a time (see OpCocgA): from a million cells on the five vectors of a pass
  // (240 MB) no longer fit L2
  const bool two = P->N >= (1LL << 20) && !P->has_mu && !P->has_mask;
  auto enqueue = [&](cudaStream_t ss) -> int {
    for (int it = 0; it < chunk; ++it) {
      {
        ProfScope ps(P, 0, ss);
        if (two) {
          OpCocgA<double, true> a{r, P0, P1, x, q, N, st};
          TRY(launch_stencil<double>(P, P->g64, 0, a, rb, ss));
        } else {
          OpCocgA<double, false> a{r, P0, P1, x, q, N, st};
          TRY(launch_stencil<double>(P, P->g64, 0, a, rb, ss));
        }
      }
      {
        ProfScope ps(P, 1, ss);
        OpCocgB<double> bb{r, q, N, st};
        TRY(launch_point<double>(P, P->g64, bb, rb, ss));
      }
    }
    return 0;
  };
  // Every grid that fits runs resident: alone it is 1.9 to 3.7 times faster than the two launches
  // up to the largest that do (52^3 and 380^2 cells, see k_cocg_resident), and with others in
  // flight faster too (see plan_resident).  The two-launch form
  // stays for larger grids, for profiling (which times its passes) and where the caller's
  // workspace has no room for the surface words (the fallback of the mixed solver), and takes
  // over where a cooperative launch is refused or a wait in one ran out.
  bool resident = c.surface && P->res_cocg.grid > 0 && !P->profiling && c.launches_left != 0;
  // A sequence started anew on the device counts on from c.iters: shift its cap and history.
  auto count_on = [&]() -> int {
    KState* hs = P->h_state;
    CK(cudaMemcpyAsync(hs, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    hs->maxiter = maxiter - c.iters;
    hs->hist = o->history ? o->history + c.iters : nullptr;
    hs->timed_out = 0;
    CK(cudaMemcpyAsync(st, hs, sizeof(KState), cudaMemcpyHostToDevice, s));
    return 0;
  };
  int restarts = 0;
  for (;;) {
    int rc = 0;
    CK(cudaMemcpyAsync(P->h_state, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const int left = maxiter - c.iters;
    if (resident && P->h_state->status == ST_RUNNING && left > 0) {
      const int nit = resident_chunk(P->res_cocg, o);
      rc = drive(P, st, nit, left, s, [&]() -> int {
        if (!c.take_launch()) return RES_REFUSED;
        const unsigned long long tag = c.tag;
        c.tag += (unsigned long long)nit;
        return launch_cocg_resident(P, r, P0, x, c.surface, st, c.scratch, tag, nit, c.limit, s);
      });
      if (rc != 0 && rc != RES_REFUSED) return rc;
    } else if (P->h_state->status == ST_RUNNING && left > 0) {
      TRY(drive(P, st, chunk, left, s, [&]() -> int {
        if (o->use_graph && !P->profiling) {
          P->launches += 2 * chunk;
          return graph_batch(P, gkind, c.ws, c.x, chunk, s, enqueue);
        }
        return enqueue(s);
      }));
    }
    if (!resident) {  // (a resident launch leaves no update owed)
      OpCocgFinal<double> fin{P0, P1, x, N, st};
      TRY(launch_point<double>(P, P->g64, fin, rb, s));
    }
    CK(cudaMemcpyAsync(P->h_state, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (resident && (P->h_state->timed_out || (rc == RES_REFUSED && P->h_state->status == ST_RUNNING))) {
      // The bricks may be a step apart, but any field is one to go on from: its residual, and
      // the two-launch form.  A step that not all CTAs took does not count.
      const int lost = P->h_state->timed_out && P->h_state->status != ST_TIMEOUT;
      c.iters += std::max(0, P->h_state->iter - lost);
      c.launches_left = 0;
      resident = false;
      OpCocgInit<double> op{c.b, x, r, N, st, 0.0, 0U, nullptr};
      TRY(launch_stencil<double>(P, P->g64, 0, op, rb, s));
      CK(cudaMemsetAsync(P0, 0, vbytes128, s));
      TRY(count_on());
      continue;
    }
    c.iters += P->h_state->iter;
    c.status = P->h_state->status;
    if (c.status == ST_RUNNING) c.status = ST_MAXITER;
    if (c.status != ST_BREAKDOWN || restarts >= 8 || c.iters >= maxiter) break;
    // Breakdown: the unconjugated form cancelled (for example a source whose
    // r^T W r is exactly zero).  Restart COCG from x + s xi, xi a hashed random
    // vector with |A0 s xi| = 0.1 |r|, which makes the new residual generic.
    ++restarts;
    const double rr_before = std::max(P->h_state->rr, 1e-300);
    const unsigned seed = 0xc0c6U + 0x9e3779b9U * (unsigned)restarts;
    {
      OpCocgInit<double> probe{nullptr, nullptr, q, N, st, 1.0, seed, nullptr};
      TRY(launch_stencil<double>(P, P->g64, 0, probe, rb, s));
    }
    CK(cudaMemcpyAsync(P->h_state, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const double axi = std::sqrt(std::max(P->h_state->rr, 1e-300));
    const double scale = 0.1 * std::sqrt(rr_before) / axi;
    {
      OpCocgInit<double> op{c.b, x, r, N, st, scale, seed, c.e2};
      TRY(launch_stencil<double>(P, P->g64, 0, op, rb, s));
    }
    CK(cudaMemcpyAsync(x, c.e2, vbytes128, cudaMemcpyDeviceToDevice, s));
    CK(cudaMemsetAsync(P0, 0, vbytes128, s));
    TRY(count_on());
  }
  if (c.status == ST_BREAKDOWN || c.status == ST_NONFINITE) {
    // still stuck: continue from the current iterate with complex128 BiCGSTAB
    // inside the refinement loop (restarting with fresh shadow vectors).
    if (c.status == ST_NONFINITE) CK(cudaMemsetAsync(c.x, 0, vbytes128, s));
    c.status = ST_RUNNING;
    TRY(refine_loop<double>(c, P->g64, 0, B, 1e-10, 64, 2 + 1000 * c.o->method));
  }
  return 0;
}

// ------------------------------------------------------------------ solve
extern "C" int fdfd_solve(fdfd_plan* P, const fdfd_solve_opts* o, const void* J, void* E, void* ws,
                          size_t ws_bytes, fdfd_solve_info* info, void* stream) {
  TRY(check_opts(P, o));
  if (!J || !E || !ws) return set_err(FDFD_ERR_ARG, "fdfd_solve: NULL J, E or workspace");
  if (((uintptr_t)ws & 255) != 0) return set_err(FDFD_ERR_ARG, "solve workspace must be 256-byte aligned");
  SolveLayout L;
  solve_layout(P, o, &L);
  if (ws_bytes < L.total) return set_err(FDFD_ERR_WORKSPACE, "solve workspace too small: %zu < %zu", ws_bytes, L.total);
  cudaStream_t s = (cudaStream_t)stream;
  P->launches = 0;
  P->profiling = o->profile != 0;
  P->ev_marks.clear();
  P->ev_used = 0;
  char* base = (char*)ws;
  const int N = (int)P->N;
  const size_t vbytes128 = 3 * (size_t)N * sizeof(double2);

  SolveCtx c;
  c.P = P;
  c.o = o;
  c.s = s;
  c.ws = ws;
  c.st = (KState*)(base + L.state);
  c.st_in = c.st + 1;
  unsigned int* ticket = (unsigned int*)(base + L.ticket);
  double* d_res = (double*)(base + L.resid);
  c.rb = RedBuf{(double*)(base + L.partials), ticket};
  c.scratch = (ResidentScratch*)(base + L.scratch);
  c.tag = 0;
  c.surface = nullptr;
  c.limit = o->wait_limit > 0 ? o->wait_limit : SPIN_LIMIT;
  c.launches_left = o->wait_limit < 0 ? -(o->wait_limit + 1) : -1;
  c.b = (cx<double>*)(base + L.b);
  c.x = (cx<double>*)E;
  c.e2 = (cx<double>*)(base + L.e2);
  c.crit = (o->criterion == FDFD_CRIT_PRECOND) ? 1 : (o->adjoint ? 2 : 0);
  c.chunk = o->chunk > 0 ? o->chunk : 16;
  c.iters = 0;
  c.outer = 0;
  c.status = ST_RUNNING;
  c.fallbacks = 0;
  const int maxiter = o->maxiter;
  BsBufs B;
  B.R0 = base + L.inner[0];
  B.R1 = base + L.inner[1];
  B.V0 = base + L.inner[2];
  B.V1 = base + L.inner[3];
  B.P0 = base + L.inner[4];
  B.P1 = base + L.inner[5];
  B.T = base + L.inner[6];
  B.x = base + L.inner[7];

  KState h = make_state(o, c.crit, maxiter, o->history);
  *P->h_state = h;
  TRY(red_init(c.rb, (size_t)max_blocks(P) * 8, s));
  CK(cudaMemsetAsync(c.scratch, 0, sizeof(ResidentScratch), s));
  CK(cudaMemcpyAsync(c.st, P->h_state, sizeof(KState), cudaMemcpyHostToDevice, s));
  // right-hand side (and guess) in the solve space; E holds the iterate
  {
    OpRhs<double> op{(const cx<double>*)J, o->has_guess ? (const cx<double>*)E : nullptr, c.b, c.x,
                     P->om_re, P->om_im, o->adjoint, P->g64.mask, N, c.st};
    TRY(launch_point<double>(P, P->g64, op, c.rb, s));
  }
  if (!o->has_guess) CK(cudaMemsetAsync(E, 0, vbytes128, s));
  CK(cudaMemcpyAsync(P->h_state, c.st, sizeof(KState), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  {
    const KState hb = *P->h_state;
    const double bbm = c.crit == 0 ? hb.bb : (c.crit == 1 ? hb.bb_pc : hb.bb_w2);
    c.tol2 = std::max(o->rtol * o->rtol * bbm, o->atol * o->atol);
    c.bnorm = std::sqrt(hb.bb);
  }

  if (o->method == FDFD_METHOD_COCG) {
    cx<double>* r = (cx<double>*)(base + L.cocg[0]);
    cx<double>* q = (cx<double>*)(base + L.cocg[1]);
    cx<double>* P0 = (cx<double>*)(base + L.cocg[2]);
    cx<double>* P1 = (cx<double>*)(base + L.cocg[3]);
    if (P->res_cocg.grid > 0) {
      // V0, V1, T and D of the fallback lie one after another and are free until it runs
      c.surface = (Word*)B.V0;
      CK(cudaMemsetAsync(c.surface, 0, 4 * vbytes128, s));
    }
    TRY(cocg_loop(c, r, q, P0, P1, B, o->has_guess != 0, 0));
  } else if (o->method == FDFD_METHOD_MIXED) {
    const double eta = o->inner_rtol > 0 ? o->inner_rtol : 1e-2;
    const int max_outer = o->max_outer > 0 ? o->max_outer : 64;
    TRY(refine_loop<float>(c, P->g32, 1, B, eta, max_outer, 1 + 1000 * o->method));
    if (c.status == ST_BREAKDOWN && c.iters < maxiter) {
      // the complex64 inner solves stopped making progress: finish with complex128
      // COCG from the current iterate, in the inner solver's memory (eight complex64
      // vectors hold four complex128 ones)
      cx<double>* r = (cx<double>*)(base + L.inner[0]);
      cx<double>* q = (cx<double>*)(base + L.inner[2]);
      cx<double>* P0 = (cx<double>*)(base + L.inner[4]);
      cx<double>* P1 = (cx<double>*)(base + L.inner[6]);
      c.status = ST_RUNNING;
      ++c.fallbacks;
      TRY(cocg_loop(c, r, q, P0, P1, B, true, 3 + 1000 * o->method));
    }
  } else {
    const double eta = o->inner_rtol > 0 ? o->inner_rtol : 1e-10;
    const int max_outer = o->max_outer > 0 ? o->max_outer : 64;
    TRY(refine_loop<double>(c, P->g64, 0, B, eta, max_outer, 2 + 1000 * o->method));
  }

  if (o->adjoint) {
    OpAdjPost<double> post{c.x, N};
    TRY(launch_point<double>(P, P->g64, post, c.rb, s));
  }
  // final FP64 check against the unmasked right-hand side
  TRY(residual_into(P, E, J, o->adjoint, d_res, c.rb, s));
  CK(cudaMemcpyAsync(P->h_state, d_res, 4 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  double hr[4];
  memcpy(hr, P->h_state, sizeof(hr));
  if (info) {
    for (int k = 0; k < 4; ++k) {
      info->kernel_ms[k] = 0.0;
      info->kernel_count[k] = 0;
    }
    if (P->profiling) prof_collect(P, info->kernel_ms, info->kernel_count);
    info->status = c.status;
    info->iterations = c.iters;
    info->outer_iterations = c.outer;
    info->kernel_launches = P->launches;
    info->residual = hr[2] > 0 ? std::sqrt(hr[0] / hr[2]) : std::sqrt(hr[0]);
    info->residual_pc = hr[3] > 0 ? std::sqrt(hr[1] / hr[3]) : std::sqrt(hr[1]);
  }
  P->profiling = false;
  return c.status == ST_CONVERGED ? 0 : c.status;
}

// ------------------------------------------------------------------ gradient
extern "C" int fdfd_eps_gradient(fdfd_plan* P, const void* E, const void* E_adj, double* grad, void* stream) {
  if (!P || !E || !E_adj || !grad) return set_err(FDFD_ERR_ARG, "fdfd_eps_gradient: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  P->launches = 0;
  OpEpsGrad<double> op{(const cx<double>*)E, (const cx<double>*)E_adj, grad, P->w2, P->g64.mask, (int)P->N};
  return launch_point<double>(P, P->g64, op, RedBuf{nullptr, nullptr}, s);
}

// ------------------------------------------------------------------ E -> H, Poynting
extern "C" int fdfd_e2h(fdfd_plan* P, const void* E, void* H, void* S, int32_t flags, void* stream) {
  if (!P || !E) return set_err(FDFD_ERR_ARG, "fdfd_e2h: NULL plan or E");
  if (!H && !S) return set_err(FDFD_ERR_ARG, "fdfd_e2h: both outputs are NULL");
  if (flags & ~(FDFD_E2H_CONJ | FDFD_E2H_H_IN)) return set_err(FDFD_ERR_ARG, "fdfd_e2h: unknown flags %d", flags);
  const int conj_h = (flags & FDFD_E2H_CONJ) != 0, h_in = (flags & FDFD_E2H_H_IN) != 0;
  if (h_in && (!H || !S)) return set_err(FDFD_ERR_ARG, "fdfd_e2h: FDFD_E2H_H_IN needs both H and S");
  const double m2 = P->om_re * P->om_re + P->om_im * P->om_im;
  if (!(m2 > 0.0)) return set_err(FDFD_ERR_ARG, "fdfd_e2h: omega is zero");
  cudaStream_t s = (cudaStream_t)stream;
  P->launches = 0;
  const cx<double> inv_miw = mkc<double>(P->om_im / m2, P->om_re / m2);  // 1 / (-i omega)
  static const int occ = occupancy(k_e2h, POINT_NT);
  k_e2h<<<point_blocks(P, occ), POINT_NT, 0, s>>>(P->g64, P->cells, (const cx<double>*)E, (cx<double>*)H, (cx<double>*)S,
                                                 inv_miw, conj_h, h_in);
  P->launches++;
  CKL();
  return 0;
}

// ------------------------------------------------------------------ TFSF / boundary sources
extern "C" int fdfd_tfsf_source(fdfd_plan* P, const void* E, const double* tf_region, void* J, int32_t flags,
                                void* stream) {
  if (!P || !E || !tf_region || !J) return set_err(FDFD_ERR_ARG, "fdfd_tfsf_source: NULL argument");
  if (E == J) return set_err(FDFD_ERR_ARG, "fdfd_tfsf_source: J must not alias E");
  if (flags & ~(FDFD_SRC_EDGES | FDFD_SRC_PERIODIC))
    return set_err(FDFD_ERR_ARG, "fdfd_tfsf_source: unknown flags %d", flags);
  if (P->has_mask)
    return set_err(FDFD_ERR_ARG, "fdfd_tfsf_source: the source operator has no PEC/PMC; use a plan without masks");
  const double m2 = P->om_re * P->om_re + P->om_im * P->om_im;
  if (!(m2 > 0.0)) return set_err(FDFD_ERR_ARG, "fdfd_tfsf_source: omega is zero");
  cudaStream_t s = (cudaStream_t)stream;
  P->launches = 0;
  OpTfsf<double> op{(const cx<double>*)E, tf_region, (cx<double>*)J, 0, (flags & FDFD_SRC_EDGES) != 0,
                    (flags & FDFD_SRC_PERIODIC) != 0, mkc<double>(P->om_im / m2, P->om_re / m2), P->g64};
  TRY(launch_stencil<double>(P, P->g64, 0, op, RedBuf{nullptr, nullptr}, s));
  op.pass = 1;
  return launch_stencil<double>(P, P->g64, 0, op, RedBuf{nullptr, nullptr}, s);
}

// ------------------------------------------------------------------ waveguide mode source
// expand_e (meanas/fdfd/waveguide_3d.py:206-257): the mode's cross-section at index s0 of
// the propagation axis, inside the transverse window [lo, hi), repeated along the whole
// axis with the per-plane phase table; and the half-space mask compute_source builds
// (:145-152): 1 on planes [mlo, mhi) of the axis, every component and transverse cell.
__global__ void k_expand_mode(const cx<double>* __restrict__ Em, const cx<double>* __restrict__ phase,
                              cx<double>* __restrict__ Eo, double* __restrict__ mask, int X, int Y, int Z,
                              int axis, int s0, int3 lo, int3 hi, int mlo, int mhi) {
  const long long N = (long long)X * Y * Z;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 3 * N;
       t += (long long)gridDim.x * blockDim.x) {
    const long long cell = t % N;
    const int c = (int)(t / N);
    const int k = (int)(cell % Z), j = (int)((cell / Z) % Y), i = (int)(cell / ((long long)Y * Z));
    const int q[3] = {i, j, k};
    const int l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z};
    bool inside = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (a != axis && (q[a] < l3[a] || q[a] >= h3[a])) inside = false;
    cx<double> v = mkc<double>(0.0, 0.0);
    if (inside) {
      int src[3] = {i, j, k};
      src[axis] = s0;
      const cx<double> e = Em[(long long)c * N + ((long long)src[0] * Y + src[1]) * Z + src[2]];
      v = phase[q[axis]] * e;
    }
    Eo[t] = v;
    if (mask) mask[t] = (q[axis] >= mlo && q[axis] < mhi) ? 1.0 : 0.0;
  }
}

static int check_mode_slice(const fdfd_plan* P, const fdfd_mode_slice* m, const char* who) {
  if (!m) return set_err(FDFD_ERR_ARG, "%s: NULL slice description", who);
  const int n[3] = {P->X, P->Y, P->Z};
  if (m->axis < 0 || m->axis > 2) return set_err(FDFD_ERR_ARG, "%s: axis %d", who, m->axis);
  if (m->polarity != 1 && m->polarity != -1) return set_err(FDFD_ERR_ARG, "%s: polarity %d", who, m->polarity);
  for (int a = 0; a < 3; ++a)
    if (m->lo[a] < 0 || m->hi[a] > n[a] || m->lo[a] >= m->hi[a])
      return set_err(FDFD_ERR_ARG, "%s: slice [%d, %d) of axis %d outside [0, %d)", who, m->lo[a], m->hi[a], a, n[a]);
  if (m->hi[m->axis] != m->lo[m->axis] + 1)
    return set_err(FDFD_ERR_ARG, "%s: the slice must select one index along the propagation axis", who);
  if (m->mask_lo < 0 || m->mask_hi > n[m->axis] || m->mask_lo > m->mask_hi)
    return set_err(FDFD_ERR_ARG, "%s: mask planes [%d, %d) outside [0, %d)", who, m->mask_lo, m->mask_hi, n[m->axis]);
  return 0;
}

static unsigned elementwise_blocks(const fdfd_plan* P, long long n) {
  const long long need = (n + 255) / 256;
  return (unsigned)std::max(1LL, std::min(need, 8LL * P->nsm));
}

extern "C" int fdfd_mode_expand(fdfd_plan* P, const void* E_mode, const void* phase, const fdfd_mode_slice* m,
                                void* E_out, double* mask_out, void* stream) {
  if (!P || !E_mode || !phase || !E_out) return set_err(FDFD_ERR_ARG, "fdfd_mode_expand: NULL argument");
  if (E_mode == E_out) return set_err(FDFD_ERR_ARG, "fdfd_mode_expand: E_out must not alias E_mode");
  TRY(check_mode_slice(P, m, "fdfd_mode_expand"));
  k_expand_mode<<<elementwise_blocks(P, 3 * P->N), 256, 0, (cudaStream_t)stream>>>(
      (const cx<double>*)E_mode, (const cx<double>*)phase, (cx<double>*)E_out, mask_out, P->X, P->Y, P->Z,
      m->axis, m->lo[m->axis], make_int3(m->lo[0], m->lo[1], m->lo[2]), make_int3(m->hi[0], m->hi[1], m->hi[2]),
      m->mask_lo, m->mask_hi);
  P->launches = 1;
  CKL();
  return 0;
}

extern "C" int fdfd_mode_source(fdfd_plan* P, const void* E_mode, const void* phase, const fdfd_mode_slice* m,
                                void* E_work, double* mask_work, void* J, void* stream) {
  if (!P || !E_mode || !phase || !E_work || !mask_work || !J)
    return set_err(FDFD_ERR_ARG, "fdfd_mode_source: NULL argument");
  if (J == E_work || J == E_mode || E_work == E_mode)
    return set_err(FDFD_ERR_ARG, "fdfd_mode_source: J, E_work and E_mode must be distinct");
  TRY(fdfd_mode_expand(P, E_mode, phase, m, E_work, mask_work, stream));
  TRY(fdfd_tfsf_source(P, E_work, mask_work, J, FDFD_SRC_EDGES, stream));
  P->launches += 1;
  return 0;
}

// ------------------------------------------------------------------ CSR solves
static int csr_view(const fdfd_csr_desc* d, CsrView* v, const char* who) {
  if (!d) return set_err(FDFD_ERR_ARG, "%s: NULL matrix", who);
  if (d->n < 1 || d->n >= (int64_t)1 << 31) return set_err(FDFD_ERR_ARG, "%s: n = %lld out of range", who,
                                                            (long long)d->n);
  if (d->nnz < 0) return set_err(FDFD_ERR_ARG, "%s: nnz = %lld", who, (long long)d->nnz);
  if (!d->indptr || (d->nnz > 0 && (!d->indices || !d->data)))
    return set_err(FDFD_ERR_ARG, "%s: NULL CSR array", who);
  v->n = (int)d->n;
  v->indptr = (const long long*)d->indptr;
  v->indices = (const int*)d->indices;
  v->data = (const cx<double>*)d->data;
  return 0;
}

// CTAs for a CSR kernel: enough for `per_cta` rows each, at most its resident slots (a second,
// partial wave of CTAs costs a kernel of this length more than a longer loop).
static unsigned csr_blocks(int n, int per_cta, int occ) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const long long need = ((long long)n + per_cta - 1) / per_cta;
  return (unsigned)std::max(1LL, std::min(need, (long long)occ * nsm));
}
static constexpr int CSR_ROWS = CSR_NT / CSR_LPR;  // rows per CTA step
#define CSR_GRID(kern, n, per_cta)                      \
  [](int n_) {                                          \
    static const int occ = occupancy(kern, CSR_NT);     \
    return csr_blocks(n_, per_cta, occ);                \
  }(n)

extern "C" int fdfd_csr_spmv(const fdfd_csr_desc* d, const void* x, void* y, void* stream) {
  CsrView A;
  TRY(csr_view(d, &A, "fdfd_csr_spmv"));
  if (!x || !y) return set_err(FDFD_ERR_ARG, "fdfd_csr_spmv: NULL vector");
  if (x == y) return set_err(FDFD_ERR_ARG, "fdfd_csr_spmv: y must not alias x");
  k_csr_spmv<<<CSR_GRID(k_csr_spmv, A.n, CSR_ROWS), CSR_NT, 0, (cudaStream_t)stream>>>(A, (const cx<double>*)x, (cx<double>*)y);
  CKL();
  return 0;
}

struct CsrLayout {
  size_t state, ticket, partials, res, vec, total;
};

static CsrLayout csr_layout(int n) {
  CsrLayout L;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = align256(off + bytes);
    return o;
  };
  L.state = take(sizeof(KState));
  L.ticket = take(sizeof(unsigned));
  L.partials = take(sizeof(double) * 8 * (size_t)8 * 2048);  // up to 8 sums x 16k CTAs
  L.res = take(2 * sizeof(double));
  L.vec = take(4 * 16 * (size_t)n);
  L.total = off;
  return L;
}

extern "C" int fdfd_csr_solve_workspace_bytes(const fdfd_csr_desc* d, size_t* bytes) {
  CsrView A;
  TRY(csr_view(d, &A, "fdfd_csr_solve_workspace_bytes"));
  if (!bytes) return set_err(FDFD_ERR_ARG, "fdfd_csr_solve_workspace_bytes: NULL output");
  *bytes = csr_layout(A.n).total;
  return 0;
}

extern "C" int fdfd_csr_solve(const fdfd_csr_desc* d, const fdfd_solve_opts* o, const void* b, void* x, void* ws,
                              size_t ws_bytes, fdfd_solve_info* info, void* stream) {
  CsrView A;
  TRY(csr_view(d, &A, "fdfd_csr_solve"));
  if (!o || !b || !x || !ws) return set_err(FDFD_ERR_ARG, "fdfd_csr_solve: NULL argument");
  const CsrLayout L = csr_layout(A.n);
  if (ws_bytes < L.total) return set_err(FDFD_ERR_WORKSPACE, "fdfd_csr_solve: workspace %zu < %zu", ws_bytes,
                                         L.total);
  if (((uintptr_t)ws & 255) != 0) return set_err(FDFD_ERR_ARG, "fdfd_csr_solve: workspace not 256-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  char* w = (char*)ws;
  KState* st = (KState*)(w + L.state);
  RedBuf rb{(double*)(w + L.partials), (unsigned*)(w + L.ticket)};
  const size_t vb = 16 * (size_t)A.n;
  cx<double>* V = (cx<double>*)(w + L.vec);
  CsrBufs B{V, (cx<double>*)((char*)V + vb), (cx<double>*)((char*)V + 2 * vb), (cx<double>*)((char*)V + 3 * vb),
            (cx<double>*)x, (const cx<double>*)b};
  KState h{};
  h.rtol = o->rtol;
  h.atol = o->atol;
  h.maxiter = o->maxiter > 0 ? o->maxiter : 10 * A.n;
  h.status = ST_RUNNING;
  CK(cudaMemcpyAsync(st, &h, sizeof(KState), cudaMemcpyHostToDevice, s));
  const unsigned grid = CSR_GRID(k_csr_init, A.n, CSR_ROWS), grid_a = CSR_GRID(k_csr_a, A.n, CSR_ROWS);
  const unsigned grid_b = CSR_GRID(k_csr_b, A.n, CSR_ROWS), grid_c = CSR_GRID(k_csr_c, A.n, CSR_NT);
  const unsigned grid_r = CSR_GRID(k_csr_residual, A.n, CSR_ROWS);
  const unsigned seed = 0x5eed5eedU;
  int launches = 0;
  TRY(red_init(rb, (size_t)std::max({grid, grid_a, grid_b, grid_c, grid_r}) * 8, s));
  k_csr_init<<<grid, CSR_NT, 0, s>>>(A, B, o->has_guess != 0, seed, st, rb);
  CKL();
  ++launches;
  const int chunk = o->chunk > 0 ? o->chunk : 16;
  int status = ST_RUNNING, iters = 0;
  for (;;) {
    int head[4];  // crit, iter, maxiter, status
    CK(cudaMemcpyAsync(head, &st->crit, sizeof(head), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    iters = head[1];
    status = head[3];
    if (status != ST_RUNNING || iters >= h.maxiter) break;
    for (int it = 0; it < chunk; ++it) {
      CK(launch_pass(k_csr_a, grid_a, CSR_NT, 0, s, A, B, seed, st, rb));
      CK(launch_pass(k_csr_b, grid_b, CSR_NT, 0, s, A, B, seed, st, rb));
      CK(launch_pass(k_csr_c, grid_c, CSR_NT, 0, s, A, B, st, rb));
      launches += 3;
    }
  }
  if (status == ST_RUNNING) status = ST_MAXITER;
  double* res = (double*)(w + L.res);
  k_csr_residual<<<grid_r, CSR_NT, 0, s>>>(A, (const cx<double>*)x, (const cx<double>*)b, res, rb);
  CKL();
  ++launches;
  double hr[2];
  CK(cudaMemcpyAsync(hr, res, sizeof(hr), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (info) {
    *info = fdfd_solve_info{};
    info->status = status;
    info->iterations = iters;
    info->kernel_launches = launches;
    info->residual = hr[1] > 0 ? std::sqrt(hr[0] / hr[1]) : std::sqrt(hr[0]);
    info->residual_pc = info->residual;
  }
  return status == ST_CONVERGED ? 0 : status;
}

// ------------------------------------------------------------------ FDTD
static int fdtd_geo(const fdfd_fdtd_desc* d, bool estep, FdtdGeo* g, const char* who) {
  if (!d) return set_err(FDFD_ERR_ARG, "%s: NULL descriptor", who);
  for (int a = 0; a < 3; ++a) {
    if (d->shape[a] < 1) return set_err(FDFD_ERR_ARG, "%s: shape[%d] = %d", who, a, d->shape[a]);
    if (!d->dxe[a] || !d->dxh[a]) return set_err(FDFD_ERR_ARG, "%s: NULL cell widths", who);
  }
  const long long n = (long long)d->shape[0] * d->shape[1] * d->shape[2];
  if (3 * n >= (1LL << 31)) return set_err(FDFD_ERR_ARG, "%s: grid too large for 32-bit indexing", who);
  if ((d->field_type != FDFD_REAL64 && d->field_type != FDFD_REAL32) ||
      (d->psi_type != FDFD_REAL64 && d->psi_type != FDFD_REAL32))
    return set_err(FDFD_ERR_ARG, "%s: bad field or psi type", who);
  if (d->form != FDFD_FDTD_PLAIN && d->form != FDFD_FDTD_CPML) return set_err(FDFD_ERR_ARG, "%s: bad form", who);
  if (estep && !d->epsilon) return set_err(FDFD_ERR_ARG, "%s: epsilon is NULL", who);
  *g = FdtdGeo{};
  g->X = d->shape[0];
  g->Y = d->shape[1];
  g->Z = d->shape[2];
  g->by_y.init((unsigned)g->Y);
  g->table = (long long)g->X + g->Y + g->Z <= FDTD_TABLE;
  for (int a = 0; a < 3; ++a) {
    g->dxb[a] = d->dxh[a];
    g->dxf[a] = d->form == FDFD_FDTD_PLAIN ? d->dxe[a] : d->dxh[a];
  }
  g->mat = estep ? d->epsilon : d->mu;
  g->dt = d->dt;
  g->cpml = d->form == FDFD_FDTD_CPML;
  if (g->cpml) {
    for (int a = 0; a < 3; ++a) {
      for (int pp = 0; pp < 2; ++pp) {
        const fdfd_fdtd_face& f = d->face[a][pp];
        if (f.thickness == 0) continue;
        if (f.thickness < 0 || f.thickness > d->shape[a])
          return set_err(FDFD_ERR_ARG, "%s: face [%d][%d] thickness %d", who, a, pp, f.thickness);
        const double* par = estep ? f.param_e : f.param_h;
        void* const* psi = estep ? f.psi_e : f.psi_h;
        if (!par || !psi[0] || !psi[1]) return set_err(FDFD_ERR_ARG, "%s: face [%d][%d] NULL arrays", who, a, pp);
        g->face[a][pp] = CpmlFace{f.thickness, par, psi[0], psi[1]};
      }
    }
  }
  return 0;
}

template <typename R, typename P, bool ESTEP, int FACES, bool TABLE>
static int fdtd_launch_as(FdtdGeo g, void* e, void* h, cudaStream_t s) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto kern = k_fdtd<R, P, ESTEP, FACES, TABLE>;
  static const int occ = occupancy(kern, FDTD_NT);
  // one CTA per resident slot, shared between the two lists by their work (a cell inside a
  // layer along z counts 1.3: 1 to 3 measured within 8 % of one another)
  g.nz = FACES == 1 ? g.Z - g.face[2][0].th - g.face[2][1].th : g.Z;
  g.by_row[0].init((unsigned)std::max(1, g.nz));
  g.by_row[1].init((unsigned)std::max(1, g.Z - g.nz));
  const long long n1 = (long long)g.X * g.Y * g.nz, n2 = (long long)g.X * g.Y * (g.Z - g.nz);
  const long long slots = (long long)occ * nsm, need1 = (n1 + FDTD_NT - 1) / FDTD_NT;
  const long long need2 = (n2 + FDTD_NT - 1) / FDTD_NT;
  long long b2 = std::min(need2, (long long)std::ceil((double)slots * 1.3 * n2 / (n1 + 1.3 * n2)));
  const long long b1 = std::min(need1, std::max(slots - b2, (long long)(n1 > 0)));
  g.slab_blocks = (int)b2;
  kern<<<(unsigned)(b1 + b2), FDTD_NT, 0, s>>>(g, (R*)e, (R*)h);
  CKL();
  return 0;
}

template <typename R, typename P, bool ESTEP>
static int fdtd_launch(const FdtdGeo& g, void* e, void* h, cudaStream_t s) {
  // the slabs of an axis overlap only when their layers outnumber its cells
  int faces = 0;
  const int dims[3] = {g.X, g.Y, g.Z};
  for (int a = 0; a < 3; ++a) {
    const int lo = g.face[a][0].th, hi = g.face[a][1].th;
    if (lo + hi > dims[a]) faces = 2;
    else if (lo + hi > 0) faces = std::max(faces, 1);
  }
  if (g.table) {
    if (faces == 0) return fdtd_launch_as<R, P, ESTEP, 0, true>(g, e, h, s);
    if (faces == 1) return fdtd_launch_as<R, P, ESTEP, 1, true>(g, e, h, s);
    return fdtd_launch_as<R, P, ESTEP, 2, true>(g, e, h, s);
  }
  if (faces == 0) return fdtd_launch_as<R, P, ESTEP, 0, false>(g, e, h, s);
  return fdtd_launch_as<R, P, ESTEP, 2, false>(g, e, h, s);
}

template <bool ESTEP>
static int fdtd_step(const fdfd_fdtd_desc* d, void* e, void* h, void* stream, const char* who) {
  FdtdGeo g;
  TRY(fdtd_geo(d, ESTEP, &g, who));
  if (!e || !h) return set_err(FDFD_ERR_ARG, "%s: NULL field", who);
  cudaStream_t s = (cudaStream_t)stream;
  const bool f32 = d->field_type == FDFD_REAL32, p32 = d->psi_type == FDFD_REAL32;
  if (f32 && p32) return fdtd_launch<float, float, ESTEP>(g, e, h, s);
  if (f32) return fdtd_launch<float, double, ESTEP>(g, e, h, s);
  if (p32) return fdtd_launch<double, float, ESTEP>(g, e, h, s);
  return fdtd_launch<double, double, ESTEP>(g, e, h, s);
}

extern "C" int fdfd_fdtd_update_h(const fdfd_fdtd_desc* d, const void* E, void* H, void* stream) {
  return fdtd_step<false>(d, const_cast<void*>(E), H, stream, "fdfd_fdtd_update_h");
}

extern "C" int fdfd_fdtd_update_e(const fdfd_fdtd_desc* d, void* E, const void* H, void* stream) {
  return fdtd_step<true>(d, E, const_cast<void*>(H), stream, "fdfd_fdtd_update_e");
}

// ------------------------------------------------------------------ allocation-free residual
// For callers that cannot allocate device memory at all (for example code running
// under an allocator that is already exhausted or frozen, or a host application
// that owns every device buffer and hands out only inputs and outputs): the FP64
// residual check with its reduction scratch in this fixed array instead of a
// caller-provided workspace.  Every device that loads the library keeps these
// bytes until the process exits.
constexpr size_t STATIC_SCRATCH_BYTES = (size_t)1 << 20;  // 1 MiB per device
static __device__ __align__(256) unsigned char g_static_scratch[STATIC_SCRATCH_BYTES];

constexpr int STATIC_MAX_DEVICES = 64;
static std::mutex g_static_mutex;
static void* g_static_addr[STATIC_MAX_DEVICES];

// Device address of g_static_scratch on the current device (looked up once per device:
// in host code the array's name is only a host-side stand-in).
static int static_scratch_address(void** out) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= STATIC_MAX_DEVICES)
    return set_err(FDFD_ERR_ARG, "fdfd_residual_static: device %d beyond %d", dev, STATIC_MAX_DEVICES);
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess)
      return set_err(FDFD_ERR_CUDA, "fdfd_residual_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    g_static_addr[dev] = p;
  }
  *out = g_static_addr[dev];
  return 0;
}

extern "C" int fdfd_residual_static(fdfd_plan* P, const void* E, const void* J, double out[4], void* stream) {
  if (!P || !E || !J || !out) return set_err(FDFD_ERR_ARG, "fdfd_residual_static: NULL argument");
  // scratch layout: [0, 256) ticket, [256, 512) the four sums, [512, ...) partial sums
  const Tiling t = make_tiling(P, 0);
  const long long parts = stencil_parts(P, t);
  const size_t need = 512 + (size_t)parts * OpResidual<double>::NRED * sizeof(double);
  if (need > STATIC_SCRATCH_BYTES)
    return set_err(FDFD_ERR_ARG,
                   "fdfd_residual_static: the grid needs %lld partial sums (%zu scratch bytes); the fixed scratch "
                   "holds %zu bytes (at most %zu partial sums) -- use fdfd_residual with a workspace",
                   parts, need, STATIC_SCRATCH_BYTES,
                   (STATIC_SCRATCH_BYTES - 512) / (OpResidual<double>::NRED * sizeof(double)));
  void* base = nullptr;
  TRY(static_scratch_address(&base));
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char* b = (unsigned char*)base;
  unsigned int* ticket = (unsigned int*)b;
  double* d_out = (double*)(b + 256);
  RedBuf rb{(double*)(b + 512), ticket};
  P->launches = 0;
  TRY(red_init(rb, (size_t)parts * OpResidual<double>::NRED, s));
  TRY(residual_into(P, E, J, 0, d_out, rb, s));
  CK(cudaMemcpyAsync(P->h_state, d_out, 4 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const double* h = (const double*)P->h_state;
  for (int i = 0; i < 4; ++i) out[i] = std::sqrt(h[i]);
  return 0;
}
