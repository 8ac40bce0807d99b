// Persistent solver of one small contact problem: many CCG iterations in one
// cooperative launch.
//
// On small grids an iteration of launched passes (cm_ccg_p2.cuh) is a chain
// of latencies: every pass starts a kernel, stages its twiddles, reads the
// solve's state, and ends with a ticket that one last block turns into the
// next scalar (periodic 256^2 FP64: seven passes of 5-10 us, of which the
// transforms take 1.3 us each).  Here the blocks stay, the twiddles stay in shared
// memory, and the passes are separated by a grid barrier (1.2-1.5 us).
//
//   rows forward of t | columns | rows inverse, sum r t | force update |
//   rows forward of f | columns | rows inverse, u, next iteration's start
//
// Solves without a hardness only: the plastic mask of the others is the sign
// of gaps that converge to zero, so it changes with the order of a sum.
//
// * A block keeps the same row pairs in every row pass, and a thread the same
//   elements, so the fields f, t, u, h are read and written by one thread
//   only.  Where every block has at most one tile, its rows of them stay in
//   shared memory for the whole launch (a barrier's acquire empties the SM's
//   L1, so from global memory every element-wise part would wait on L2 again:
//   3400-4400 cycles for 16 elements a thread instead of about 1200).  The
//   spectrum goes through L2.
// * A reduction's partials are published by the barrier that follows it; every
//   block reads all of them in block order, and applies the same scalar step
//   (fin_*) to its own copy of the state, so all blocks branch alike and each
//   meets exactly the barriers the others meet.
// * The sum of squared gaps of the next iteration, G, needs that iteration's
//   offset (the mean gap), known only after a reduction.  It is formed from
//   sums of the gaps measured from the present offset, off:
//   G = S2 - 2 d S1 + A d^2, d = new offset - off, which cancels only as far
//   as the offset moves against the residual within one iteration.
//
// What bounds it: the chain of barriers (2400-2900 cycles each on 33-148 blocks,
// the same for flags per block and for arrivals per warp) and of a few warps'
// instruction latencies.  So four elements per thread (eight took 34 us an
// iteration of periodic 256^2 FP64, four 30), one loop body for both operators
// (with every pass written out and unrolled the iteration's code left the
// instruction cache: 48 us), poll and abort in one load, and the divisions of
// the convergence step side by side.  Per iteration, FP64: periodic 64^2 30 us,
// 256^2 31, 512^2 34, 768^2 61, free 128^2 33, 512^2 61 (launched passes 65-80);
// mixed alike.  Where every SM has many tiles, or a long side takes the
// transforms in shared memory, the launched passes' larger butterflies win:
// solo_pays (cm_plan.cu) has the rule and both sides' times.
//
// Waits are bounded (CM_BARRIER_TIMEOUT_CYCLES): a block that gives up raises
// the abort word, every other wait sees it, and the solve ends with
// CMS_TIMEOUT.
#pragma once
#include <algorithm>
#include <cstddef>
#include <mutex>

#include "cm_ccg_p2.cuh"
#include "cm_gen.cuh"
#include "cm_launch.h"
#include "cm_op_p2.cuh"

// The transform along x of a solve: the register-resident one of length code
// lx, or (lx < 0) fx on 2^lw columns at a time.
struct SoloX {
  int lx, lw;
  GenFft fx;
};

namespace {

constexpr int T = CM_SOLO_THREADS;

// row passes: the thread layout of length code L.  Four elements (of each part)
// per thread: with a row pair or two per SM the passes are bound by the
// instruction latency of its few warps, so more threads with less work each win
template <int L>
struct SoloRow {
  static constexpr int LR = 2;
  typedef FftLen<L, LR> P;
  static constexpr int N = P::N, E = P::E, NP = T / P::TPS;
  static_assert(P::TPS <= T && T % P::TPS == 0, "a row pair fits the block");
};

// column pass: groups of two columns
template <int L>
struct SoloCol {
  static constexpr int LR = L == 10 ? 3 : 2, LW = 1, W = 2;
  typedef FftLen<L, LR> P;
  static constexpr int N = P::N, E = P::E, GROUP = W * P::TPS, NG = T / GROUP;
  static_assert(GROUP <= T && T % GROUP == 0, "a column group fits the block");
};

constexpr int NWARP = T / 32;

// what the passes of one launch share
struct SoloShared {
  CcgState st;                    // this block's copy
  double part[NWARP][CM_SOLO_NV];  // a reduction's partials, by warp
  double tot[CM_SOLO_NV];    // a reduction's result
  int ok;
};

struct SoloBarrier {
  unsigned target = 0;  // arrivals that complete the next barrier
};

// The count of arrivals and the abort word of a grid barrier in one load: a
// poll is then one L2 round trip.
CM_DEVINL void ld_acquire_pair(const GridBarrier* bar, unsigned& count, unsigned& abort) {
  static_assert(offsetof(GridBarrier, gen) == 4, "count and gen share an aligned pair");
  asm volatile("ld.acquire.gpu.global.v2.u32 {%0, %1}, [%2];"
               : "=r"(count), "=r"(abort) : "l"(&bar->count) : "memory");
}

// Every block of the grid meets.  The first thread's arrival releases what
// the block wrote before; its last poll acquires what the others wrote.  The
// word after the count (GridBarrier::gen) carries the abort of this barrier.
CM_DEVINL bool solo_barrier(GridBarrier* bar, SoloBarrier& b, int* ok_sm,
                            long long limit = CM_BARRIER_TIMEOUT_CYCLES) {
  b.target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.add.release.gpu.global.u32 [%0], 1;" ::"l"(&bar->count) : "memory");
    int ok = 1;
    const long long t0 = clock64();
    while (true) {
      unsigned count, abort;
      ld_acquire_pair(bar, count, abort);
      if (abort) { ok = 0; break; }
      if ((int)(count - b.target) >= 0) break;
      if (clock64() - t0 > limit) {
        atomicExch(&bar->gen, 1u);
        ok = 0;
        break;
      }
    }
    *ok_sm = ok;
  }
  __syncthreads();
  return *ok_sm != 0;
}

// Second half of a reduction over the grid: the block's partials of nv values
// (sh.part, by warp) to the grid's, the barrier, and every block's sum of all
// of them in block order, left in sh.tot.  Bit i of maxima: value i is a
// maximum, else a sum.  The partial buffers alternate: a block writes a buffer
// again only two reductions later, behind a barrier that every block passes
// only once it has read that buffer.
__device__ __noinline__ bool solo_combine(SoloShared& sh, GridBarrier* bar, SoloBarrier& b,
                                          double* partials, int& buf, int nv, unsigned maxima) {
  double* P = partials + (size_t)buf * CM_SOLO_MAX_BLOCKS * CM_SOLO_NV;
  buf ^= 1;
  __syncthreads();
  const int i = threadIdx.x;
  if (i < nv) {
    const bool is_max = (maxima >> i) & 1;
    double x = sh.part[0][i];
#pragma unroll
    for (int w = 1; w < NWARP; ++w)
      x = is_max ? fmax(x, sh.part[w][i]) : x + sh.part[w][i];
    P[(size_t)i * CM_SOLO_MAX_BLOCKS + blockIdx.x] = x;
  }
  if (!solo_barrier(bar, b, &sh.ok)) return false;
  const int lane = threadIdx.x & 31;
  const int k = threadIdx.x >> 5;  // one value per warp
  if (k < nv) {
    const bool is_max = (maxima >> k) & 1;
    const double* Pk = P + (size_t)k * CM_SOLO_MAX_BLOCKS;
    double x = is_max ? -INFINITY : 0.0;
#pragma unroll 1
    for (int c = lane; c < (int)gridDim.x; c += 160) {
      double y[5];
#pragma unroll
      for (int m = 0; m < 5; ++m)
        y[m] = c + 32 * m < (int)gridDim.x ? __ldcg(Pk + c + 32 * m) : (is_max ? -INFINITY : 0.0);
#pragma unroll
      for (int m = 0; m < 5; ++m) x = is_max ? fmax(x, y[m]) : x + y[m];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double got = __shfl_xor_sync(0xffffffffu, x, o);
      x = is_max ? fmax(x, got) : x + got;
    }
    if (lane == 0) sh.tot[k] = x;
  }
  __syncthreads();
  return true;
}

// Reduce v over the grid at a barrier; the result is in sh.tot.  Every value
// is a sum or a maximum (a minimum goes in negated).
template <int NV>
CM_DEVINL bool solo_reduce(SoloShared& sh, GridBarrier* bar, SoloBarrier& b, double* partials,
                           int& buf, const double (&v)[NV], const bool (&maxima)[NV]) {
  static_assert(NV <= NWARP && NV <= CM_SOLO_NV, "one value per warp");
  constexpr int LNP = NV <= 1 ? 0 : NV <= 2 ? 1 : NV <= 4 ? 2 : NV <= 8 ? 3 : NV <= 16 ? 4 : 5;
  constexpr int NP = 1 << LNP, SPAN = 32 / NP;
  double w[NP];
  bool mx[NP];
  unsigned mask = 0;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    w[i] = i < NV ? v[i < NV ? i : 0] : 0.0;
    mx[i] = i < NV && maxima[i < NV ? i : 0];
    mask |= mx[i] ? 1u << i : 0u;
  }
  warp_fold<NP, 16>(w, mx);
  const int lane = threadIdx.x & 31;
  if (lane % SPAN == 0 && lane / SPAN < NV) sh.part[threadIdx.x >> 5][lane / SPAN] = w[0];
  return solo_combine(sh, bar, b, partials, buf, NV, mask);
}

// ---------------------------------------------------------------------------
// column pass, one function per column length
// ---------------------------------------------------------------------------
template <typename R, int L>
__device__ __noinline__ void solo_stage_x(typename CT<R>::C* tws, const typename CT<R>::C* tw) {
  stage_twiddles<L, SoloCol<L>::LR, T, false>(tws, tw);
}

template <typename R, int L>
__device__ __noinline__ void solo_col(const OpArgs<R>& a, int out_rows,
                                      const typename CT<R>::C* twx, typename CT<R>::C* bufA,
                                      typename CT<R>::C* bufB) {
  typedef typename CT<R>::C C;
  typedef SoloCol<L> Sh;
  typedef typename Sh::P P;
  constexpr int NX = Sh::N, W = Sh::W, E = Sh::E;
  const int ny = a.ny;
  const int c = threadIdx.x & (W - 1);
  const int tt = (threadIdx.x >> Sh::LW) & (P::TPS - 1);
  const int j = threadIdx.x >> (Sh::LW + P::LTPS);
  const int units = ny / 2 + 1;
  const int ngroups = (units + W - 1) >> Sh::LW;
  const int base = j * NX * W + c;
  const int tlw = a.lw, tW = 1 << tlw;
  for (int g0 = blockIdx.x * Sh::NG; g0 < ngroups; g0 += gridDim.x * Sh::NG) {
    const int k = (g0 + j) * W + c;
    const bool ok = k < units;
    const int km = k == 0 ? 0 : ny - k;
    C v[E];
    col_split_load<C, P::TPS, E, true>(v, a.spec, ny, k, km, tt, a.in_rows, ok);
    const R* __restrict__ tb = a.tab + ((size_t)(k >> tlw) * NX << tlw) + (k & (tW - 1));
    R tv[E];
#pragma unroll
    for (int q = 0; q < E; ++q)
      tv[q] = ok ? __ldg(tb + ((size_t)kfreq<L, Sh::LR>(tt, q) << tlw)) : (R)0;
    fft_len<C, false, L, Sh::LR, false>(v, bufA, bufB, base, W, tt, twx);
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = cscale(v[q], tv[q]);
    __syncthreads();
    fft_len<C, true, L, Sh::LR, false>(v, bufA, bufB, base, W, tt, twx);
    col_pack_store<C, P::TPS, W, E>(v, a.spec, ny, k, km, tt, out_rows, ok);
    __syncthreads();
  }
}

template <typename R>
CM_DEVINL void solo_stage_x_any(const SoloX& X, GenFft& fx, typename CT<R>::C* twx,
                                const typename CT<R>::C* tw) {
  switch (X.lx) {
#define CM_CASE(L) case L: solo_stage_x<R, L>(twx, tw); break;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: gen_stage_tables(fx, X.fx, twx, tw); break;
  }
}

template <typename R>
__device__ __noinline__ void solo_col_gen(const OpArgs<R>& a, int out_rows, const GenFft& fx, int lw,
                                          const typename CT<R>::C* twx, typename CT<R>::C* bufA,
                                          typename CT<R>::C* bufB) {
  const int units = a.ny / 2 + 1;
  for (int k0 = blockIdx.x << lw; k0 < units; k0 += gridDim.x << lw)
    gen_col_tile<R>(a, fx, k0, lw, out_rows, twx, bufA, bufB);
}

template <typename R>
CM_DEVINL void solo_col_any(const SoloX& X, const GenFft& fx, const OpArgs<R>& a, int out_rows,
                            const typename CT<R>::C* twx, typename CT<R>::C* bufA,
                            typename CT<R>::C* bufB) {
  switch (X.lx) {
#define CM_CASE(L) case L: solo_col<R, L>(a, out_rows, twx, bufA, bufB); break;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: solo_col_gen<R>(a, out_rows, fx, X.lw, twx, bufA, bufB); break;
  }
}

// (a column of the generic transform alone where two do not leave room for
// the fields)
template <typename R>
SoloX solo_x(int lx, const GenFft& gx) {
  SoloX X;
  X.lx = -1;
  switch (lx) {
#define CM_CASE(L) case L: X.lx = L; break;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
  }
  X.fx = gx;
  X.lw = gen_col_lw<R>(gx.n);
  gen_set_tile(&X.fx, 1 << X.lw);
  return X;
}

// transform elements of a column tile of X, and its tiles for ny columns
inline int solo_col_elems(const SoloX& X) {
  return X.lx < 0 ? X.fx.n << X.lw : T * (X.lx >= 32 ? 12 : X.lx == 10 ? 8 : 4);
}
inline int solo_col_width(const SoloX& X) {
  switch (X.lx) {
#define CM_CASE(L) case L: return SoloCol<L>::NG * SoloCol<L>::W;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return 1 << X.lw;
  }
}

// dynamic shared memory of a block: both twiddle tables, two buffers, and (rows
// > 0) the block's rows of u, f[2], t and h
inline size_t solo_smem(int nx, int ny, int elems, size_t csize, int rows, int ty) {
  return (size_t)(nx + ny + 2 * (elems + (elems >> 3) + 1) + 1) * csize +
         (size_t)rows * (ny + 4 * ty) * (csize / 2);
}

// SMs of the current device, or 0 when it takes no cooperative launch
inline int solo_sms() {
  int dev = 0, nsm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return 0;
  return nsm;
}

template <typename K, typename... Args>
int solo_cooperative(K kernel, const SoloPlan& sp, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sp.grid);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = sp.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? 0 : 1;
}

// resident blocks per SM of a persistent kernel with smem bytes, or -1
template <typename K>
int solo_per_sm(K kernel, size_t smem) {
  static std::mutex mu;
  std::lock_guard<std::mutex> g(mu);
  if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           CM_SMEM_DYN_MAX) != cudaSuccess)
    return -1;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, T, smem) != cudaSuccess) return -1;
  return n;
}

// Fields of the block's rows [x0, x0 + rows) where the passes find them: in
// shared memory (copied in) when resident, else in place.  Pointers are such
// that the solve's own indices apply in both cases.
template <typename R>
struct SoloFields {
  R *u, *t, *f0, *f1;
  const R* h;
  int x0, rows_t, rows_u;
  // a row that is there, for lanes whose own is not (their value is dropped)
  size_t rb_none, ru_none;
  CM_DEVINL void open(const CcgArgs<R>& a, int rows, bool resident, R* sm) {
    const int N = a.ny, ty = a.ty;
    x0 = rows * blockIdx.x;
    rows_t = max(0, min(rows, a.tx - x0));
    rows_u = max(0, min(rows, a.u_rows - x0));
    u = a.u;
    t = a.t;
    h = a.h;
    f0 = a.f[0];
    f1 = a.f[1];
    rb_none = resident ? (size_t)x0 * ty : 0;
    ru_none = resident ? (size_t)x0 * N : 0;
    if (!resident) return;
    R* const su = sm;
    R* const sf = su + (size_t)rows * N;
    const int nf = rows_t * ty, st4 = rows * ty;
    for (int i = threadIdx.x; i < rows_u * N; i += T) su[i] = __ldcg(a.u + (size_t)x0 * N + i);
    for (int i = threadIdx.x; i < nf; i += T) {
      const size_t g = (size_t)x0 * ty + i;
      sf[i] = __ldcg(a.f[0] + g);
      sf[st4 + i] = __ldcg(a.f[1] + g);
      sf[2 * st4 + i] = __ldcg(a.t + g);
      sf[3 * st4 + i] = __ldcg(a.h + g);
    }
    __syncthreads();
    const ptrdiff_t ot = (ptrdiff_t)x0 * ty;
    u = su - (ptrdiff_t)x0 * N;
    f0 = sf - ot;
    f1 = sf + st4 - ot;
    t = sf + 2 * st4 - ot;
    h = sf + 3 * st4 - ot;
  }
  CM_DEVINL void close(const CcgArgs<R>& a, bool resident) const {
    if (!resident) return;
    const int N = a.ny, ty = a.ty;
    for (int i = threadIdx.x; i < rows_u * N; i += T) a.u[(size_t)x0 * N + i] = u[(size_t)x0 * N + i];
    for (int i = threadIdx.x; i < rows_t * ty; i += T) {
      const size_t g = (size_t)x0 * ty + i;
      a.f[0][g] = f0[g];
      a.f[1][g] = f1[g];
      a.t[g] = t[g];
    }
  }
};

// The scalar step at the end of an iteration, by warp 0 (sh.tot: max |du|,
// maximum penetration, max |f|, contact points, sum of their gaps, S1, S2, sum
// f): convergence, and the next iteration's offset, G and conjugation factor.
CM_DEVINL void solo_converge(SoloShared& sh, double off64) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  CcgState& S = sh.st;
  const double *r = sh.tot, n_new = r[3];
  // the step's divisions side by side, one per lane
  const double tf = -r[7], mh = S.p.max_surface + S.offset, A = (double)S.A_cg;
  const double num = lane == 0 ? tf - (S.p.load_control ? S.p.F : S.last_tf)
                     : lane == 1 ? mh - S.last_mh : lane == 2 ? S.G : r[4];
  const double den = lane == 0 ? tf : lane == 1 ? mh : lane == 2 ? A : n_new;
  const double quot = num / den;
  ConvergeQuotients cq;
  cq.rel_tf = __shfl_sync(0xffffffffu, quot, 0);
  cq.rel_mh = __shfl_sync(0xffffffffu, quot, 1);
  cq.g_mean = __shfl_sync(0xffffffffu, quot, 2);
  const double mean_gap = __shfl_sync(0xffffffffu, quot, 3);
  if (lane == 0) {
    double ff[2] = {r[7], r[2]};
    fin_force(S, ff);
    ccg_converge_q(S, r[0], r[1], cq);
    if (!S.done) {
      // the next iteration's start: an elastic solve always takes a CG step
      S.A_contact = S.A_cg = (long long)n_new;
      S.sum_cg = r[4];
      if (S.p.load_control) S.offset = n_new > 0 ? mean_gap : 0.0;
      const double d = S.offset - off64;
      double G = r[6] - 2.0 * d * r[5] + n_new * d * d;
      if (G < 0) G = 0;  // rounding (a NaN stays NaN)
      double gv[1] = {G};
      fin_gsum(S, gv);
    }
  }
}

}  // namespace

// the kernel for any row length (cm_solo_gen.cu)
template <typename R>
SoloPlan ccg_solo_gen_plan(const CcgArgs<R>& a, const SoloX& X, const GenFft& gy);
template <typename R>
int ccg_solo_gen_launch(const CcgArgs<R>& a, const SoloX& X, GenFft gy, const SoloPlan& sp, int iters,
                        GridBarrier* bar, double* partials, cudaStream_t s);
