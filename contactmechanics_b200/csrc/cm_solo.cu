// Persistent solver of one small contact problem: many CCG iterations in one
// cooperative launch.
//
// On small grids an iteration of launched passes (cm_ccg_p2.cuh) is a chain
// of latencies: every pass starts a kernel, stages its twiddles, reads the
// solve's state, and ends with a ticket that one last block turns into the
// next scalar (periodic 256^2 FP64: seven passes of 5-10 us, of which the
// transforms take 1.3 us each).  Here the blocks stay, the twiddles stay in shared
// memory, and the passes are separated by a grid barrier (about 1 us).
//
//   rows forward of t | columns | rows inverse, sum r t | force update |
//   rows forward of f | columns | rows inverse, u, next iteration's start
//
// Solves without a hardness only: the plastic mask of the others is the sign
// of gaps that converge to zero, so it changes with the order of a sum.
//
// * A block keeps the same row pairs in every row pass, and a thread the same
//   elements, so the fields f, t, u, h are read and written by one thread
//   only and are cached by its SM's L1; the spectrum goes through L2.
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
// Waits are bounded (CM_BARRIER_TIMEOUT_CYCLES): a block that gives up raises
// the abort word, every other wait sees it, and the solve ends with
// CMS_TIMEOUT.
#include <algorithm>
#include <cstddef>
#include <mutex>

#include "cm_ccg_p2.cuh"
#include "cm_launch.h"
#include "cm_op_p2.cuh"

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

// transform elements of a block: its widest pass
__host__ __device__ constexpr int solo_elems(int ly, int lx) {
  const int row = ly >= 32 ? 12 : 4, col = lx >= 32 ? 12 : lx == 10 ? 8 : 4;
  return T * (row > col ? row : col);
}

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
CM_DEVINL bool solo_barrier(GridBarrier* bar, SoloBarrier& b, int* ok_sm) {
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
      if (clock64() - t0 > CM_BARRIER_TIMEOUT_CYCLES) {
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
CM_DEVINL void solo_col_any(int lx, const OpArgs<R>& a, int out_rows, const typename CT<R>::C* twx,
                            typename CT<R>::C* bufA, typename CT<R>::C* bufB) {
  switch (lx) {
#define CM_CASE(L) case L: solo_col<R, L>(a, out_rows, twx, bufA, bufB); break;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
  }
}

// ---------------------------------------------------------------------------
// the solver
// ---------------------------------------------------------------------------
template <typename R, int L>
__global__ void __launch_bounds__(T, 1)
k_ccg_solo(const __grid_constant__ CcgArgs<R> a, int lx, int iters, int resident, GridBarrier* bar,
           double* partials) {
  typedef typename CT<R>::C C;
  typedef SoloRow<L> Sh;
  typedef typename Sh::P P;
  constexpr int N = Sh::N, NP = Sh::NP, E = Sh::E, LR = Sh::LR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SoloShared sh;
  C* twy = reinterpret_cast<C*>(smem_raw);
  C* twx = twy + N;
  C* bufA = twx + a.op.nx;
  C* bufB = bufA + smem_padded(solo_elems(L, lx));
  stage_twiddles<L, LR, T, false>(twy, a.op.twy);
  switch (lx) {
#define CM_CASE(X) case X: solo_stage_x<R, X>(twx, a.op.twx); break;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
  }
  constexpr int NW = (int)(sizeof(CcgState) / sizeof(int4));
  for (int i = threadIdx.x; i < NW; i += T)
    reinterpret_cast<int4*>(&sh.st)[i] = __ldcg(reinterpret_cast<const int4*>(a.st) + i);
  __syncthreads();
  SoloBarrier b;
  int pbuf = 0;
  const int s = threadIdx.x >> P::LTPS, tt = threadIdx.x & (P::TPS - 1);
  const int lane = threadIdx.x & 31;
  const int tx = a.tx, ty = a.ty;
  const double funif = -sh.st.p.F / sh.st.p.n_surface;
  const int tiles_t = (tx + 2 * NP - 1) / (2 * NP), tiles_u = (a.u_rows + 2 * NP - 1) / (2 * NP);
  R* u = a.u;
  R* t = a.t;
  const R* h = a.h;
  R* f0 = a.f[0];
  R* f1 = a.f[1];
  // Every block has at most one tile: its rows of the fields stay in shared
  // memory for the whole launch.  (A barrier's acquire empties the SM's L1, so
  // from global memory every element-wise part waits on L2 again: 3400-4400
  // cycles for 16 elements a thread instead of about 1200.)  The same generic
  // pointers serve both cases.
  const int x0 = 2 * NP * blockIdx.x;
  const int rows_t = max(0, min(2 * NP, tx - x0)), rows_u = max(0, min(2 * NP, a.u_rows - x0));
  if (resident) {
    R* sm = reinterpret_cast<R*>(bufB + smem_padded(solo_elems(L, lx)) + 1);
    R* const su = sm;
    R* const sf = su + 2 * NP * N;
    const int nf = rows_t * ty, st4 = 2 * NP * ty;
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
  // rows without topography read a row that is there (the first of the block's
  // rows in shared memory, whether they hold topography or not, or of the
  // field), columns beyond it their row's first element, and drop the value
  const size_t rb_none = resident ? (size_t)x0 * ty : 0, ru_none = resident ? (size_t)x0 * N : 0;
  bool alive = true;
  for (int iter = 0; iter < iters && !sh.st.done; ++iter) {
    const int par = sh.st.parity & 1;
    const R off = (R)sh.st.offset;
    const R* const fa_buf = par ? f1 : f0;
    R* const fn_buf = par ? f0 : f1;
    double sgt = 0.0, srt = 0.0, s_f = 0.0;
    R amax = 0;
    // step 0: r = G t and the step length; step 1: the force update and
    // u = G f.  One body for both: the transforms' code is shared (the loop's
    // code has to stay in the instruction cache: with every pass written out
    // and its loops unrolled, instruction fetches tripled the time of the
    // element-wise parts)
#pragma unroll 1
    for (int step = 0; step < 2; ++step) {
      const R beta = (R)sh.st.beta;
      const int uniform = sh.st.uniform, apply_nc = sh.st.apply_nc;
      const double scale = sh.st.scale, tau64 = sh.st.tau;
#pragma unroll 1
      for (int tile = blockIdx.x; tile < tiles_t; tile += gridDim.x) {
        const int xa = 2 * (tile * NP + s);
        C v[E];
#pragma unroll 1
        for (int w = 0; w < 2; ++w) {
          const int x = xa + w;
          const bool in_x = x < tx;
          const size_t rb = in_x ? (size_t)x * ty : rb_none, ru = in_x ? (size_t)x * N : ru_none;
          const R* const f_in = step == 0 ? fa_buf : fn_buf;
          R fv[E], uv[E], hv[E], tv[E];
#pragma unroll
          for (int q = 0; q < E; ++q) {
            const int y = tt + q * P::TPS, yy = y < ty ? y : 0;
            fv[q] = f_in[rb + yy];
            uv[q] = u[ru + yy];
            hv[q] = h[rb + yy];
            tv[q] = t[rb + yy];
          }
          if (step == 0) {
            // search direction (:276-279)
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const int y = tt + q * P::TPS;
              R tn = 0;
              if (in_x && y < ty) {
                const R g = (uv[q] - hv[q]) - off;
                if (fv[q] < 0) {
                  tn = (R)(g + beta * tv[q]);
                  sgt += (double)g * (double)tn;
                }
                t[rb + y] = tn;
              }
              v[q].x = w ? v[q].x : tn;
              v[q].y = tn;
            }
          } else {
            // final force of the iteration (:362-389)
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const int y = tt + q * P::TPS;
              R fr = 0;
              if (in_x && y < ty) {
                double f = uniform ? funif : scale * (double)fv[q];
                const R g = (uv[q] - hv[q]) - off;
                if (apply_nc && fv[q] == (R)0 && g < 0) f += tau64 * (double)g;
                fr = (R)f;
                fn_buf[rb + y] = fr;
                s_f += (double)fr;
                amax = fmax(amax, fabs(fr));
              }
              v[q].x = w ? v[q].x : fr;
              v[q].y = fr;
            }
          }
        }
        fft_len<C, false, L, LR, false>(v, bufA, bufB, s * N, 1, tt, twy);
        if (xa < tx) {
          C* srow = a.op.spec + (size_t)(xa >> 1) * N;
#pragma unroll
          for (int q = 0; q < E; ++q) srow[kfreq<L, LR>(tt, q)] = v[q];
        }
        __syncthreads();
      }
      if (!(alive = solo_barrier(bar, b, &sh.ok))) break;
      const int rows_out = step == 0 ? tx : a.u_rows;
      solo_col_any<R>(lx, a.op, rows_out, twx, bufA, bufB);
      if (!(alive = solo_barrier(bar, b, &sh.ok))) break;
      // inverse rows; step 1: convergence and the next iteration's start
      // (:239-270, 391-434)
      const double off64 = sh.st.offset;
      R du = 0, pmax = -INFINITY;
      int n_c = 0;
      double s_cg = 0, s1 = 0, s2 = 0;
      const int tiles = step == 0 ? tiles_t : tiles_u;
#pragma unroll 1
      for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int xa = 2 * (tile * NP + s);
        C v[E];
        const C* srow = a.op.spec + (size_t)(xa >> 1) * N;
#pragma unroll
        for (int q = 0; q < E; ++q)
          v[q] = xa < rows_out ? __ldcg(srow + kfreq<L, LR>(tt, q)) : czero<C>();
        fft_len<C, true, L, LR, false>(v, bufA, bufB, s * N, 1, tt, twy);
        if (step == 0) {
          // sum r t (:287-294)
#pragma unroll 1
          for (int w = 0; w < 2; ++w) {
            const int x = xa + w;
            if (x >= tx) break;
            const R* trow = t + (size_t)x * ty;
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const int y = tt + q * P::TPS;
              const R tv = trow[y < ty ? y : 0];
              if (y < ty) srt += (double)(w ? v[q].y : v[q].x) * (double)tv;
            }
          }
        } else {
#pragma unroll 1
          for (int w = 0; w < 2; ++w) {
            const int x = xa + w;
            if (x >= a.u_rows) break;
            const bool in_x = x < tx;
            const size_t rb = in_x ? (size_t)x * ty : rb_none;
            R uo[E], hv[E], fn[E], fa[E];
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const int y = tt + q * P::TPS, yy = y < ty ? y : 0;
              uo[q] = u[(size_t)x * N + y];
              hv[q] = h[rb + yy];
              fn[q] = fn_buf[rb + yy];
              fa[q] = fa_buf[rb + yy];
            }
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const int y = tt + q * P::TPS;
              const R val = w ? v[q].y : v[q].x;
              du = fmax(du, fabs(val - uo[q]));
              u[(size_t)x * N + y] = val;
              if (in_x && y < ty) {
                const R pen = (hv[q] + off) - val;
                pmax = fmax(pmax, fa[q] < 0 ? pen : (R)0);
                const bool c = fn[q] < 0;
                const R g = val - hv[q];
                n_c += c;
                // the reference sums c g^2 over the whole topography, so a NaN
                // gap outside the contact set makes G NaN as well
                const double gs = (double)g - off64;
                if (c) {
                  s_cg += (double)g;
                  s1 += gs;
                  s2 += gs * gs;
                } else if (isnan(g)) {
                  s2 += (double)g;
                }
              }
            }
          }
        }
        __syncthreads();
      }
      if (step == 0) {
        const double r2[2] = {sgt, srt};
        const bool m2[2] = {false, false};
        if (!(alive = solo_reduce<2>(sh, bar, b, partials, pbuf, r2, m2))) break;
        if (threadIdx.x == 0) {
          sh.st.sum_cgt = sh.tot[0];
          double rt[1] = {sh.tot[1]};
          fin_tau(sh.st, rt);
        }
        __syncthreads();
        // force update, projection, constraint bookkeeping (:296, 320-389)
        const R tau = (R)sh.st.tau;
        int n_nc = 0;
        R max_t = 0;
        double s_fp = 0;
#pragma unroll 1
        for (int tile = blockIdx.x; tile < tiles_t; tile += gridDim.x) {
#pragma unroll 1
          for (int w = 0; w < 2; ++w) {
            const int x = 2 * (tile * NP + s) + w;
            if (x >= tx) break;
            const size_t rb = (size_t)x * ty, ru = (size_t)x * N;
#pragma unroll 1
            for (int q0 = 0; q0 < E; q0 += 4) {
              R fv[4], uv[4], hv[4], tv[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int y = tt + (q0 + q) * P::TPS, yy = y < ty ? y : 0;
                fv[q] = fa_buf[rb + yy];
                uv[q] = u[ru + yy];
                hv[q] = h[rb + yy];
                tv[q] = t[rb + yy];
              }
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int y = tt + (q0 + q) * P::TPS;
                if (y >= ty) continue;
                const R g = (uv[q] - hv[q]) - off;
                const R fn = fv[q] < 0 ? (R)(fv[q] + tau * tv[q]) : fv[q];
                const bool tensile = fn >= 0;
                if (tensile) max_t = fmax(max_t, fn);
                n_nc += tensile && g < 0;
                const R fp = tensile ? (R)0 : fn;
                s_fp += (double)fp;
                fn_buf[rb + y] = fp;
              }
            }
          }
        }
        const double v3[3] = {s_fp, (double)n_nc, (double)max_t};
        const bool m3[3] = {false, false, true};
        if (!(alive = solo_reduce<3>(sh, bar, b, partials, pbuf, v3, m3))) break;
        if (threadIdx.x == 0) {
          double v5[5] = {0.0, 0.0, sh.tot[2], sh.tot[0], sh.tot[1]};
          fin_update(sh.st, v5);
        }
        __syncthreads();
      } else {
        const double v8[8] = {(double)du, (double)pmax, (double)amax, (double)n_c, s_cg, s1, s2, s_f};
        const bool m8[8] = {true, true, true, false, false, false, false, false};
        if (!(alive = solo_reduce<8>(sh, bar, b, partials, pbuf, v8, m8))) break;
        if (threadIdx.x < 32) {
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
        __syncthreads();
      }
    }
    if (!alive) break;
  }
  if (!alive && threadIdx.x == 0) {
    sh.st.status = CMS_TIMEOUT;
    sh.st.done = 1;
  }
  __syncthreads();
  if (resident) {
    for (int i = threadIdx.x; i < rows_u * N; i += T) a.u[(size_t)x0 * N + i] = u[(size_t)x0 * N + i];
    for (int i = threadIdx.x; i < rows_t * ty; i += T) {
      const size_t g = (size_t)x0 * ty + i;
      a.f[0][g] = f0[g];
      a.f[1][g] = f1[g];
      a.t[g] = t[g];
    }
  }
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < NW; i += T)
      reinterpret_cast<int4*>(a.st)[i] = reinterpret_cast<const int4*>(&sh.st)[i];
}

// dynamic shared memory of a block: both twiddle tables, two buffers, and (rows
// > 0) the block's rows of u, f[2], t and h
constexpr size_t solo_smem(int nx, int ny, int elems, size_t csize, int rows, int ty) {
  return (size_t)(nx + ny + 2 * (elems + (elems >> 3) + 1) + 1) * csize +
         (size_t)rows * (ny + 4 * ty) * (csize / 2);
}

std::mutex g_solo_mu;

int solo_row_pairs(int ly) {
  switch (ly) {
#define CM_CASE(L) case L: return SoloRow<L>::NP;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return 0;
  }
}
int solo_col_groups(int lx) {
  switch (lx) {
#define CM_CASE(L) case L: return SoloCol<L>::NG;
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return 0;
  }
}

template <typename R, int L>
int solo_run(const CcgArgs<R>& a, int lx, const SoloPlan& sp, int iters, GridBarrier* bar,
             double* partials, cudaStream_t s) {
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
  return cudaLaunchKernelEx(&cfg, k_ccg_solo<R, L>, a, lx, iters, sp.resident, bar,
                            partials) == cudaSuccess ? 0 : 1;
}

template <typename R, int L>
int solo_per_sm(size_t smem) {
  std::lock_guard<std::mutex> g(g_solo_mu);
  if (cudaFuncSetAttribute((const void*)k_ccg_solo<R, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           CM_SMEM_DYN_MAX) != cudaSuccess)
    return -1;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ccg_solo<R, L>, T, smem) != cudaSuccess)
    return -1;
  return n;
}

}  // namespace

// Launch shape of the persistent kernel for a solve on a domain of length
// codes lx, ly: one tile of the widest pass per block, at most one resident
// wave; grid 0 when the domain or the device does not take it.
template <typename R>
SoloPlan ccg_solo_plan(const CcgArgs<R>& a, int lx, int ly) {
  SoloPlan sp;
  const int np = solo_row_pairs(ly), ng = solo_col_groups(lx);
  int dev = 0, nsm = 0, coop = 0;
  if (!np || !ng || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return sp;
  const int rows = (a.u_rows + 2 * np - 1) / (2 * np);
  const int cols = ((a.op.ny / 2 + 1 + 1) / 2 + ng - 1) / ng;
  const size_t cs = sizeof(typename CT<R>::C);
  for (int resident = 1; resident >= 0; --resident) {
    const size_t smem = solo_smem(a.op.nx, a.op.ny, solo_elems(ly, lx), cs, resident ? 2 * np : 0, a.ty);
    if (smem > CM_SMEM_DYN_MAX) continue;
    int per_sm = 0;
    switch (ly) {
#define CM_CASE(L) case L: per_sm = solo_per_sm<R, L>(smem); break;
      CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    }
    if (per_sm < 1) {
      cudaGetLastError();
      continue;
    }
    const int grid = std::min({std::max(rows, cols), per_sm * nsm, CM_SOLO_MAX_BLOCKS});
    if (resident && grid < rows) continue;
    sp.grid = grid;
    sp.resident = resident;
    sp.smem = smem;
    return sp;
  }
  return sp;
}

template <typename R>
int ccg_solo_launch(const CcgArgs<R>& a, int lx, int ly, const SoloPlan& sp, int iters,
                    GridBarrier* bar, double* partials, cudaStream_t s) {
  // arrivals count from zero in every launch
  if (cudaMemsetAsync(bar, 0, sizeof(GridBarrier), s) != cudaSuccess) return 1;
  switch (ly) {
#define CM_CASE(L) case L: return solo_run<R, L>(a, lx, sp, iters, bar, partials, s);
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return -1;
  }
}

template SoloPlan ccg_solo_plan<float>(const CcgArgs<float>&, int, int);
template SoloPlan ccg_solo_plan<double>(const CcgArgs<double>&, int, int);
template int ccg_solo_launch<float>(const CcgArgs<float>&, int, int, const SoloPlan&, int,
                                    GridBarrier*, double*, cudaStream_t);
template int ccg_solo_launch<double>(const CcgArgs<double>&, int, int, const SoloPlan&, int,
                                     GridBarrier*, double*, cudaStream_t);
