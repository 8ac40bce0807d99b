// The persistent solver (cm_solo.cuh) for domains whose rows have
// register-resident transforms.
#include "cm_solo.cuh"

namespace {

// ---------------------------------------------------------------------------
// the solver
// ---------------------------------------------------------------------------
template <typename R, int L>
__global__ void __launch_bounds__(T, 1)
k_ccg_solo(const __grid_constant__ CcgArgs<R> a, const __grid_constant__ SoloX X, int elems, int iters,
           int resident, GridBarrier* bar, double* partials) {
  typedef typename CT<R>::C C;
  typedef SoloRow<L> Sh;
  typedef typename Sh::P P;
  constexpr int N = Sh::N, NP = Sh::NP, E = Sh::E, LR = Sh::LR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SoloShared sh;
  __shared__ GenFft fx;
  C* twy = reinterpret_cast<C*>(smem_raw);
  C* twx = twy + N;
  C* bufA = twx + a.op.nx;
  C* bufB = bufA + smem_padded(elems);
  stage_twiddles<L, LR, T, false>(twy, a.op.twy);
  solo_stage_x_any<R>(X, fx, twx, a.op.twx);
  constexpr int NW = (int)(sizeof(CcgState) / sizeof(int4));
  for (int i = threadIdx.x; i < NW; i += T)
    reinterpret_cast<int4*>(&sh.st)[i] = __ldcg(reinterpret_cast<const int4*>(a.st) + i);
  __syncthreads();
  SoloBarrier b;
  int pbuf = 0;
  const int s = threadIdx.x >> P::LTPS, tt = threadIdx.x & (P::TPS - 1);
  const int tx = a.tx, ty = a.ty;
  const double funif = -sh.st.p.F / sh.st.p.n_surface;
  const int tiles_t = (tx + 2 * NP - 1) / (2 * NP), tiles_u = (a.u_rows + 2 * NP - 1) / (2 * NP);
  SoloFields<R> fld;
  fld.open(a, 2 * NP, resident, reinterpret_cast<R*>(bufB + smem_padded(elems) + 1));
  R* const u = fld.u;
  R* const t = fld.t;
  const R* const h = fld.h;
  R* const f0 = fld.f0;
  R* const f1 = fld.f1;
  const size_t rb_none = fld.rb_none, ru_none = fld.ru_none;
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
      solo_col_any<R>(X, fx, a.op, rows_out, twx, bufA, bufB);
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
        solo_converge(sh, off64);
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
  fld.close(a, resident);
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < NW; i += T)
      reinterpret_cast<int4*>(a.st)[i] = reinterpret_cast<const int4*>(&sh.st)[i];
}

template <typename R, int L>
SoloPlan solo_plan(const CcgArgs<R>& a, const SoloX& X) {
  SoloPlan sp;
  const int nsm = solo_sms(), np = SoloRow<L>::NP;
  const int rows = (a.u_rows + 2 * np - 1) / (2 * np);
  const int width = solo_col_width(X), cols = (a.op.ny / 2 + width) / width;
  sp.elems = std::max(T * SoloRow<L>::E, solo_col_elems(X));
  for (int resident = 1; resident >= 0 && nsm; --resident) {
    sp.resident = resident;
    sp.smem = solo_smem(a.op.nx, a.op.ny, sp.elems, sizeof(typename CT<R>::C), resident ? 2 * np : 0, a.ty);
    if (sp.smem > CM_SMEM_DYN_MAX) continue;
    const int per_sm = solo_per_sm(k_ccg_solo<R, L>, sp.smem);
    if (per_sm < 1) {
      cudaGetLastError();
      continue;
    }
    const int grid = std::min({std::max(rows, cols), per_sm * nsm, CM_SOLO_MAX_BLOCKS});
    if (resident && grid < rows) continue;
    sp.grid = grid;
    return sp;
  }
  return sp;
}

}  // namespace

template <typename R>
SoloPlan ccg_solo_plan(const CcgArgs<R>& a, int lx, int ly, const GenFft& gx, const GenFft& gy) {
  SoloX X = solo_x<R>(lx, gx);
  switch (ly) {
#define CM_CASE(L) case L: return solo_plan<R, L>(a, X);
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return ccg_solo_gen_plan<R>(a, X, gy);
  }
}

template <typename R>
int ccg_solo_launch(const CcgArgs<R>& a, int lx, int ly, const GenFft& gx, const GenFft& gy,
                    const SoloPlan& sp, int iters, GridBarrier* bar, double* partials,
                    cudaStream_t s) {
  // arrivals count from zero in every launch
  if (cudaMemsetAsync(bar, 0, sizeof(GridBarrier), s) != cudaSuccess) return 1;
  const SoloX X = solo_x<R>(lx, gx);
  switch (ly) {
#define CM_CASE(L) \
  case L: return solo_cooperative(k_ccg_solo<R, L>, sp, s, a, X, sp.elems, iters, sp.resident, bar, partials);
    CM_SOLO_LEN_CASES(CM_CASE)
#undef CM_CASE
    default: return ccg_solo_gen_launch<R>(a, X, gy, sp, iters, bar, partials, s);
  }
}

#define CM_INST(R)                                                                               \
  template SoloPlan ccg_solo_plan<R>(const CcgArgs<R>&, int, int, const GenFft&, const GenFft&); \
  template int ccg_solo_launch<R>(const CcgArgs<R>&, int, int, const GenFft&, const GenFft&,     \
                                  const SoloPlan&, int, GridBarrier*, double*, cudaStream_t);
CM_INST(float)
CM_INST(double)
