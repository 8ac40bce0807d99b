// The persistent solver (cm_solo.cuh) for domains whose rows have any other
// length: the same passes on transforms in shared memory (cm_gen.cuh).  Element
// e of a tile of np row pairs is column e % ny of pair e / ny, in the same
// thread in every pass.
#include "cm_solo.cuh"

namespace {

template <typename R>
__global__ void __launch_bounds__(T, 1)
k_ccg_solo_gen(const __grid_constant__ CcgArgs<R> a, const __grid_constant__ SoloX X,
               const __grid_constant__ GenFft FY, int np, FastDiv dny, int elems, int iters,
               int resident, GridBarrier* bar, double* partials) {
  typedef typename CT<R>::C C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SoloShared sh;
  __shared__ GenFft fx, fy;
  const int N = a.op.ny;
  C* twy = reinterpret_cast<C*>(smem_raw);
  C* twx = twy + N;
  C* bufA = twx + a.op.nx;
  C* bufB = bufA + smem_padded(elems);
  gen_stage_tables(fy, FY, twy, a.op.twy);
  solo_stage_x_any<R>(X, fx, twx, a.op.twx);
  constexpr int NW = (int)(sizeof(CcgState) / sizeof(int4));
  for (int i = threadIdx.x; i < NW; i += T)
    reinterpret_cast<int4*>(&sh.st)[i] = __ldcg(reinterpret_cast<const int4*>(a.st) + i);
  __syncthreads();
  SoloBarrier b;
  int pbuf = 0;
  const int tx = a.tx, ty = a.ty;
  const double funif = -sh.st.p.F / sh.st.p.n_surface;
  const int pairs_t = (tx + 1) >> 1, pairs_u = (a.u_rows + 1) >> 1;
  SoloFields<R> fld;
  fld.open(a, 2 * np, resident, reinterpret_cast<R*>(bufB + smem_padded(elems) + 1));
  R* const u = fld.u;
  R* const t = fld.t;
  const R* const h = fld.h;
  const size_t rb_none = fld.rb_none, ru_none = fld.ru_none;
  bool alive = true;
  for (int iter = 0; iter < iters && !sh.st.done; ++iter) {
    const int par = sh.st.parity & 1;
    const R off = (R)sh.st.offset;
    const R* const fa_buf = par ? fld.f1 : fld.f0;
    R* const fn_buf = par ? fld.f0 : fld.f1;
    double sgt = 0.0, srt = 0.0, s_f = 0.0;
    R amax = 0;
#pragma unroll 1
    for (int step = 0; step < 2; ++step) {
      const R beta = (R)sh.st.beta;
      const int uniform = sh.st.uniform, apply_nc = sh.st.apply_nc;
      const double scale = sh.st.scale, tau64 = sh.st.tau;
      const R* const f_in = step == 0 ? fa_buf : fn_buf;
#pragma unroll 1
      for (int p0 = blockIdx.x * np; p0 < pairs_t; p0 += gridDim.x * np) {
        const int cnt = min(np, pairs_t - p0);
        struct In { R f[2], u[2], h[2], t[2]; };
        batched_loop<2>(cnt * N, [&](int e) {
          const int p = fdiv(dny, e), y = e - p * N, yy = y < ty ? y : 0;
          In v;
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int x = 2 * (p0 + p) + w;
            const size_t rb = (x < tx ? (size_t)x * ty : rb_none) + yy;
            v.f[w] = f_in[rb];
            v.u[w] = u[(x < tx ? (size_t)x * N : ru_none) + yy];
            v.h[w] = h[rb];
            v.t[w] = t[rb];
          }
          return v;
        }, [&](int e, const In& v) {
          const int p = fdiv(dny, e), y = e - p * N;
          R z[2];
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int x = 2 * (p0 + p) + w;
            z[w] = 0;
            if (x >= tx || y >= ty) continue;
            const size_t ic = (size_t)x * ty + y;
            const R g = (v.u[w] - v.h[w]) - off;
            if (step == 0) {
              // search direction (:276-279)
              if (v.f[w] < 0) {
                z[w] = (R)(g + beta * v.t[w]);
                sgt += (double)g * (double)z[w];
              }
              t[ic] = z[w];
            } else {
              // final force of the iteration (:362-389)
              double f = uniform ? funif : scale * (double)v.f[w];
              if (apply_nc && v.f[w] == (R)0 && g < 0) f += tau64 * (double)g;
              z[w] = (R)f;
              fn_buf[ic] = z[w];
              s_f += (double)z[w];
              amax = fmax(amax, fabs(z[w]));
            }
          }
          bufA[e] = cmake<C>(z[0], z[1]);
        });
        __syncthreads();
        const C* res = gen_fft<C, false, false>(bufA, bufB, fy, cnt, 0, twy);
        C* dst = a.op.spec + (size_t)p0 * N;
        for (int e = threadIdx.x; e < cnt * N; e += T) dst[e] = res[e];
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
      const int pairs = step == 0 ? pairs_t : pairs_u;
#pragma unroll 1
      for (int p0 = blockIdx.x * np; p0 < pairs; p0 += gridDim.x * np) {
        const int cnt = min(np, pairs - p0);
        const C* src = a.op.spec + (size_t)p0 * N;
        batched_loop<4>(cnt * N, [&](int e) { return __ldcg(src + e); }, [&](int e, C v) { bufA[e] = v; });
        __syncthreads();
        const C* res = gen_fft<C, true, false>(bufA, bufB, fy, cnt, 0, twy);
        if (step == 0) {
          // sum r t (:287-294)
          struct T2 { R a, b; };
          batched_loop<4>(cnt * N, [&](int e) {
            const int p = fdiv(dny, e), y = e - p * N, yy = y < ty ? y : 0, x = 2 * (p0 + p);
            return T2{t[(size_t)x * ty + yy], t[(x + 1 < tx ? (size_t)(x + 1) * ty : rb_none) + yy]};
          }, [&](int e, T2 v) {
            const int p = fdiv(dny, e), y = e - p * N, x = 2 * (p0 + p);
            if (y >= ty) return;
            const C z = res[e];
            srt += (double)z.x * (double)v.a;
            if (x + 1 < tx) srt += (double)z.y * (double)v.b;
          });
        } else {
          struct UF { R uo[2], h[2], fn[2], fa[2]; };
          batched_loop<2>(cnt * N, [&](int e) {
            const int p = fdiv(dny, e), y = e - p * N, yy = y < ty ? y : 0;
            UF v;
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int x = 2 * (p0 + p) + w;
              const size_t rb = (x < tx ? (size_t)x * ty : rb_none) + yy;
              v.uo[w] = u[x < a.u_rows ? (size_t)x * N + y : ru_none];
              v.h[w] = h[rb];
              v.fn[w] = fn_buf[rb];
              v.fa[w] = fa_buf[rb];
            }
            return v;
          }, [&](int e, const UF& v) {
            const int p = fdiv(dny, e), y = e - p * N;
            const C z = res[e];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int x = 2 * (p0 + p) + w;
              if (x >= a.u_rows) continue;
              const R val = w ? z.y : z.x;
              du = fmax(du, fabs(val - v.uo[w]));
              u[(size_t)x * N + y] = val;
              if (x < tx && y < ty) {
                const R pen = (v.h[w] + off) - val;
                pmax = fmax(pmax, v.fa[w] < 0 ? pen : (R)0);
                const bool c = v.fn[w] < 0;
                const R g = val - v.h[w];
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
          });
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
        for (int p0 = blockIdx.x * np; p0 < pairs_t; p0 += gridDim.x * np) {
          const int cnt = min(np, pairs_t - p0);
          struct In { R f[2], u[2], h[2], t[2]; };
          batched_loop<2>(cnt * N, [&](int e) {
            const int p = fdiv(dny, e), y = e - p * N, yy = y < ty ? y : 0;
            In v;
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int x = 2 * (p0 + p) + w;
              const size_t rb = (x < tx ? (size_t)x * ty : rb_none) + yy;
              v.f[w] = fa_buf[rb];
              v.u[w] = u[(x < tx ? (size_t)x * N : ru_none) + yy];
              v.h[w] = h[rb];
              v.t[w] = t[rb];
            }
            return v;
          }, [&](int e, const In& v) {
            const int p = fdiv(dny, e), y = e - p * N;
            if (y >= ty) return;
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int x = 2 * (p0 + p) + w;
              if (x >= tx) continue;
              const R g = (v.u[w] - v.h[w]) - off;
              const R fn = v.f[w] < 0 ? (R)(v.f[w] + tau * v.t[w]) : v.f[w];
              const bool tensile = fn >= 0;
              if (tensile) max_t = fmax(max_t, fn);
              n_nc += tensile && g < 0;
              const R fp = tensile ? (R)0 : fn;
              s_fp += (double)fp;
              fn_buf[(size_t)x * ty + y] = fp;
            }
          });
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

// Row pairs of a tile: one tile per SM where the domain allows it, but no
// fewer elements than the block has threads.
int gen_pairs(int ny, int pairs, int nsm) {
  return std::max({1, (pairs + nsm - 1) / nsm, std::min(T / ny, pairs)});
}

}  // namespace

template <typename R>
SoloPlan ccg_solo_gen_plan(const CcgArgs<R>& a, const SoloX& X, const GenFft& gy) {
  SoloPlan sp;
  const int nsm = solo_sms(), pairs = (a.op.nx + 1) / 2;
  const int width = solo_col_width(X), cols = (a.op.ny / 2 + width) / width;
  for (int resident = 1; resident >= 0 && nsm; --resident) {
    // without resident fields a block may walk several tiles of one pair
    sp.np = resident ? gen_pairs(gy.n, pairs, nsm) : std::max(1, std::min(T / gy.n, pairs));
    sp.elems = std::max(sp.np * gy.n, solo_col_elems(X));
    sp.resident = resident;
    sp.smem = solo_smem(a.op.nx, a.op.ny, sp.elems, sizeof(typename CT<R>::C), resident ? 2 * sp.np : 0, a.ty);
    if (sp.smem > CM_SMEM_DYN_MAX) continue;
    const int per_sm = solo_per_sm(k_ccg_solo_gen<R>, sp.smem);
    if (per_sm < 1) {
      cudaGetLastError();
      continue;
    }
    const int rows = (pairs + sp.np - 1) / sp.np;
    const int grid = std::min({std::max(rows, cols), per_sm * nsm, CM_SOLO_MAX_BLOCKS});
    if (resident && grid < rows) continue;
    sp.grid = grid;
    return sp;
  }
  return sp;
}

template <typename R>
int ccg_solo_gen_launch(const CcgArgs<R>& a, const SoloX& X, GenFft gy, const SoloPlan& sp, int iters,
                        GridBarrier* bar, double* partials, cudaStream_t s) {
  gen_set_tile(&gy, sp.np);
  return solo_cooperative(k_ccg_solo_gen<R>, sp, s, a, X, gy, sp.np, make_fastdiv(gy.n), sp.elems, iters,
                          sp.resident, bar, partials);
}

#define CM_INST(R)                                                                          \
  template SoloPlan ccg_solo_gen_plan<R>(const CcgArgs<R>&, const SoloX&, const GenFft&);   \
  template int ccg_solo_gen_launch<R>(const CcgArgs<R>&, const SoloX&, GenFft, const SoloPlan&, int, \
                                      GridBarrier*, double*, cudaStream_t);
CM_INST(float)
CM_INST(double)
