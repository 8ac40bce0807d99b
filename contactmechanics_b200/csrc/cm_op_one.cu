// The operator of a small domain with sides 2^k of 64 to 1024 in one cooperative
// launch: the row, column and inverse row passes (cm_op_p2.cuh) separated by grid
// barriers.
//
// Three launches cost the host about 8 us of a call, more than the GPU needs on
// small grids; one launch stages both twiddle tables once and crosses two
// barriers of about 1.3 us.  Four elements per thread, as in the persistent
// solver: the passes are bound by the latency of a few warps per SM and by the
// fetch of instructions that each run once (ncu, 64^2: 8 warps wait for an
// instruction, 5 at a barrier, per issue).  Per call,
// one launch against three: FP64 64^2 10.9 / 15.0 us, 256^2 13.4 / 16.5,
// 512^2 14.4 / 18.5, FP32 512^2 12.8 / 15.4; from 1024^2 on the launched
// passes' longer butterflies win (30.8 / 24.2), as they do for sides 3 * 2^m
// (192^2 22.0 / 18.6) and, but for the host's part, for others (500 x 300
// 22.6 / 22.9).
#include "cm_solo.cuh"

// the sides it serves
#define CM_ONE_CASES(X) X(6) X(7) X(8) X(9) X(10)

namespace {

template <typename R>
CM_DEVINL void one_stage_x(int lx, typename CT<R>::C* twx, const typename CT<R>::C* tw) {
  switch (lx) {
#define CM_CASE(L) case L: solo_stage_x<R, L>(twx, tw); break;
    CM_ONE_CASES(CM_CASE)
#undef CM_CASE
  }
}

template <typename R>
CM_DEVINL void one_col(int lx, const OpArgs<R>& a, const typename CT<R>::C* twx, typename CT<R>::C* bufA,
                       typename CT<R>::C* bufB) {
  switch (lx) {
#define CM_CASE(L) case L: solo_col<R, L>(a, a.out_rows, twx, bufA, bufB); break;
    CM_ONE_CASES(CM_CASE)
#undef CM_CASE
  }
}

// The last use of the barrier in a launch: the last block leaves it zeroed for
// the next one (launches on the same plan follow each other, replays of a
// captured graph included).
CM_DEVINL void one_release(GridBarrier* bar) {
  __syncthreads();
  if (threadIdx.x == 0 && take_ticket(&bar->pad) == gridDim.x - 1) {
    bar->count = 0;
    bar->gen = 0;
    bar->pad = 0;
  }
}

// This block's wait gave up, or saw that another's had (a block was not
// scheduled for two seconds): NaN in the rows that the block would have
// written, tiles of `rows` of them, and the plan's word that the host reads
// before the next call.  Blocks that got through the last barrier write their
// own rows, whose inputs are complete; so every row is one or the other.
template <typename R>
__device__ __noinline__ void one_failed(const OpArgs<R>& a, int rows, int* gave_up) {
  for (int xt = rows * blockIdx.x; xt < a.out_rows; xt += rows * gridDim.x)
    for (int x = xt; x < min(xt + rows, a.out_rows); ++x)
      for (int y = threadIdx.x; y < a.out_cols; y += T) a.out[(size_t)x * a.out_ld + y] = (R)NAN;
  if (threadIdx.x == 0) {
    *(volatile int*)gave_up = 1;
    __threadfence_system();
  }
}

template <typename R, int L>
__global__ void __launch_bounds__(T, 1)
k_op_one(const __grid_constant__ OpArgs<R> a, int lx, int elems, GridBarrier* bar, long long limit,
         int* gave_up) {
  typedef typename CT<R>::C C;
  typedef SoloRow<L> Sh;
  typedef typename Sh::P P;
  constexpr int N = Sh::N, NP = Sh::NP, E = Sh::E, LR = Sh::LR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int ok;
  C* twy = reinterpret_cast<C*>(smem_raw);
  C* twx = twy + N;
  C* bufA = twx + a.nx;
  C* bufB = bufA + smem_padded(elems);
  stage_twiddles<L, LR, T, false>(twy, a.twy);
  one_stage_x<R>(lx, twx, a.twx);
  __syncthreads();
  SoloBarrier b;
  const int s = threadIdx.x >> P::LTPS, tt = threadIdx.x & (P::TPS - 1);
#pragma unroll 1
  for (int xt = 2 * NP * blockIdx.x; xt < a.in_rows; xt += 2 * NP * gridDim.x) {
    const int xa = xt + 2 * s;
    C v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int y = tt + q * P::TPS;
      v[q] = czero<C>();
      if (y < a.in_cols) {
        if (xa < a.in_rows) v[q].x = __ldg(a.in + (size_t)xa * a.in_ld + y);
        if (xa + 1 < a.in_rows) v[q].y = __ldg(a.in + (size_t)(xa + 1) * a.in_ld + y);
      }
    }
    fft_len<C, false, L, LR, false>(v, bufA, bufB, s * N, 1, tt, twy);
    if (xa < a.in_rows) {
      C* srow = a.spec + (size_t)(xa >> 1) * N;
#pragma unroll
      for (int q = 0; q < E; ++q) srow[kfreq<L, LR>(tt, q)] = v[q];
    }
    __syncthreads();
  }
  bool alive = solo_barrier(bar, b, &ok, limit);
  if (alive) {
    one_col<R>(lx, a, twx, bufA, bufB);
    alive = solo_barrier(bar, b, &ok, limit);
  }
  if (alive) {
#pragma unroll 1
    for (int xt = 2 * NP * blockIdx.x; xt < a.out_rows; xt += 2 * NP * gridDim.x) {
      const int xa = xt + 2 * s;
      const C* srow = a.spec + (size_t)(xa >> 1) * N;
      C v[E];
#pragma unroll
      for (int q = 0; q < E; ++q)
        v[q] = xa < a.out_rows ? __ldcg(srow + kfreq<L, LR>(tt, q)) : czero<C>();
      fft_len<C, true, L, LR, false>(v, bufA, bufB, s * N, 1, tt, twy);
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const int y = tt + q * P::TPS;
        if (y >= a.out_cols) continue;
        if (xa < a.out_rows) a.out[(size_t)xa * a.out_ld + y] = v[q].x;
        if (xa + 1 < a.out_rows) a.out[(size_t)(xa + 1) * a.out_ld + y] = v[q].y;
      }
      __syncthreads();
    }
  } else {
    one_failed(a, 2 * NP, gave_up);
  }
  one_release(bar);
}

}  // namespace

// Launch shape of the operator's kernel on a domain of length codes lx, ly;
// grid 0 when the domain or the device does not take it.
template <typename R>
SoloPlan op_one_plan(int nx, int ny, int lx, int ly) {
  SoloPlan sp;
  const int nsm = solo_sms();
  if (!nsm || lx < 6 || lx > 10) return sp;
  SoloX X;
  X.lx = lx;
  X.lw = 0;
  int per_sm = 0;
  const void* kern = nullptr;
  switch (ly) {
#define CM_CASE(L)                             \
  case L:                                      \
    sp.np = SoloRow<L>::NP;                    \
    sp.elems = T * SoloRow<L>::E;              \
    kern = (const void*)k_op_one<R, L>;        \
    break;
    CM_ONE_CASES(CM_CASE)
#undef CM_CASE
    default: return sp;
  }
  sp.elems = std::max(sp.elems, solo_col_elems(X));
  sp.smem = solo_smem(nx, ny, sp.elems, 2 * sizeof(R), 0, 0);
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM_DYN_MAX) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, T, sp.smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return sp;
  }
  const int rows = (nx / 2 + sp.np - 1) / sp.np;
  const int width = solo_col_width(X), cols = (ny / 2 + width) / width;
  sp.grid = std::min(std::max(rows, cols), per_sm * nsm);
  return sp;
}

template <typename R>
int op_one_launch(const OpArgs<R>& a, int lx, int ly, const SoloPlan& sp, GridBarrier* bar,
                  long long limit, int* gave_up, cudaStream_t s) {
  switch (ly) {
#define CM_CASE(L) case L: return solo_cooperative(k_op_one<R, L>, sp, s, a, lx, sp.elems, bar, limit, gave_up);
    CM_ONE_CASES(CM_CASE)
#undef CM_CASE
    default: return -1;
  }
}

#define CM_INST(R)                                                                    \
  template SoloPlan op_one_plan<R>(int, int, int, int);                               \
  template int op_one_launch<R>(const OpArgs<R>&, int, int, const SoloPlan&, GridBarrier*, long long, \
                                int*, cudaStream_t);
CM_INST(float)
CM_INST(double)
