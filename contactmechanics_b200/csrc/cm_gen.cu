// Operator passes for sides of any length (cm_gen.cuh): the launches and the
// radix plans.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "cm_gen.cuh"
#include "cm_launch.h"

namespace {

template <typename R>
__global__ void __launch_bounds__(512)
k_gen_row_fwd(const __grid_constant__ OpArgs<R> a, const __grid_constant__ GenFft F, int np, FastDiv dn) {
  typedef typename CT<R>::C C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ GenFft f;
  const int n = F.n;
  C* tw = reinterpret_cast<C*>(smem_raw);
  C* bufA = tw + n;
  C* bufB = bufA + np * n;
  pdl_trigger();
  gen_stage_tables(f, F, tw, a.twy);
  pdl_wait();
  const int npairs = (a.in_rows + 1) >> 1;
  for (int p0 = blockIdx.x * np; p0 < npairs; p0 += gridDim.x * np) {
    const int cnt = min(np, npairs - p0);
    batched_loop<4>(cnt * n, [&](int e) {
      const int s = fdiv(dn, e), y = e - s * n, x = 2 * (p0 + s);
      C v = czero<C>();
      if (y < a.in_cols) {
        v.x = __ldg(a.in + (size_t)x * a.in_ld + y);
        if (x + 1 < a.in_rows) v.y = __ldg(a.in + (size_t)(x + 1) * a.in_ld + y);
      }
      return v;
    }, [&](int e, C v) { bufA[e] = v; });
    __syncthreads();
    const C* res = gen_fft<C, false, false>(bufA, bufB, f, cnt, 0, tw);
    C* dst = a.spec + (size_t)p0 * n;
    for (int e = threadIdx.x; e < cnt * n; e += blockDim.x) dst[e] = res[e];
    __syncthreads();
  }
}

template <typename R>
__global__ void __launch_bounds__(512)
k_gen_col(const __grid_constant__ OpArgs<R> a, const __grid_constant__ GenFft F, int lw) {
  typedef typename CT<R>::C C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ GenFft f;
  C* tw = reinterpret_cast<C*>(smem_raw);
  C* bufA = tw + F.n;
  C* bufB = bufA + (F.n << lw);
  pdl_trigger();
  gen_stage_tables(f, F, tw, a.twx);
  pdl_wait();
  __syncthreads();
  const int units = a.ny / 2 + 1;
  for (int k0 = blockIdx.x << lw; k0 < units; k0 += gridDim.x << lw)
    gen_col_tile<R>(a, f, k0, lw, a.out_rows, tw, bufA, bufB);
}

template <typename R>
__global__ void __launch_bounds__(512)
k_gen_row_inv(const __grid_constant__ OpArgs<R> a, const __grid_constant__ GenFft F, int np, FastDiv dn) {
  typedef typename CT<R>::C C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ GenFft f;
  const int n = F.n;
  C* tw = reinterpret_cast<C*>(smem_raw);
  C* bufA = tw + n;
  C* bufB = bufA + np * n;
  pdl_trigger();
  gen_stage_tables(f, F, tw, a.twy);
  pdl_wait();
  const int npairs = (a.out_rows + 1) >> 1;
  for (int p0 = blockIdx.x * np; p0 < npairs; p0 += gridDim.x * np) {
    const int cnt = min(np, npairs - p0);
    const C* src = a.spec + (size_t)p0 * n;
    batched_loop<4>(cnt * n, [&](int e) { return src[e]; }, [&](int e, C v) { bufA[e] = v; });
    __syncthreads();
    const C* res = gen_fft<C, true, false>(bufA, bufB, f, cnt, 0, tw);
    for (int e = threadIdx.x; e < cnt * n; e += blockDim.x) {
      const int s = fdiv(dn, e), y = e - s * n, x = 2 * (p0 + s);
      if (y >= a.out_cols) continue;
      const C z = res[e];
      a.out[(size_t)x * a.out_ld + y] = z.x;
      if (x + 1 < a.out_rows) a.out[(size_t)(x + 1) * a.out_ld + y] = z.y;
    }
    __syncthreads();
  }
}

// Radices of n with the least cost: a constant per stage (its trip through
// shared memory and the barrier) plus a little per input of the butterfly;
// other primes by their direct sums.
struct RadixPlan {
  double cost = 0;
  std::vector<int> rad;
};

const RadixPlan& plan_radices(int n, std::map<int, RadixPlan>& memo) {
  auto it = memo.find(n);
  if (it != memo.end()) return it->second;
  RadixPlan best;
  if (n > 1) {
    best.cost = 1e30;
    auto consider = [&](int r, double c) {
      const RadixPlan& rest = plan_radices(n / r, memo);
      if (rest.cost + c < best.cost) {
        best.cost = rest.cost + c;
        best.rad = rest.rad;
        best.rad.push_back(r);
      }
    };
#define CM_CASE(RR) if (n % RR == 0) consider(RR, 16.0 + RR);
    CM_GEN_RADICES(CM_CASE)
#undef CM_CASE
    int m = n;
    for (int p : {2, 3, 5, 7})
      while (m % p == 0) m /= p;
    for (int p = 11; m > 1; p += 2)
      if (m % p == 0) {
        consider(p, 32.0 + p);
        break;
      }
  }
  return memo[n] = best;
}

}  // namespace

// Big direct stages first (no twiddles on their inputs), then odd radices (a
// stage writes runs of as many elements as the stages before it covered, so
// the first strides should share no factor with the banks), then even ones.
void make_gen_fft(int n, GenFft* F) {
  std::map<int, RadixPlan> memo;
  std::vector<int> rad = plan_radices(n, memo).rad;
  // (only lengths beyond any pass have more)
  if ((int)rad.size() > CM_GEN_STAGES) rad.resize(CM_GEN_STAGES);
  std::sort(rad.begin(), rad.end(), [](int a, int b) {
    const bool ba = a > 16 || a == 11 || a == 13, bb = b > 16 || b == 11 || b == 13;
    if (ba != bb) return ba;
    if ((a & 1) != (b & 1)) return (a & 1) != 0;
    return a > b;
  });
  *F = GenFft();
  F->n = n;
  F->nst = (int)rad.size();
  int Ns = 1;
  for (int i = 0; i < F->nst; ++i) {
    GenStage& S = F->st[i];
    S.r = rad[i];
    S.Ns = Ns;
    S.m = n / rad[i];
    S.step = n / (Ns * rad[i]);
    S.dm = make_fastdiv(S.m);
    S.dns = make_fastdiv(Ns);
    S.db = make_fastdiv(1);  // set per launch: butterflies of a tile
    Ns *= rad[i];
  }
}

// butterflies of a tile of nseq sequences, for the direct stages' item index
void gen_set_tile(GenFft* F, int nseq) {
  for (int i = 0; i < F->nst; ++i) F->st[i].db = make_fastdiv(F->st[i].m * nseq);
}

namespace {

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

int threads_for(int elems) {
  int t = 128;
  while (t < 512 && t * 6 < elems) t *= 2;
  return t;
}

template <typename K>
bool gen_prepare(K kernel) {
  return cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              CM_SMEM_DYN_MAX) == cudaSuccess;
}

template <typename R>
bool gen_ready() {
  static std::once_flag once;
  static bool ok = false;
  std::call_once(once, [] {
    ok = gen_prepare(k_gen_row_fwd<R>) && gen_prepare(k_gen_col<R>) && gen_prepare(k_gen_row_inv<R>);
  });
  return ok;
}

}  // namespace

// Row pairs of a tile for a pass of npairs pairs of length n: about a thousand
// elements, so that small grids spread over the SMs (a pass of 500 x 300 has
// 84 tiles of 3 pairs), one pair for long rows.
static int gen_row_pairs(int n, int npairs) { return std::max(1, std::min(1024 / n, npairs)); }

// log2 of the columns of a tile: 32 bytes of consecutive spectrum, fewer when
// two buffers and the twiddles do not fit.
template <typename R>
int gen_col_lw(int n) {
  const size_t cs = 2 * sizeof(R);
  int lw = sizeof(R) == 8 ? 1 : 2;
  while (lw > 0 && (size_t)n * (1 + (2u << lw)) * cs > CM_SMEM_DYN_MAX / 2) --lw;
  return lw;
}

template <typename R>
bool gen_fits(int n) {
  return (size_t)3 * n * 2 * sizeof(R) <= CM_SMEM_DYN_MAX;
}

template <typename R>
int gen_row_fwd(const OpArgs<R>& a, GenFft F, cudaStream_t s) {
  if (!gen_ready<R>()) return 1;
  const int npairs = (a.in_rows + 1) / 2, np = gen_row_pairs(F.n, npairs);
  gen_set_tile(&F, np);
  const size_t smem = (size_t)(1 + 2 * np) * F.n * 2 * sizeof(R);
  const int grid = std::min((npairs + np - 1) / np, 8 * sm_count());
  k_gen_row_fwd<R><<<grid, threads_for(np * F.n), smem, s>>>(a, F, np, make_fastdiv(F.n));
  return 0;
}

template <typename R>
int gen_col(const OpArgs<R>& a, GenFft F, cudaStream_t s) {
  if (!gen_ready<R>()) return 1;
  const int lw = gen_col_lw<R>(F.n), tiles = (a.ny / 2 + 1 + (1 << lw) - 1) >> lw;
  gen_set_tile(&F, 1 << lw);
  const size_t smem = (size_t)F.n * (1 + (2u << lw)) * 2 * sizeof(R);
  const int grid = std::min(tiles, 8 * sm_count());
  launch_pdl(k_gen_col<R>, grid, threads_for(F.n << lw), smem, s, a, F, lw);
  return 0;
}

template <typename R>
int gen_row_inv(const OpArgs<R>& a, GenFft F, cudaStream_t s) {
  if (!gen_ready<R>()) return 1;
  const int npairs = (a.out_rows + 1) / 2, np = gen_row_pairs(F.n, npairs);
  gen_set_tile(&F, np);
  const size_t smem = (size_t)(1 + 2 * np) * F.n * 2 * sizeof(R);
  const int grid = std::min((npairs + np - 1) / np, 8 * sm_count());
  launch_pdl(k_gen_row_inv<R>, grid, threads_for(np * F.n), smem, s, a, F, np, make_fastdiv(F.n));
  return 0;
}

template bool gen_fits<float>(int);
template bool gen_fits<double>(int);
template int gen_col_lw<float>(int);
template int gen_col_lw<double>(int);
template int gen_row_fwd<float>(const OpArgs<float>&, GenFft, cudaStream_t);
template int gen_row_fwd<double>(const OpArgs<double>&, GenFft, cudaStream_t);
template int gen_col<float>(const OpArgs<float>&, GenFft, cudaStream_t);
template int gen_col<double>(const OpArgs<double>&, GenFft, cudaStream_t);
template int gen_row_inv<float>(const OpArgs<float>&, GenFft, cudaStream_t);
template int gen_row_inv<double>(const OpArgs<double>&, GenFft, cudaStream_t);
