// The elastic operator u = IFFT(T . FFT(f)) (FFTElasticHalfSpace.py:573-611,
// free :1141-1197) for power-of-two domains (sides 64..8192), as three
// passes over caller buffers:
//
//   k_op_row_fwd  row pairs (2p, 2p+1) with rows < in_rows: one complex
//                 transform of z = f[2p] + i f[2p+1] per pair, stored as it
//                 comes out of the registers: Z_p(k), k = 0..ny-1, at
//                 spec[p * ny + k] (the pair-major spectrum);
//   k_op_col      every column k = 0..ny/2 of the half spectrum: the column
//                 X_x(k) of row x = 2p + b is split off the pair transforms
//                 in registers (X_2p(k) = (Z_p(k) + conj Z_p(ny-k)) / 2,
//                 X_2p+1(k) = (Z_p(k) - conj Z_p(ny-k)) / 2i; rows >= in_rows
//                 are zero), transformed along x, multiplied by the real
//                 Green's table, transformed back, and packed again for the
//                 inverse row transforms: W_p(k) = Xh_2p(k) + i Xh_2p+1(k) and
//                 W_p(ny-k) = conj Xh_2p(k) + i conj Xh_2p+1(k), pairs with rows
//                 < out_rows written back in place;
//   k_op_row_inv  row pairs with rows < out_rows: one inverse complex
//                 transform of W_p per pair straight from the spectrum; the
//                 real part is row 2p, the imaginary part row 2p+1.
//
// The row passes thus read and write the spectrum in whole rows from the
// transform registers, with no shared-memory split or pack pass; the split
// and the pack are arithmetic in the column pass, whose two rows of a pair
// sit in neighbouring threads (a shuffle exchanges them).  A column group
// covers W consecutive columns (W = 32 bytes of complex values, so every
// spectrum access of a warp fills whole 32-byte sectors; fewer when the
// shared memory of a long column does not allow it).
//
// Arguments travel by value (no descriptor upload), so a call is a plain
// sequence of three launches on the caller's stream.  Blocks walk their
// tiles with a grid stride, so the twiddle tables are staged once per block;
// the transforms are the register-resident engines of cm_fft_p2.cuh (row
// passes and column pass 2^LR elements per thread).
#pragma once
#include "cm_fft_p2.cuh"
#include "cm_kernels.cuh"
#include "cm_launch.h"

// resident blocks per SM the FP64 row passes are compiled for: two blocks
// of 256 threads (at most 128 registers a thread) hide more latency than one
#ifndef CM_FP64_ROW_MINB
#define CM_FP64_ROW_MINB 2
#endif

// threads of an FP32 row-pass block (at least one transform) and the
// resident blocks per SM it is compiled for
#ifndef CM_ROW_F32_BASE
#define CM_ROW_F32_BASE 512
#endif
#ifndef CM_ROW_F32_MINB
#define CM_ROW_F32_MINB 2
#endif

// threads of a column-pass block when a column group is smaller
#ifndef CM_COL_BASE
#define CM_COL_BASE 256
#endif

// ... for a grid with too few columns to give every second SM such a block (512^2
// FP64: 33 blocks of 256 threads, 129 of 64; plastic 512^2 solve 9.3 -> 8.5 ms,
// operator FP64 384^2 21.6 -> 15.0 us).  With more columns the larger blocks
// stage fewer twiddles (512 x 2048 24.9 us, 26.9 with blocks of 64); columns of
// 3 * 2^m points keep to the small ones (768 x 1536 FP64 41.1 and 41.0 us).
#ifndef CM_COL_BASE_SHORT
#define CM_COL_BASE_SHORT 64
#endif

// log2 of the elements per thread of the column pass's transforms
#ifndef CM_COL_LR_F32
#define CM_COL_LR_F32 4
#endif
#ifndef CM_COL_LR_F64
#define CM_COL_LR_F64 4
#endif

// log2 of the columns of a column group (at most; fewer when its shared
// memory does not fit): 32 bytes of complex values
#ifndef CM_COL_LW_F32
#define CM_COL_LW_F32 2
#endif
#ifndef CM_COL_LW_F64
#define CM_COL_LW_F64 1
#endif

// Whether the column pass of type R and length code L is sized for two blocks
// per SM.  FP64 columns of 2^11: one buffer each, so that one block's loads
// run under the other's transforms (operator 2048^2 99.5 -> 90.8 us); of 2^10
// there are too few blocks to pair (22.9 -> 30.9 us), and 3 * 2^m loses more by
// the second barrier (1536^2 63.8 -> 68.9).
#ifndef CM_COL_PAIR
#define CM_COL_PAIR(R, L) (sizeof(R) == 8 && (L) == 11)
#endif

// log2 of the elements per thread of the solver's displacement pass
// (k_ccg_row_inv<MODE_F>): its epilogue reads four fields per element, so it
// keeps eight elements per thread and twice the resident warps
#ifndef CM_ROW_LR_INVF_F32
#define CM_ROW_LR_INVF_F32 3
#endif

// log2 of the elements per thread of the row passes' transforms (3: the
// radix-8 engine, 4: the radix-16 one)
#ifndef CM_ROW_LR_F32
#define CM_ROW_LR_F32 4
#endif
#ifndef CM_ROW_LR_F64
#define CM_ROW_LR_F64 3
#endif

// log2 of the elements per thread of each power-of-two part of a length
// 3 * 2^m (three parts, so a thread holds three times as many), and the
// threads of a row-pass block for those lengths.  Four elements a part in
// FP32 too: the solver passes' epilogues then keep their fields in
// registers (mixed solves 8-20 % faster than with eight, periodic 768..3072).
#ifndef CM_T3_LR_F32
#define CM_T3_LR_F32 2
#endif
#ifndef CM_T3_LR_F64
#define CM_T3_LR_F64 2
#endif
#ifndef CM_T3_ROW_BASE
#define CM_T3_ROW_BASE 256
#endif

// log2 of the FP64 rows from which the operator's row passes load the next tile
// before they transform the present one: with one or two blocks per SM nothing
// else runs under the loads (operator FP64 4096^2 393 -> 369 us, 2048^2 90.5 ->
// 88.4); shorter rows have a tile or two per block (1024^2 22.9 -> 23.3)
#ifndef CM_ROW_AHEAD
#define CM_ROW_AHEAD 11
#endif

// default log2 elements per thread (per part) of the row passes for length
// code L (cm_fft_p2.cuh): FP64 transforms of length 2^13 take 16 elements
// per thread (512 threads a sequence)
template <typename R>
constexpr int row_lr(int code) {
  return code >= 32 ? (sizeof(R) == 8 ? CM_T3_LR_F64 : CM_T3_LR_F32)
                    : sizeof(R) == 8 ? (code >= 13 ? 4 : CM_ROW_LR_F64) : CM_ROW_LR_F32;
}

// threads of one block of the row passes for the transform of length code
// LOGN (2^LOGN, or 3 * 2^m for LOGN = CM_T3(m)) with 2^LRV elements of each
// power-of-two part per thread.  ONEBUF: the ping-pong buffers and the
// staged twiddles do not fit a block's shared memory (FP64 at 2^13), so the
// transform runs on one buffer with the twiddles read from global memory;
// ONESTG: one buffer and the staged twiddles fit (FP64 at 3 * 2^11).
template <typename R, int LOGN, int LRV = row_lr<R>(LOGN), int SHORT = 0>
struct OpShape {
  typedef typename CT<R>::C C;
  typedef FftLen<LOGN, LRV> P;
  static constexpr int N = P::N;
  static constexpr int LR = LRV;
  static constexpr int E = P::E;  // elements per thread
  static constexpr int TPS = P::TPS;
  // (SHORT: threads of a block for rows of up to 512 points)
  static constexpr int BASE = SHORT && N <= 512 ? SHORT
                              : P::F == 3 ? CM_T3_ROW_BASE
                                        : (sizeof(R) == 8 ? 256 : CM_ROW_F32_BASE) >> (LR - 3);
  static constexpr int THREADS = TPS > BASE ? TPS : BASE;
  static constexpr int NP = THREADS / TPS;  // row pairs per block
  static constexpr size_t BUF = (size_t)(NP * N + ((NP * N) >> 3) + 1) * sizeof(C);
  static constexpr bool TWO = N * sizeof(C) + 2 * BUF <= CM_SMEM_DYN_MAX;
  // ONESTG: one buffer with the twiddles staged (FP64 at 3 * 2^11)
  static constexpr bool ONESTG = !TWO && N * sizeof(C) + BUF <= CM_SMEM_DYN_MAX;
  static constexpr bool ONEBUF = !TWO && !ONESTG;
  static constexpr size_t SMEM = TWO ? N * sizeof(C) + 2 * BUF : ONESTG ? N * sizeof(C) + BUF : BUF;
  static constexpr size_t STAGE = TWO ? 2 * BUF : BUF;  // bytes for staging input rows
  // resident blocks per SM the kernels are compiled for; one when a block
  // holds more than half of the shared memory
  static constexpr int MINB = SMEM > CM_SMEM_DYN_MAX / 2 ? 1
                              : sizeof(R) == 8 ? CM_FP64_ROW_MINB : CM_ROW_F32_MINB;
  // whether the operator's row passes load the next tile's elements before they
  // transform the present one (registers of the loads in flight)
  static constexpr bool AHEAD = sizeof(R) == 8 && E <= 8 && P::F == 1 && LOGN >= CM_ROW_AHEAD;
  static size_t smem() { return SMEM; }
};

// Column pass for columns of length code LOGX: 16 elements per thread for
// 2^LOGX (3 x 2^LR for 3 * 2^m), groups of W = 2^LW columns with the column
// index fastest across threads.  FEW: for grids of few columns, where two
// buffers (one barrier an exchange) and, for them, a column less per group beat
// whole sectors and pairs of blocks: as long as it takes no more waves of
// blocks, or for 3 * 2^m no more than 8/5 times as many (FP64 operator 2048 x
// 384 37.1 us, 29.6 so; 4096 x 256 33.0 and 26.1, 4096 x 384, two waves against
// one, 50.4 and 57.9; 3072 x 256 31.3 and 23.2, 3072 x 768, three against two,
// 70.3 and 64.6, 3072 x 1024, four against two, 70.7 and 76.3).
template <typename R, int LOGX, int BASE = CM_COL_BASE, bool FEW = false>
struct ColShape {
  typedef typename CT<R>::C C;
  static constexpr int LR = LenCode<LOGX>::F == 3 ? (sizeof(R) == 8 ? CM_T3_LR_F64 : CM_T3_LR_F32)
                            : sizeof(R) == 8 ? CM_COL_LR_F64 : CM_COL_LR_F32;
  typedef FftLen<LOGX, LR> P;
  static constexpr int NX = P::N;
  static constexpr int E = P::E;  // elements per thread
  static constexpr int TPS = P::TPS;
  // shared memory of nbuf buffers of 2^lw columns beside the staged twiddles
  static constexpr size_t smem_for(int lw, int nbuf) {
    return (size_t)(NX + nbuf * (NX << lw)) * sizeof(C);
  }
  // 32 bytes of complex values per column group (whole sectors of the spectrum),
  // fewer if not even one buffer of them fits
  static constexpr int LW_PREF = sizeof(C) == 8 ? CM_COL_LW_F32 : CM_COL_LW_F64;
  static constexpr bool fits(int lw, int nbuf) { return smem_for(lw, nbuf) <= CM_SMEM_DYN_MAX; }
  static constexpr bool takes(int lw) { return fits(lw, FEW ? 2 : 1) && (P::TPS << lw) <= 512; }
  static constexpr int LW = takes(LW_PREF) ? LW_PREF : takes(LW_PREF - 1) ? LW_PREF - 1 : 0;
  static constexpr int W = 1 << LW;
  static constexpr int GROUP = W * TPS;
  static constexpr int THREADS = GROUP > BASE ? GROUP : BASE;
  static constexpr int NG = THREADS / GROUP;  // column groups per block
  static constexpr size_t BUF = (size_t)NG * NX * W * sizeof(C);
  // Two buffers (an exchange costs one barrier) unless one buffer (two
  // barriers) lets two blocks share an SM or is all that fits; without room for
  // the twiddles beside one buffer they are read from the global table (ONEBUF:
  // FP64 at 2^13).
  static constexpr size_t TWS = NX * sizeof(C);
  static constexpr bool PAIRED = CM_COL_PAIR(R, LOGX) && !FEW;
  static constexpr bool FIT2 = TWS + 2 * BUF <= CM_SMEM_DYN_MAX, FIT1 = TWS + BUF <= CM_SMEM_DYN_MAX;
  static constexpr bool PAIR2 = 2 * (TWS + 2 * BUF) <= CM_SMEM_DYN_MAX, PAIR1 = 2 * (TWS + BUF) <= CM_SMEM_DYN_MAX;
  static constexpr bool TWO = FIT2 && (PAIR2 || !PAIR1 || !PAIRED);
  static constexpr bool ONESTG = !TWO && FIT1;
  static constexpr bool ONEBUF = !TWO && !ONESTG;
  static constexpr size_t SMEM = TWO ? TWS + 2 * BUF : ONESTG ? TWS + BUF : BUF;
  // resident blocks per SM the registers are sized for
  static constexpr int MINB = PAIRED && 2 * SMEM <= CM_SMEM_DYN_MAX && THREADS <= 256 ? 2 : 1;
  static size_t smem() { return SMEM; }
};

// The operator's own row passes: blocks of 64 threads on rows of up to 512
// points, for the same reason as CM_COL_BASE_SHORT (a solve's row passes keep
// theirs, the order of their sums with it).  FP64 rows of 64, 384 and 512
// points go back to the large blocks where those give every second SM one: the
// small ones, each with the twiddles of a row or two, are then too many (2048 x
// 384 29.8 us, 25.1 in large blocks; 8192 x 512 146 and 131; 6144 x 64 37.6 and
// 34.3; but 1024 x 384 22.1 and 23.1, 6144 x 256 41.7 and 43.6).
template <typename R, int LOGN, bool SMALL = true>
using OpRowShape = OpShape<R, LOGN, row_lr<R>(LOGN), SMALL ? 64 : 0>;
template <typename R, int LOGN>
constexpr bool op_row_both() {
  return sizeof(R) == 8 && (LenCode<LOGN>::N <= 64 || (LenCode<LOGN>::N > 256 && LenCode<LOGN>::N <= 512));
}

template <typename R, int LOGN, bool SMALL = true>
__global__ void __launch_bounds__(OpRowShape<R, LOGN, SMALL>::THREADS, OpRowShape<R, LOGN, SMALL>::MINB)
k_op_row_fwd(OpArgs<R> a) {
  typedef typename CT<R>::C C;
  typedef OpRowShape<R, LOGN, SMALL> Sh;
  typedef typename Sh::P P;
  constexpr int N = P::N, NP = Sh::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tws = reinterpret_cast<C*>(smem_raw);
  C* bufA = Sh::ONEBUF ? tws : tws + N;
  C* bufB = bufA + smem_padded(NP * N);
  pdl_trigger();
  const C* tw = stage_twiddles<LOGN, Sh::LR, Sh::THREADS, Sh::ONEBUF>(tws, a.twy);
  pdl_wait();
  __syncthreads();
  const int s = threadIdx.x >> P::LTPS, tt = threadIdx.x & (P::TPS - 1);
  const int npairs = (a.in_rows + 1) >> 1;
  auto load = [&](C (&v)[Sh::E], int p) {
    const int xa = 2 * p;
#pragma unroll
    for (int q = 0; q < Sh::E; ++q) {
      const int y = tt + q * P::TPS;
      R ra = 0, rb = 0;
      if (y < a.in_cols) {
        if (xa < a.in_rows) ra = __ldg(a.in + (size_t)xa * a.in_ld + y);
        if (xa + 1 < a.in_rows) rb = __ldg(a.in + (size_t)(xa + 1) * a.in_ld + y);
      }
      v[q] = cmake<C>(ra, rb);
    }
  };
  C ahead[Sh::E];
  if (Sh::AHEAD) load(ahead, blockIdx.x * NP + s);
  for (int p0 = blockIdx.x * NP; p0 < npairs; p0 += gridDim.x * NP) {
    const int p = p0 + s;
    C v[Sh::E];
    if (Sh::AHEAD) {
#pragma unroll
      for (int q = 0; q < Sh::E; ++q) v[q] = ahead[q];
      load(ahead, p + gridDim.x * NP);
    } else {
      load(v, p);
    }
    fft_len<C, false, LOGN, Sh::LR, Sh::ONEBUF, Sh::ONESTG>(v, bufA, bufB, s * N, 1, tt, tw);
    if (p < npairs) {
      C* __restrict__ row = a.spec + (size_t)p * N;
#pragma unroll
      for (int q = 0; q < Sh::E; ++q) row[kfreq<LOGN, Sh::LR>(tt, q)] = v[q];
    }
    __syncthreads();  // buffers free for the next pairs
  }
}

// Loads of one column unit k of the pair-major spectrum (rows x = 2p + b of
// the thread's elements x = tt + q TPS, b = tt & 1): both rows of a pair load
// Z_p(k) and Z_p(ny - k) (neighbouring lanes, one request) and each splits
// off its own row.  Rows >= in_rows are zero.  CG: loads bypass L1 (a launch
// whose other blocks write the spectrum).
template <typename C, int TPS, int E, bool CG = false>
CM_DEVINL void col_split_load(C (&v)[E], const C* __restrict__ spec, int ny, int k, int km, int tt,
                              int in_rows, bool ok) {
  typedef decltype(v[0].x) R;
  const int b = tt & 1;
  const C* __restrict__ sk = spec + k + (size_t)(tt >> 1) * ny;
  const C* __restrict__ skm = spec + km + (size_t)(tt >> 1) * ny;
  const int pstep = (TPS / 2) * ny;
  constexpr int CH = E % 8 == 0 ? 8 : 4;  // loads in flight per chunk
#pragma unroll
  for (int h = 0; h < E; h += CH) {
    C z[CH], zm[CH];
#pragma unroll
    for (int q = h; q < h + CH; ++q) {
      const int x = tt + q * TPS;
      z[q - h] = czero<C>();
      zm[q - h] = czero<C>();
      if (ok && x < in_rows) {
        z[q - h] = CG ? __ldcg(sk + (size_t)q * pstep) : sk[(size_t)q * pstep];
        zm[q - h] = CG ? __ldcg(skm + (size_t)q * pstep) : skm[(size_t)q * pstep];
      }
    }
#pragma unroll
    for (int q = h; q < h + CH; ++q) {
      const C zk = z[q - h], zn = zm[q - h];
      v[q] = b ? cmake<C>((zk.y + zn.y) * (R)0.5, (zn.x - zk.x) * (R)0.5)
               : cmake<C>((zk.x + zn.x) * (R)0.5, (zk.y - zn.y) * (R)0.5);
    }
  }
}

// Pack the filtered column back into the pair-major spectrum: the even row of
// a pair writes W_p(k) = Xh_2p + i Xh_2p+1 (real parts only for the
// self-conjugate columns 0 and ny/2), the odd row W_p(ny - k); pairs with
// rows < out_rows.
template <typename C, int TPS, int W, int E>
CM_DEVINL void col_pack_store(const C (&v)[E], C* __restrict__ spec, int ny, int k, int km, int tt,
                              int out_rows, bool ok) {
  const int b = tt & 1;
  const int pairs_out = (out_rows + 1) >> 1;
  const bool selfc = (k == 0) || (2 * k == ny);
  const bool writes = ok && !(b && selfc);
  C* __restrict__ dst = spec + (b ? km : k) + (size_t)(tt >> 1) * ny;
  const int pstep = (TPS / 2) * ny;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const C a = v[q];
    C o;
    o.x = __shfl_xor_sync(0xffffffffu, a.x, W);
    o.y = __shfl_xor_sync(0xffffffffu, a.y, W);
    const int pp = (tt >> 1) + q * (TPS / 2);
    if (!writes || pp >= pairs_out) continue;
    dst[(size_t)q * pstep] = !b ? (selfc ? cmake<C>(a.x, o.x) : cmake<C>(a.x - o.y, a.y + o.x))
                                : cmake<C>(o.x + a.y, a.x - o.y);
  }
}

template <typename R, int LOGX, int BASE = CM_COL_BASE, bool FEW = false>
__global__ void __launch_bounds__(ColShape<R, LOGX, BASE, FEW>::THREADS, ColShape<R, LOGX, BASE, FEW>::MINB)
k_op_col(OpArgs<R> a) {
  typedef typename CT<R>::C C;
  typedef ColShape<R, LOGX, BASE, FEW> Sh;
  typedef typename Sh::P P;
  constexpr int NX = P::N, W = Sh::W, LW = Sh::LW, E = Sh::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tws = reinterpret_cast<C*>(smem_raw);
  C* bufA = Sh::ONEBUF ? tws : tws + NX;
  C* bufB = bufA + Sh::NG * NX * W;
  if (!a.st) pdl_trigger();  // (one call's inverse rows; a solve's launches follow its tiles)
  const C* tw = stage_twiddles<LOGX, Sh::LR, Sh::THREADS, Sh::ONEBUF>(tws, a.twx);
  pdl_wait();
  if (a.st && (a.st->done || (a.cg_only && a.st->branch != 0))) return;
  __syncthreads();
  const int ny = a.ny;
  const int c = threadIdx.x & (W - 1);
  const int tt = (threadIdx.x >> LW) & (P::TPS - 1);
  const int j = threadIdx.x >> (LW + P::LTPS);
  const int units = ny / 2 + 1;
  const int ngroups = (units + W - 1) >> LW;
  const int base = j * NX * W + c;
  const int tlw = a.lw, tW = 1 << tlw;  // the table's column tiles
  for (int g0 = blockIdx.x * Sh::NG; g0 < ngroups; g0 += gridDim.x * Sh::NG) {
    const int k = (g0 + j) * W + c;
    const bool ok = k < units;
    const int km = k == 0 ? 0 : ny - k;  // the mirror column (ny need not be a power of two)
    C v[E];
    col_split_load<C, P::TPS, E>(v, a.spec, ny, k, km, tt, a.in_rows, ok);
    fft_len<C, false, LOGX, Sh::LR, Sh::ONEBUF, Sh::ONESTG>(v, bufA, bufB, base, W, tt, tw);
    if (a.fwd_real) {
      // forward transform only: the real part of the 2D transform, in the
      // natural (nx, ny/2 + 1) layout (a real, even kernel's Green's table)
      if (ok) {
#pragma unroll
        for (int q = 0; q < E; ++q) a.fwd_real[(size_t)kfreq<LOGX, Sh::LR>(tt, q) * units + k] = v[q].x;
      }
      __syncthreads();
      continue;
    }
    // the table's row of register q: its frequency index along x
    const R* __restrict__ tb = a.tab + ((size_t)(k >> tlw) * NX << tlw) + (k & (tW - 1)) +
                               (P::F == 1 ? (size_t)tt << tlw : 0);
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const size_t row = P::F == 1 ? (size_t)(q * P::TPS) : (size_t)kfreq<LOGX, Sh::LR>(tt, q);
      v[q] = cscale(v[q], ok ? __ldg(tb + (row << tlw)) : (R)0);
    }
    __syncthreads();
    fft_len<C, true, LOGX, Sh::LR, Sh::ONEBUF, Sh::ONESTG>(v, bufA, bufB, base, W, tt, tw);
    col_pack_store<C, P::TPS, W, E>(v, a.spec, ny, k, km, tt, a.out_rows, ok);
    __syncthreads();  // buffers free for the next group
  }
  // (a no-op after the one above; a test for it spills: 8192^2 FP64 1423 us a
  // launch, 1362 without)
  pdl_trigger();
}

template <typename R, int LOGN, bool SMALL = true>
__global__ void __launch_bounds__(OpRowShape<R, LOGN, SMALL>::THREADS, OpRowShape<R, LOGN, SMALL>::MINB)
k_op_row_inv(OpArgs<R> a) {
  typedef typename CT<R>::C C;
  typedef OpRowShape<R, LOGN, SMALL> Sh;
  typedef typename Sh::P P;
  constexpr int N = P::N, NP = Sh::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tws = reinterpret_cast<C*>(smem_raw);
  C* bufA = Sh::ONEBUF ? tws : tws + N;
  C* bufB = bufA + smem_padded(NP * N);
  pdl_trigger();
  const C* tw = stage_twiddles<LOGN, Sh::LR, Sh::THREADS, Sh::ONEBUF>(tws, a.twy);
  pdl_wait();
  __syncthreads();
  const int s = threadIdx.x >> P::LTPS, tt = threadIdx.x & (P::TPS - 1);
  const int npairs = (a.out_rows + 1) >> 1;
  auto load = [&](C (&v)[Sh::E], int p) {
    const C* __restrict__ row = a.spec + (size_t)p * N;
#pragma unroll
    for (int q = 0; q < Sh::E; ++q) v[q] = p < npairs ? row[kfreq<LOGN, Sh::LR>(tt, q)] : czero<C>();
  };
  C ahead[Sh::E];
  if (Sh::AHEAD) load(ahead, blockIdx.x * NP + s);
  for (int p0 = blockIdx.x * NP; p0 < npairs; p0 += gridDim.x * NP) {
    const int p = p0 + s, xa = 2 * p;
    C v[Sh::E];
    if (Sh::AHEAD) {
#pragma unroll
      for (int q = 0; q < Sh::E; ++q) v[q] = ahead[q];
      load(ahead, p + gridDim.x * NP);
    } else {
      load(v, p);
    }
    fft_len<C, true, LOGN, Sh::LR, Sh::ONEBUF, Sh::ONESTG>(v, bufA, bufB, s * N, 1, tt, tw);
#pragma unroll
    for (int q = 0; q < Sh::E; ++q) {
      const int y = tt + q * P::TPS;
      if (y >= a.out_cols) continue;
      if (xa < a.out_rows) a.out[(size_t)xa * a.out_ld + y] = v[q].x;
      if (xa + 1 < a.out_rows) a.out[(size_t)(xa + 1) * a.out_ld + y] = v[q].y;
    }
    __syncthreads();  // buffers free for the next pairs
  }
}
