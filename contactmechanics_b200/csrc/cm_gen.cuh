// Transforms of any length in shared memory, and the operator passes built on
// them: the counterpart of cm_fft_p2.cuh / cm_op_p2.cuh for sides that are
// neither 2^k nor 3 * 2^m, on the same pair-major spectrum (a domain may take
// one engine along x and the other along y).
//
// A Stockham transform whose radices (2..10, 12, 14, 15, 16) are chosen per
// length for the fewest stages: every stage is a trip through shared memory
// and a block barrier, and on the grids this serves the passes are bound by
// that chain, not by arithmetic (500 = 10 * 5 * 10, 360 = 9 * 4 * 10).  Small
// DFTs use the symmetry of their outputs (cos and sin sums of x_p +- x_(r-p))
// and constants; divisions by stage sizes are multiply-shift.
//
// Other prime factors r take one stage of direct sums with the same symmetry:
// the pairs x_p +- x_(r-p) are formed once in place, then a thread
// accumulates the outputs q and r - q for two q at a time, 4 r^2 / 4 real
// multiply-adds a butterfly spread over r / 4 threads, the root's index kept
// by addition.  (Recomputing twiddled inputs and (p q) mod r inside a double
// loop on one thread per butterfly, the 73-point stages of a 511 x 256
// domain took 534 us a column pass; here 12.)
// Its rounding against numpy in 64 bits, mixed-radix passes / these (medians of
// five rough fields): displacements 1010 x 1370 FP64 8.4e-16 / 6.5e-16, 590 x 610
// FP32 2.7e-7 / 1.8e-7; forces, whose stiffness amplifies the shortest waves,
// 299 x 253 FP64 7.2e-15 / 6.9e-15, 1010 x 1370 3.5e-14 / 3.7e-14, 1990 x 64 (a
// factor 199) 7.3e-14 / 8.9e-14.
//
// Operator FP64, mixed-radix passes / these: 500 x 300 49.2 / 22.6 us, 1000^2
// 63.6 / 50, 167^2 2750 / 33, 511 x 256 565 / 20.5.  Bound by the stages'
// latency and instruction fetches on small grids: radices up to 5, 6 or 9 only gave the same times up to
// 500^2 and lost at 1000^2 (47 -> 58-63).
#pragma once
#include "cm_fft_p2.cuh"
#include "cm_kernels.cuh"
#include "cm_launch.h"

template <typename C, bool INV>
CM_DEVINL void gdft2(C& a, C& b) {
  const C t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

// c -+ i s: the outputs q and r - q of a DFT of odd length from their cos sum
// c and sin sum s
template <bool INV, typename C>
CM_DEVINL void gpair(C c, C s, C& yq, C& yr) {
  yq = INV ? cmake<C>(c.x - s.y, c.y + s.x) : cmake<C>(c.x + s.y, c.y - s.x);
  yr = INV ? cmake<C>(c.x + s.y, c.y - s.x) : cmake<C>(c.x - s.y, c.y + s.x);
}

template <typename C, bool INV>
CM_DEVINL void gdft3(C& x0, C& x1, C& x2) {
  typedef decltype(x0.x) R;
  const R s3 = (R)0.86602540378443864676;
  const C a = cadd(x1, x2), b = cscale(csub(x1, x2), s3);
  const C m = cmake<C>(x0.x - (R)0.5 * a.x, x0.y - (R)0.5 * a.y);
  x0 = cadd(x0, a);
  gpair<INV>(m, b, x1, x2);
}

template <typename C, bool INV>
CM_DEVINL void gdft5(C& x0, C& x1, C& x2, C& x3, C& x4) {
  typedef decltype(x0.x) R;
  const R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;
  const R s1 = (R)0.95105651629515357212, s2 = (R)0.58778525229247312917;
  const C a1 = cadd(x1, x4), b1 = csub(x1, x4), a2 = cadd(x2, x3), b2 = csub(x2, x3);
  const C m1 = cmake<C>(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
  const C m2 = cmake<C>(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
  const C n1 = cmake<C>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
  const C n2 = cmake<C>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
  x0 = cadd(x0, cadd(a1, a2));
  gpair<INV>(m1, n1, x1, x4);
  gpair<INV>(m2, n2, x2, x3);
}

template <typename C, bool INV>
CM_DEVINL void gdft7(C& x0, C& x1, C& x2, C& x3, C& x4, C& x5, C& x6) {
  typedef decltype(x0.x) R;
  const R c1 = (R)0.62348980185873353053, c2 = (R)-0.22252093395631440429,
          c3 = (R)-0.90096886790241912624;
  const R s1 = (R)0.78183148246802980871, s2 = (R)0.97492791218182360702,
          s3 = (R)0.43388373911755812048;
  const C a1 = cadd(x1, x6), b1 = csub(x1, x6), a2 = cadd(x2, x5), b2 = csub(x2, x5);
  const C a3 = cadd(x3, x4), b3 = csub(x3, x4);
  const C m1 = cmake<C>(x0.x + c1 * a1.x + c2 * a2.x + c3 * a3.x, x0.y + c1 * a1.y + c2 * a2.y + c3 * a3.y);
  const C m2 = cmake<C>(x0.x + c2 * a1.x + c3 * a2.x + c1 * a3.x, x0.y + c2 * a1.y + c3 * a2.y + c1 * a3.y);
  const C m3 = cmake<C>(x0.x + c3 * a1.x + c1 * a2.x + c2 * a3.x, x0.y + c3 * a1.y + c1 * a2.y + c2 * a3.y);
  const C n1 = cmake<C>(s1 * b1.x + s2 * b2.x + s3 * b3.x, s1 * b1.y + s2 * b2.y + s3 * b3.y);
  const C n2 = cmake<C>(s2 * b1.x - s3 * b2.x - s1 * b3.x, s2 * b1.y - s3 * b2.y - s1 * b3.y);
  const C n3 = cmake<C>(s3 * b1.x - s1 * b2.x + s2 * b3.x, s3 * b1.y - s1 * b2.y + s2 * b3.y);
  x0 = cadd(x0, cadd(a1, cadd(a2, a3)));
  gpair<INV>(m1, n1, x1, x6);
  gpair<INV>(m2, n2, x2, x5);
  gpair<INV>(m3, n3, x3, x4);
}

// a W9^M, M in {1, 2, 4}
template <bool INV, int M, typename C>
CM_DEVINL C gw9(C a) {
  typedef decltype(a.x) R;
  const R c = M == 1 ? (R)0.76604444311897803520 : M == 2 ? (R)0.17364817766693034885
                                                          : (R)-0.93969262078590838405;
  const R s = M == 1 ? (R)0.64278760968653932632 : M == 2 ? (R)0.98480775301220805937
                                                          : (R)0.34202014332566873304;
  return INV ? cmake<C>(a.x * c - a.y * s, a.x * s + a.y * c)
             : cmake<C>(a.x * c + a.y * s, a.y * c - a.x * s);
}

// DFT of length RR in registers, natural order in and out.  Lengths with
// coprime factors use the prime-factor index maps (no twiddles between).
template <typename C, bool INV, int RR>
CM_DEVINL void gdft(C (&v)[RR]) {
  if constexpr (RR == 2) gdft2<C, INV>(v[0], v[1]);
  else if constexpr (RR == 3) gdft3<C, INV>(v[0], v[1], v[2]);
  else if constexpr (RR == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (RR == 5) gdft5<C, INV>(v[0], v[1], v[2], v[3], v[4]);
  else if constexpr (RR == 7) gdft7<C, INV>(v[0], v[1], v[2], v[3], v[4], v[5], v[6]);
  else if constexpr (RR == 8) Dft<INV, 8, C>::run(v, nullptr, 8);
  else if constexpr (RR == 16) dft16<INV>(v);
  else if constexpr (RR == 9) {
    C y[9];  // y[n2][k1]
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
      C a = v[n2], b = v[3 + n2], c = v[6 + n2];
      gdft3<C, INV>(a, b, c);
      y[3 * n2] = a; y[3 * n2 + 1] = b; y[3 * n2 + 2] = c;
    }
    y[4] = gw9<INV, 1>(y[4]);
    y[5] = gw9<INV, 2>(y[5]);
    y[7] = gw9<INV, 2>(y[7]);
    y[8] = gw9<INV, 4>(y[8]);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      C a = y[k1], b = y[3 + k1], c = y[6 + k1];
      gdft3<C, INV>(a, b, c);
      v[k1] = a; v[k1 + 3] = b; v[k1 + 6] = c;
    }
  } else if constexpr (RR == 6 || RR == 10 || RR == 14) {
    constexpr int H = RR / 2;
    constexpr int K2 = RR == 6 ? 4 : RR == 10 ? 6 : 8;  // output step of the odd factor
    C y[2][H];
#pragma unroll
    for (int n1 = 0; n1 < 2; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < H; ++n2) y[n1][n2] = v[(H * n1 + 2 * n2) % RR];
      gdft<C, INV, H>(y[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < H; ++k2) {
      gdft2<C, INV>(y[0][k2], y[1][k2]);
#pragma unroll
      for (int k1 = 0; k1 < 2; ++k1) v[(H * k1 + K2 * k2) % RR] = y[k1][k2];
    }
  } else if constexpr (RR == 12) {
    C y[4][3];
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 3; ++n2) y[n1][n2] = v[(3 * n1 + 4 * n2) % 12];
      gdft3<C, INV>(y[n1][0], y[n1][1], y[n1][2]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) {
      dft4<INV>(y[0][k2], y[1][k2], y[2][k2], y[3][k2]);
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1) v[(9 * k1 + 4 * k2) % 12] = y[k1][k2];
    }
  } else {
    static_assert(RR == 15, "radix");
    C y[3][5];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 5; ++n2) y[n1][n2] = v[(5 * n1 + 3 * n2) % 15];
      gdft5<C, INV>(y[n1][0], y[n1][1], y[n1][2], y[n1][3], y[n1][4]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 5; ++k2) {
      gdft3<C, INV>(y[0][k2], y[1][k2], y[2][k2]);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) v[(10 * k1 + 6 * k2) % 15] = y[k1][k2];
    }
  }
}

#define CM_GEN_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16)

// Where element i of sequence s sits: rows s * n + i, columns i << lw | s.
template <bool COL>
struct GenLayout {
  int n, lw;
  CM_DEVINL int at(int s, int i) const { return COL ? (i << lw) + s : s * n + i; }
};

// One stage of radix RR.  scale(s, i): factor of input element i of sequence
// s (the Green's table before an inverse column transform), or 1.
template <typename C, bool INV, bool COL, int RR, typename Scale>
CM_DEVINL void gen_stage(const C* src, C* dst, const GenStage& S, int n, int nseq, int lw,
                         const C* tw, Scale scale) {
  const int m = S.m, B = m * nseq, Ns = S.Ns;
  const GenLayout<COL> L{n, lw};
  for (int bi = threadIdx.x; bi < B; bi += blockDim.x) {
    const int s = COL ? bi & ((1 << lw) - 1) : fdiv(S.dm, bi);
    const int j = COL ? bi >> lw : bi - s * m;
    const int k = j - fdiv(S.dns, j) * Ns;
    C v[RR];
#pragma unroll
    for (int q = 0; q < RR; ++q) v[q] = src[L.at(s, j + q * m)];
    scale.template apply<RR>(v, s, j, m);
    if (Ns > 1) {
      const int idx = k * S.step;
#pragma unroll
      for (int q = 1; q < RR; ++q) {
        const C w = tw[q * idx];
        v[q] = INV ? cmulc(v[q], w) : cmul(v[q], w);
      }
    }
    gdft<C, INV, RR>(v);
    const int o = (j - k) * RR + k;
#pragma unroll
    for (int q = 0; q < RR; ++q) dst[L.at(s, o + q * Ns)] = v[q];
  }
  __syncthreads();
}

// One stage of any other (odd) radix r: see the head of this file.
template <typename C, bool INV, bool COL, typename Scale>
CM_DEVINL void gen_stage_prime(C* src, C* dst, const GenStage& S, int n, int nseq, int lw,
                               const C* tw, Scale scale) {
  typedef decltype(src->x) R;
  const int r = S.r, m = S.m, Ns = S.Ns, h = (r - 1) >> 1;
  const int B = S.db.d;  // butterflies of a full tile (the last may have fewer sequences)
  const GenLayout<COL> L{n, lw};
  for (int bi = threadIdx.x; bi < B * h; bi += blockDim.x) {
    const int p1 = fdiv(S.db, bi), b = bi - p1 * B, p = p1 + 1;
    const int s = COL ? b & ((1 << lw) - 1) : fdiv(S.dm, b);
    if (s >= nseq) continue;
    const int j = COL ? b >> lw : b - s * m;
    C *xa = src + L.at(s, j + p * m), *xb = src + L.at(s, j + (r - p) * m);
    C va[1] = {*xa}, vb[1] = {*xb};
    scale.template apply<1>(va, s, j + p * m, m);
    scale.template apply<1>(vb, s, j + (r - p) * m, m);
    if (Ns > 1) {
      const int idx = (j - fdiv(S.dns, j) * Ns) * S.step;
      const C wa = tw[p * idx], wb = tw[(r - p) * idx];
      va[0] = INV ? cmulc(va[0], wa) : cmul(va[0], wa);
      vb[0] = INV ? cmulc(vb[0], wb) : cmul(vb[0], wb);
    }
    *xa = cadd(va[0], vb[0]);
    *xb = csub(va[0], vb[0]);
  }
  __syncthreads();
  const int ws = S.m;  // W_r = tw[n / r]
  const int ng = (h + 1) >> 1;
  for (int bi = threadIdx.x; bi < B * ng; bi += blockDim.x) {
    const int g = fdiv(S.db, bi), b = bi - g * B;
    const int s = COL ? b & ((1 << lw) - 1) : fdiv(S.dm, b);
    if (s >= nseq) continue;
    const int j = COL ? b >> lw : b - s * m;
    const int k = j - fdiv(S.dns, j) * Ns;
    const int q0 = 2 * g + 1, q1 = q0 + 1;
    C x0[1] = {src[L.at(s, j)]};
    scale.template apply<1>(x0, s, j, m);
    C c0 = x0[0], c1 = x0[0], s0 = czero<C>(), s1 = czero<C>(), y0 = x0[0];
    int i0 = 0, i1 = 0;
    for (int p = 1; p <= h; ++p) {
      i0 += q0; if (i0 >= r) i0 -= r;
      i1 += q1; if (i1 >= r) i1 -= r;
      const C a = src[L.at(s, j + p * m)], d = src[L.at(s, j + (r - p) * m)];
      const C w0 = tw[i0 * ws], w1 = tw[i1 * ws];  // cos - i sin
      c0.x += w0.x * a.x; c0.y += w0.x * a.y;
      s0.x -= w0.y * d.x; s0.y -= w0.y * d.y;
      c1.x += w1.x * a.x; c1.y += w1.x * a.y;
      s1.x -= w1.y * d.x; s1.y -= w1.y * d.y;
      if (g == 0) y0 = cadd(y0, a);
    }
    const int o = (j - k) * r + k;
    C yq, yr;
    gpair<INV>(c0, s0, yq, yr);
    dst[L.at(s, o + q0 * Ns)] = yq;
    dst[L.at(s, o + (r - q0) * Ns)] = yr;
    if (q1 <= h) {
      gpair<INV>(c1, s1, yq, yr);
      dst[L.at(s, o + q1 * Ns)] = yq;
      dst[L.at(s, o + (r - q1) * Ns)] = yr;
    }
    if (g == 0) dst[L.at(s, o)] = y0;
  }
  __syncthreads();
}

struct GenNoScale {
  template <int RR, typename C>
  CM_DEVINL void apply(C (&)[RR], int, int, int) const {}
};

// Green's table of columns k0.. (column tiles of width 2^tlw, rows of length
// nx): factor of element x of column s
template <typename R>
struct GenTableScale {
  const R* tab;
  int nx, tlw, k0, units;
  template <int RR, typename C>
  CM_DEVINL void apply(C (&v)[RR], int s, int j, int m) const {
    const int k = k0 + s;
    const R* tb = tab + (((size_t)(k >> tlw) * nx) << tlw) + (k & ((1 << tlw) - 1));
    R f[RR];
#pragma unroll
    for (int q = 0; q < RR; ++q) f[q] = k < units ? __ldg(tb + ((size_t)(j + q * m) << tlw)) : (R)0;
#pragma unroll
    for (int q = 0; q < RR; ++q) v[q] = cscale(v[q], f[q]);
  }
};

template <typename C, bool INV, bool COL, typename Scale>
CM_DEVINL void gen_stage_any(C* src, C* dst, const GenStage& S, int n, int nseq, int lw,
                             const C* tw, Scale scale) {
  switch (S.r) {
#define CM_CASE(RR) case RR: gen_stage<C, INV, COL, RR>(src, dst, S, n, nseq, lw, tw, scale); break;
    CM_GEN_RADICES(CM_CASE)
#undef CM_CASE
    default: gen_stage_prime<C, INV, COL>(src, dst, S, n, nseq, lw, tw, scale); break;
  }
}

// Transform nseq sequences (columns: 2^lw of them) that start in a; b is a
// buffer of the same size.  Begins after and ends with a block barrier;
// returns the buffer that holds the result.  The first stage applies `scale`
// to its inputs (a transform of length 1 has no stage: unscaled).
template <typename C, bool INV, bool COL, typename Scale = GenNoScale>
__device__ __noinline__ C* gen_fft(C* a, C* b, const GenFft& F, int nseq, int lw, const C* tw,
                                   Scale scale = Scale()) {
  for (int st = 0; st < F.nst; ++st) {
    if (st == 0) gen_stage_any<C, INV, COL>(a, b, F.st[0], F.n, nseq, lw, tw, scale);
    else gen_stage_any<C, INV, COL>(a, b, F.st[st], F.n, nseq, lw, tw, GenNoScale());
    C* t = a;
    a = b;
    b = t;
  }
  return a;
}

// Column units k0 .. k0 + 2^lw of the pair-major spectrum: split off the row
// pairs (see cm_op_p2.cuh), transform, multiply by the table, transform back,
// pack.  Loads bypass L1 (a launch whose other blocks write the spectrum).
template <typename R>
CM_DEVINL void gen_col_tile(const OpArgs<R>& a, const GenFft& F, int k0, int lw, int out_rows,
                            const typename CT<R>::C* tw, typename CT<R>::C* bufA,
                            typename CT<R>::C* bufB) {
  typedef typename CT<R>::C C;
  const int nx = a.nx, ny = a.ny, W = 1 << lw, units = ny / 2 + 1;
  const int pin = (a.in_rows + 1) >> 1;  // pairs with input rows
  struct ZZ { C z, m; };
  const GenLayout<true> L{nx, lw};
  batched_loop<4>(pin << lw, [&](int e) {
    const int p = e >> lw, k = k0 + (e & (W - 1));
    ZZ v{czero<C>(), czero<C>()};
    if (k < units) {
      v.z = __ldcg(a.spec + (size_t)p * ny + k);
      v.m = __ldcg(a.spec + (size_t)p * ny + (k == 0 ? 0 : ny - k));
    }
    return v;
  }, [&](int e, const ZZ& v) {
    const int p = e >> lw, c = e & (W - 1), x = 2 * p;
    bufA[L.at(c, x)] = cmake<C>((v.z.x + v.m.x) * (R)0.5, (v.z.y - v.m.y) * (R)0.5);
    if (x + 1 < nx)
      bufA[L.at(c, x + 1)] = x + 1 < a.in_rows
                                 ? cmake<C>((v.z.y + v.m.y) * (R)0.5, (v.m.x - v.z.x) * (R)0.5)
                                 : czero<C>();
  });
  for (int e = (2 * pin << lw) + threadIdx.x; e < nx << lw; e += blockDim.x) bufA[e] = czero<C>();
  __syncthreads();
  C* res = gen_fft<C, false, true>(bufA, bufB, F, W, lw, tw);
  C* other = res == bufA ? bufB : bufA;
  const GenTableScale<R> scale{a.tab, nx, a.lw, k0, units};
  if (F.nst == 0) {  // one row
    for (int e = threadIdx.x; e < W; e += blockDim.x) {
      C v[1] = {res[e]};
      scale.template apply<1>(v, e, 0, 1);
      res[e] = v[0];
    }
    __syncthreads();
  } else {
    res = gen_fft<C, true, true, GenTableScale<R>>(res, other, F, W, lw, tw, scale);
  }
  const int pout = (out_rows + 1) >> 1;
  for (int e = threadIdx.x; e < pout << lw; e += blockDim.x) {
    const int p = e >> lw, c = e & (W - 1), k = k0 + c, x = 2 * p;
    if (k >= units) continue;
    const C A = res[L.at(c, x)], B = x + 1 < nx ? res[L.at(c, x + 1)] : czero<C>();
    C* row = a.spec + (size_t)p * ny;
    if (k == 0 || 2 * k == ny) {
      row[k] = cmake<C>(A.x, B.x);
    } else {
      row[k] = cmake<C>(A.x - B.y, A.y + B.x);
      row[ny - k] = cmake<C>(A.x + B.y, B.x - A.y);
    }
  }
  __syncthreads();
}

// stage the plan and the twiddles of one length
template <typename C>
CM_DEVINL void gen_stage_tables(GenFft& F, const GenFft& src, C* tws, const C* __restrict__ tw) {
  const int nint = (int)(sizeof(GenFft) / sizeof(int));
  for (int i = threadIdx.x; i < nint; i += blockDim.x)
    reinterpret_cast<int*>(&F)[i] = reinterpret_cast<const int*>(&src)[i];
  for (int i = threadIdx.x; i < src.n; i += blockDim.x) tws[i] = __ldg(tw + i);
}
