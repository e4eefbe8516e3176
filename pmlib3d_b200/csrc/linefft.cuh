// linefft.cuh -- line FFTs of the y and z passes: 16-byte line vectors, transformed in
// place in shared memory.
//
// A tile holds the points of a few neighbouring lines, interleaved by position: the
// vector of line group g at position q sits at buf[q * LG + g].  A vector is 16 bytes:
// in FP32 one point of two lines whose kx indices are neighbours, as (re, re, im, im),
// so that every addition, product and twiddle of the codelets is one FP32x2
// instruction for both lines (no mixing of real and imaginary halves); in FP64 one
// point of one line.  An FP32x2 or FP64 instruction takes two issue cycles of a
// scheduler's 128-lane FMA pipe either way (measured: 2.05 cycles for packed add, mul,
// fma, with or without negated or broadcast operands), so the packed form halves the
// issue slots of the FP32 lines and leaves their other half to loads and indices.
//
// Free axes: the second half of a line's 2n points is zero padding.  The transform is
// split into the two transforms of the even and of the odd frequencies,
//   X[2k + h] = sum_{j < n} (x[j] w_{2n}^{h j}) w_n^{j k},        h = 0, 1,
// each of the n data points, so no butterfly works on padding; the inverse is
//   x[j] = E[j] + conj(w_{2n}^j) O[j],  j < n   (the truncated half is never formed).
// The two halves are positions [0, n) and [n, 2n).
//
// n = r0 r1 r2 (at most three phases).  Phase p works on digit p of the position.
// Consecutive digits form groups; the sizes of the groups are pairwise coprime, and the
// transform over the groups needs no twiddles (Good 1958: row sum_g (n / n_g) i_g mod n
// of the input, frequency by the Chinese remainder of the groups' frequencies); inside
// a group of several digits the phases are decimation in frequency with twiddles
// w_{n_g}.  The first forward phase reads rows of global memory through that row map and
// the last inverse phase writes them, so the map costs no pass of its own.
#pragma once

#include "common.cuh"
#include "fft.cuh"

namespace pmgpu {

// u / d for u < 2^31 by multiply-high (Granlund-Montgomery): l = ceil(log2 d),
// m = floor(2^32 (2^l - d) / d) + 1, q = (umulhi(u, m) + u) >> l
struct FastDiv {
  unsigned d, m, l;
};
static inline FastDiv make_fastdiv(unsigned d) {
  FastDiv f;
  f.d = d;
  unsigned l = 0;
  while ((1ull << l) < d) l++;
  f.l = l;
  f.m = (unsigned)((((1ull << l) - d) << 32) / d + 1);
  return f;
}
__host__ __device__ __forceinline__ unsigned fdiv(unsigned u, const FastDiv &f) {
#ifdef __CUDA_ARCH__
  return (__umulhi(u, f.m) + u) >> f.l;
#else
  return (unsigned)((((unsigned long long)u * f.m) >> 32) + u) >> f.l;
#endif
}

// radices with a register DFT
__host__ __device__ constexpr bool reg_radix(int r) {
  return r == 2 || r == 3 || r == 4 || r == 5 || r == 6 || r == 7 || r == 8 || r == 9 || r == 10 || r == 11 ||
         r == 12 || r == 13 || r == 16 || r == 17;
}
// first digits of a split plan: a thread holds both halves of such a butterfly
__host__ __device__ constexpr bool split_radix(int r) { return r <= 13 || r == 17; }
// further composite radices, FP32 schedules only
__host__ __device__ constexpr bool reg_radix_wide(int r) { return r == 18 || r == 20 || r == 22 || r == 24; }

constexpr int LP_MAX = 3;
struct LinePlan {
  int n;              // points of a (half) transform
  int split;          // 1: line of 2n points whose second half is zero padding
  int np;
  int rad[LP_MAX];    // radix of each phase, outermost first
  int str[LP_MAX];    // position stride of the phase's digit
  int tmul[LP_MAX];   // twiddles after the phase: w_n^(tmul (r / tin) k); 0: none
  int tin[LP_MAX];    // product of the digits of the later groups
  int rstep;          // input rows between consecutive values of digit 0
  FastDiv dstr[LP_MAX], dtin[LP_MAX];
  // Bluestein: a line of length bn (with a prime factor above 17) of which brows points
  // are data is transformed as a convolution of length n >= bn + brows - 1 (the phases
  // above describe that length)
  int bl, bn, brows;
};
// points of a line
__host__ __device__ inline int plan_points(const LinePlan &p) { return p.split ? 2 * p.n : p.n; }

// ------------------------------------------------------------------ line vectors
// T: float2 (two FP32 lines), float (one FP32 line), double (one FP64 line)
template <typename T> struct LineT;
template <> struct LineT<float2> { typedef float R; typedef float4 V; typedef float4 W; static constexpr int G = 2; };
template <> struct LineT<float> { typedef float R; typedef float2 V; typedef float2 W; static constexpr int G = 1; };
template <> struct LineT<double> { typedef double R; typedef double2 V; typedef double2 W; static constexpr int G = 1; };

template <typename T> struct LV { T re, im; };

__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 pset(float2, float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 pmulp(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfmap(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <typename T> __device__ __forceinline__ T padd(T a, T b) { return a + b; }
template <typename T> __device__ __forceinline__ T psub(T a, T b) { return a - b; }
template <typename T> __device__ __forceinline__ T pneg(T a) { return -a; }
template <typename T> __device__ __forceinline__ T pset(T, T s) { return s; }
// products that the compiler does not contract with a later sum, so that every kernel rounds
// alike
__device__ __forceinline__ float pmulp(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double pmulp(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float pfmap(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double pfmap(double a, double b, double c) { return fma(a, b, c); }

template <typename T> __device__ __forceinline__ LV<T> lzero() {
  typedef typename LineT<T>::R R;
  return {pset(T(), R(0)), pset(T(), R(0))};
}
template <typename T> __device__ __forceinline__ LV<T> ladd(LV<T> a, LV<T> b) { return {padd(a.re, b.re), padd(a.im, b.im)}; }
template <typename T> __device__ __forceinline__ LV<T> lsub(LV<T> a, LV<T> b) { return {psub(a.re, b.re), psub(a.im, b.im)}; }
// a + i b, a - i b
template <typename T> __device__ __forceinline__ LV<T> ladd_i(LV<T> a, LV<T> b) { return {psub(a.re, b.im), padd(a.im, b.re)}; }
template <typename T> __device__ __forceinline__ LV<T> lsub_i(LV<T> a, LV<T> b) { return {padd(a.re, b.im), psub(a.im, b.re)}; }
// a w and a conj(w), w broadcast to the lines of the vector
template <typename T> __device__ __forceinline__ LV<T> lmul(LV<T> a, T wr, T wi) {
  return {pfmap(a.re, wr, pneg(pmulp(a.im, wi))), pfmap(a.re, wi, pmulp(a.im, wr))};
}
template <typename T> __device__ __forceinline__ LV<T> lmulc(LV<T> a, T wr, T wi) {
  return {pfmap(a.re, wr, pmulp(a.im, wi)), pfmap(a.im, wr, pneg(pmulp(a.re, wi)))};
}

// loads and stores of vectors and of twiddles (W holds re and im for every line)
__device__ __forceinline__ LV<float2> vget(const float4 &v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 vput(const LV<float2> &a) { return make_float4(a.re.x, a.re.y, a.im.x, a.im.y); }
__device__ __forceinline__ LV<double> vget(const double2 &v) { return {v.x, v.y}; }
__device__ __forceinline__ double2 vput(const LV<double> &a) { return make_double2(a.re, a.im); }
__device__ __forceinline__ LV<float> vget(const float2 &v) { return {v.x, v.y}; }
__device__ __forceinline__ float2 vput(const LV<float> &a) { return make_float2(a.re, a.im); }
template <typename T> __device__ __forceinline__ typename LineT<T>::W wput(typename cplx_t<typename LineT<T>::R>::type w);
template <> __device__ __forceinline__ float4 wput<float2>(float2 w) { return make_float4(w.x, w.x, w.y, w.y); }
template <> __device__ __forceinline__ float2 wput<float>(float2 w) { return w; }
template <> __device__ __forceinline__ double2 wput<double>(double2 w) { return w; }

// A row of a spectral array holds, for every pair of neighbouring kx and every
// component, (re, re, im, im) in FP32, and (re, im) for every kx and component in FP64.
// Vector g of the tile row at `row`: FP32 pairs and FP64 are consecutive 16-byte vectors;
// a single FP32 line picks its two words out of the pair (row: the pair's first word
// plus the kx parity, g: component).
__device__ __forceinline__ LV<float2> gload(const float4 *row, int g, float2) { return vget(__ldg(row + g)); }
__device__ __forceinline__ LV<double> gload(const double2 *row, int g, double) { return vget(__ldg(row + g)); }
__device__ __forceinline__ LV<float> gload(const float2 *row, int g, float) {
  const float *p = reinterpret_cast<const float *>(row) + 4 * g;
  return {__ldg(p), __ldg(p + 2)};
}
__device__ __forceinline__ void gstore(float4 *row, int g, const LV<float2> &a) { row[g] = vput(a); }
__device__ __forceinline__ void gstore(double2 *row, int g, const LV<double> &a) { row[g] = vput(a); }
__device__ __forceinline__ void gstore(float2 *row, int g, const LV<float> &a) {
  float *p = reinterpret_cast<float *>(row) + 4 * g;
  p[0] = a.re;
  p[2] = a.im;
}

// ------------------------------------------------------------------ codelets
template <int R, bool INV, typename T> __device__ __forceinline__ void ldft(LV<T> *v);

// a exp(-+ 2 pi i m / N), m known after unrolling; quarter turns cost no product
template <int N, bool INV, typename T> __device__ __forceinline__ LV<T> lrot(LV<T> a, int m) {
  typedef typename LineT<T>::R R;
  if (m % N == 0) return a;
  if ((4 * m) % N == 0) {
    const int q = (4 * m / N) & 3;  // quarter turns
    if (q == 2) return {pneg(a.re), pneg(a.im)};
    if ((q == 1) != INV) return {a.im, pneg(a.re)};  // times -i
    return {pneg(a.im), a.re};                       // times +i
  }
  const T c = pset(T(), cs_c<R>(N, m)), s = pset(T(), cs_s<R>(N, m));
  return INV ? lmul<T>(a, c, s) : lmulc<T>(a, c, s);
}

// odd R: pairs (j, R - j) share cosine terms and antisymmetric sine terms
template <int R, bool INV, typename T> __device__ __forceinline__ void ldft_odd(LV<T> *v) {
  typedef typename LineT<T>::R S;
  constexpr int h = (R - 1) / 2;
  LV<T> s[h + 1], d[h + 1];
  const LV<T> x0 = v[0];
  LV<T> sum = x0;
#pragma unroll
  for (int j = 1; j <= h; j++) {
    s[j] = ladd(v[j], v[R - j]);
    d[j] = lsub(v[j], v[R - j]);
    sum = ladd(sum, s[j]);
  }
  v[0] = sum;
#pragma unroll
  for (int k = 1; k <= h; k++) {
    LV<T> a = x0, b;
#pragma unroll
    for (int j = 1; j <= h; j++) {
      const int m = (j * k) % R;
      const T c = pset(T(), cs_c<S>(R, m)), sn = pset(T(), cs_s<S>(R, m));
      a.re = pfmap(s[j].re, c, a.re);
      a.im = pfmap(s[j].im, c, a.im);
      b.re = j == 1 ? pmulp(d[j].re, sn) : pfmap(d[j].re, sn, b.re);
      b.im = j == 1 ? pmulp(d[j].im, sn) : pfmap(d[j].im, sn, b.im);
    }
    v[k] = INV ? ladd_i(a, b) : lsub_i(a, b);
    v[R - k] = INV ? lsub_i(a, b) : ladd_i(a, b);
  }
}

// N = R1 R2: j = R2 j1 + j2, k = k1 + R1 k2
template <int R1, int R2, bool INV, typename T> __device__ __forceinline__ void ldft_comp(LV<T> *v) {
  constexpr int N = R1 * R2;
  LV<T> y[N];
#pragma unroll
  for (int j2 = 0; j2 < R2; j2++) {
    LV<T> t[R1];
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) t[j1] = v[R2 * j1 + j2];
    ldft<R1, INV, T>(t);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) y[j2 * R1 + k1] = lrot<N, INV, T>(t[k1], (j2 * k1) % N);
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    LV<T> t[R2];
#pragma unroll
    for (int j2 = 0; j2 < R2; j2++) t[j2] = y[j2 * R1 + k1];
    ldft<R2, INV, T>(t);
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) v[k1 + R1 * k2] = t[k2];
  }
}

// N = R1 R2, R1 and R2 coprime: no twiddles (j = R2 j1 + R1 j2 mod N, k by remainders)
template <int R1, int R2, bool INV, typename T> __device__ __forceinline__ void ldft_pfa(LV<T> *v) {
  constexpr int N = R1 * R2;
  LV<T> y[N];
#pragma unroll
  for (int j2 = 0; j2 < R2; j2++) {
    LV<T> t[R1];
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) t[j1] = v[(R2 * j1 + R1 * j2) % N];
    ldft<R1, INV, T>(t);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) y[j2 * R1 + k1] = t[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    LV<T> t[R2];
#pragma unroll
    for (int j2 = 0; j2 < R2; j2++) t[j2] = y[j2 * R1 + k1];
    ldft<R2, INV, T>(t);
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) {
      int k = k1;
#pragma unroll
      for (int q = 0; q < R2; q++)
        if ((k1 + R1 * q) % R2 == k2) k = k1 + R1 * q;
      v[k] = t[k2];
    }
  }
}

template <int R, bool INV, typename T> __device__ __forceinline__ void ldft(LV<T> *v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const LV<T> a = v[0], b = v[1];
    v[0] = ladd(a, b);
    v[1] = lsub(a, b);
  } else if constexpr (R == 4) {
    const LV<T> t0 = ladd(v[0], v[2]), t1 = lsub(v[0], v[2]), t2 = ladd(v[1], v[3]), t3 = lsub(v[1], v[3]);
    v[0] = ladd(t0, t2);
    v[2] = lsub(t0, t2);
    v[1] = INV ? ladd_i(t1, t3) : lsub_i(t1, t3);
    v[3] = INV ? lsub_i(t1, t3) : ladd_i(t1, t3);
  } else if constexpr (R == 6) {
    ldft_pfa<2, 3, INV, T>(v);
  } else if constexpr (R == 8) {
    ldft_comp<4, 2, INV, T>(v);
  } else if constexpr (R == 9) {
    ldft_comp<3, 3, INV, T>(v);
  } else if constexpr (R == 10) {
    ldft_pfa<2, 5, INV, T>(v);
  } else if constexpr (R == 12) {
    ldft_pfa<4, 3, INV, T>(v);
  } else if constexpr (R == 16) {
    ldft_comp<4, 4, INV, T>(v);
  } else if constexpr (R == 18) {
    ldft_pfa<2, 9, INV, T>(v);
  } else if constexpr (R == 20) {
    ldft_pfa<4, 5, INV, T>(v);
  } else if constexpr (R == 22) {
    ldft_pfa<2, 11, INV, T>(v);
  } else if constexpr (R == 24) {
    ldft_pfa<8, 3, INV, T>(v);
  } else {
    ldft_odd<R, INV, T>(v);
  }
}

// ------------------------------------------------------------------ phases
// The outer ends of a transform: load(row, g) gives the input of line group g at `row`,
// store(row, g, v) takes the output.  LineIo: a tile's rows in global memory, `in` / `out`
// at row 0 with strides in vectors (single FP32 lines: pointer to the first word, stride
// in 8-byte units).
template <typename T> struct LineIo {
  const typename LineT<T>::V *in;
  typename LineT<T>::V *out;
  long long rs_in, rs_out;
  int rows_in, rows_out;  // rows beyond are zero / not wanted (unsplit plans)
  __device__ __forceinline__ LV<T> load(int row, int g) const { return gload(in + (long long)row * rs_in, g, T()); }
  __device__ __forceinline__ void store(int row, int g, const LV<T> &v) const {
    gstore(out + (long long)row * rs_out, g, v);
  }
};
// Dynamic shared memory by byte offset: accesses through the declared array are compiled
// as shared-memory accesses with 32-bit addresses.
template <typename E> __device__ __forceinline__ E *line_smem_at(unsigned off) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<E *>(smem_raw + off);
}
// offsets of a pass's tables and of the tile buffer
struct LineTabs {
  unsigned tw;     // w_n^q
  unsigned tws;    // w_{2n}^q, q < n (split plans)
  unsigned rbase;  // input row of butterfly r of phase 0 at digit 0
  unsigned buf;
};

// A plan as the phases see it: the run-time plan with its LG vectors a position ...
struct RtPlan {
  static constexpr bool RT = true;
  const LinePlan &pl;
  int lg;
  FastDiv dlg;
  __device__ __forceinline__ int n() const { return pl.n; }
  __device__ __forceinline__ bool split() const { return pl.split != 0; }
  __device__ __forceinline__ int str(int p) const { return pl.str[p]; }
  __device__ __forceinline__ int tmul(int p) const { return pl.tmul[p]; }
  __device__ __forceinline__ int rstep() const { return pl.rstep; }
  __device__ __forceinline__ int LG() const { return lg; }
  __device__ __forceinline__ unsigned divLG(unsigned u) const { return fdiv(u, dlg); }
  __device__ __forceinline__ unsigned divstr(int p, unsigned u) const { return fdiv(u, pl.dstr[p]); }
  __device__ __forceinline__ unsigned divtin(int p, unsigned u) const { return fdiv(u, pl.dtin[p]); }
};
// ... and one known to the compiler: N points of digits R0 R1 R2, LGV vectors a position.
// Index arithmetic becomes constants and the phases unroll; the arithmetic is the same.
__host__ __device__ constexpr int ct_gcd(int a, int b) { return b ? ct_gcd(b, a % b) : a; }
template <int N_, int SPLIT_, int LGV, int R0, int R1 = 1, int R2 = 1> struct CtPlan {
  static constexpr bool RT = false;
  static constexpr int N = N_, SPLIT = SPLIT_, NP = R2 > 1 ? 3 : R1 > 1 ? 2 : 1;
  static_assert(R0 * R1 * R2 == N_, "the radices multiply to the length");
  __host__ __device__ static constexpr int rad(int p) { return p == 0 ? R0 : p == 1 ? R1 : R2; }
  __host__ __device__ static constexpr int str(int p) { return p == 0 ? R1 * R2 : p == 1 ? R2 : 1; }
  __host__ __device__ static constexpr bool share(int i, int j) { return ct_gcd(rad(i), rad(j)) > 1; }
  // group of a digit (lineplan_from's rule)
  __host__ __device__ static constexpr int grp(int p) {
    return p == 0 ? 0 : p == 1 ? (share(0, 1) || share(0, 2) ? 0 : 1) : (share(1, 2) || share(0, 2) ? grp(1) : grp(1) + 1);
  }
  __host__ __device__ static constexpr int inner(int p) {  // later digits of the same group
    int v = 1;
    for (int q = p + 1; q < NP; q++) v *= grp(q) == grp(p) ? rad(q) : 1;
    return v;
  }
  __host__ __device__ static constexpr int tin(int p) { return str(p) / inner(p); }
  __host__ __device__ static constexpr int tmul(int p) { return inner(p) > 1 ? N / (rad(p) * inner(p)) : 0; }
  __host__ __device__ static constexpr bool twiddles() { return tmul(0) || (NP > 1 && tmul(1)) || (NP > 2 && tmul(2)); }
  __host__ __device__ static constexpr int rstep() {
    return N / (rad(0) * inner(0)) * inner(0) % N;
  }
  __host__ __device__ static constexpr int n() { return N; }
  __host__ __device__ static constexpr bool split() { return SPLIT != 0; }
  __host__ __device__ static constexpr int LG() { return LGV; }
  __device__ static constexpr unsigned divLG(unsigned u) { return u / (unsigned)LGV; }
  __device__ static constexpr unsigned divstr(int p, unsigned u) { return u / (unsigned)str(p); }
  __device__ static constexpr unsigned divtin(int p, unsigned u) { return u / (unsigned)tin(p); }
  // the run-time plan is this one
  __host__ static bool is(const LinePlan &pl) {
    if (pl.bl || pl.n != N || pl.split != SPLIT || pl.np != NP || pl.rstep != rstep()) return false;
    for (int p = 0; p < NP; p++)
      if (pl.rad[p] != rad(p) || pl.str[p] != str(p) || pl.tmul[p] != tmul(p) || pl.tin[p] != tin(p)) return false;
    return true;
  }
};

template <int RAD, bool INV, typename T>
__device__ __forceinline__ void ltwiddle(LV<T> *a, unsigned tw, int tb) {
#pragma unroll
  for (int k = 1; k < RAD; k++) {
    const LV<T> w = vget(line_smem_at<typename LineT<T>::W>(tw)[tb * k]);
    a[k] = INV ? lmulc<T>(a[k], w.re, w.im) : lmul<T>(a[k], w.re, w.im);
  }
}

// One phase over the tile's LG line groups.  glob: the outer end of the transform (the
// input of forward phase 0, the output of inverse phase 0) is `io`; gin: an inverse
// phase that reads the spectrum, by position, from `io`; gout: a forward phase that
// writes it there.
template <int RAD, bool INV, typename T, typename IO, typename PL>
__device__ __forceinline__ void lphase(const PL &pl, int p, const LineTabs &tb, const IO &io, bool glob, bool gin,
                                       bool gout) {
  typedef typename LineT<T>::V V;
  typedef typename LineT<T>::W W;
  const int s = pl.str(p), n = pl.n(), tm = pl.tmul(p), LG = pl.LG();
  const int sv = s * LG;
  V *const buf = line_smem_at<V>(tb.buf);
  constexpr bool SPLIT0 = split_radix(RAD);
  if (SPLIT0 && p == 0 && glob && pl.split()) {
    // both halves of a butterfly in one thread: its rows are read (written) once
    if constexpr (SPLIT0) {
      const unsigned total = (unsigned)s * (unsigned)LG;
#pragma unroll 1
      for (unsigned u = threadIdx.x; u < total; u += blockDim.x) {
        const unsigned r = pl.divLG(u);
        const int g = (int)(u - r * (unsigned)LG);
        const int ti = tm ? tm * (int)pl.divtin(0, r) : 0;
        const int row0 = line_smem_at<int>(tb.rbase)[r];
        const W *tws = line_smem_at<W>(tb.tws);
        LV<T> x[RAD];
        if constexpr (!INV) {
          int row = row0;
#pragma unroll
          for (int j = 0; j < RAD; j++) {
            x[j] = io.load(row, g);
            row += pl.rstep();
            if (row >= n) row -= n;
          }
#pragma unroll
          for (int h = 0; h < 2; h++) {
            LV<T> a[RAD];
            row = row0;
#pragma unroll
            for (int j = 0; j < RAD; j++) {
              a[j] = x[j];
              if (h) {
                const LV<T> w = vget(tws[row]);
                a[j] = lmul<T>(x[j], w.re, w.im);
                row += pl.rstep();
                if (row >= n) row -= n;
              }
            }
            ldft<RAD, false, T>(a);
            if (tm) ltwiddle<RAD, false, T>(a, tb.tw, ti);
            if (gout) {
#pragma unroll
              for (int k = 0; k < RAD; k++) io.store(h * n + (int)r + k * s, g, a[k]);
            } else {
              V *dst = buf + (h * n + (int)r) * LG + g;
#pragma unroll
              for (int k = 0; k < RAD; k++) dst[k * sv] = vput(a[k]);
            }
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            LV<T> a[RAD];
            if (gin) {
#pragma unroll
              for (int k = 0; k < RAD; k++) a[k] = io.load(h * n + (int)r + k * s, g);
            } else {
              const V *src = buf + (h * n + (int)r) * LG + g;
#pragma unroll
              for (int k = 0; k < RAD; k++) a[k] = vget(src[k * sv]);
            }
            if (tm) ltwiddle<RAD, true, T>(a, tb.tw, ti);
            ldft<RAD, true, T>(a);
            if (h == 0) {
#pragma unroll
              for (int j = 0; j < RAD; j++) x[j] = a[j];
            } else {
              int row = row0;
#pragma unroll
              for (int j = 0; j < RAD; j++) {
                const LV<T> w = vget(tws[row]);
                const LV<T> o = lmulc<T>(a[j], w.re, w.im);
                io.store(row, g, ladd(x[j], o));
                row += pl.rstep();
                if (row >= n) row -= n;
              }
            }
          }
        }
      }
    }
    return;
  }
  const unsigned total = (unsigned)((pl.split() ? 2 * n : n) / RAD) * (unsigned)LG;
#pragma unroll 1
  for (unsigned u = threadIdx.x; u < total; u += blockDim.x) {
    const unsigned b = pl.divLG(u);
    const int g = (int)(u - b * (unsigned)LG);
    const unsigned beta = pl.divstr(p, b);
    const int r = (int)(b - beta * (unsigned)s);
    const int pos0 = (int)beta * (s * RAD) + r;
    const int ti = tm ? tm * (int)pl.divtin(p, (unsigned)r) : 0;
    LV<T> a[RAD];
    const bool outer = p == 0 && glob;  // unsplit plan, rows through the row map
    if (!INV && outer) {
      int row = line_smem_at<int>(tb.rbase)[r];
#pragma unroll
      for (int j = 0; j < RAD; j++) {
        a[j] = lzero<T>();
        if (row < io.rows_in) a[j] = io.load(row, g);
        row += pl.rstep();
        if (row >= n) row -= n;
      }
    } else if (INV && gin) {
#pragma unroll
      for (int j = 0; j < RAD; j++) a[j] = io.load(pos0 + j * s, g);
    } else {
      const V *src = buf + pos0 * LG + g;
#pragma unroll
      for (int j = 0; j < RAD; j++) a[j] = vget(src[j * sv]);
    }
    if (INV && tm) ltwiddle<RAD, true, T>(a, tb.tw, ti);
    ldft<RAD, INV, T>(a);
    if (!INV && tm) ltwiddle<RAD, false, T>(a, tb.tw, ti);
    if (INV && outer) {
      int row = line_smem_at<int>(tb.rbase)[r];
#pragma unroll
      for (int j = 0; j < RAD; j++) {
        if (row < io.rows_out) io.store(row, g, a[j]);
        row += pl.rstep();
        if (row >= n) row -= n;
      }
    } else if (!INV && gout) {
#pragma unroll
      for (int k = 0; k < RAD; k++) io.store(pos0 + k * s, g, a[k]);
    } else {
      V *dst = buf + pos0 * LG + g;
#pragma unroll
      for (int k = 0; k < RAD; k++) dst[k * sv] = vput(a[k]);
    }
  }
}

// WIDE: the radices above 17 too (FP32 schedules of the y and z passes)
template <bool INV, bool WIDE, typename T, typename IO>
__device__ __forceinline__ void lphase_any(const RtPlan &rp, int p, const LineTabs &tb, const IO &io, bool glob,
                                           bool gin, bool gout) {
  const LinePlan &pl = rp.pl;
#define PMGPU_LP(r) case r: lphase<r, INV, T, IO, RtPlan>(rp, p, tb, io, glob, gin, gout); break;
  switch (pl.rad[p]) {
    PMGPU_LP(1) PMGPU_LP(2) PMGPU_LP(3) PMGPU_LP(4) PMGPU_LP(5) PMGPU_LP(6) PMGPU_LP(7) PMGPU_LP(8) PMGPU_LP(9)
    PMGPU_LP(10) PMGPU_LP(11) PMGPU_LP(12) PMGPU_LP(13) PMGPU_LP(16) PMGPU_LP(17)
    default:
      if constexpr (WIDE && sizeof(typename LineT<T>::R) == 4) {
        switch (pl.rad[p]) {
          PMGPU_LP(18) PMGPU_LP(20) PMGPU_LP(22) PMGPU_LP(24)
          default: break;  // plans only hold register radices
        }
      }
      break;
  }
#undef PMGPU_LP
}

// ------------------------------------------------------------------ Bluestein
// Transform of lines of length bn as a circular convolution of length n (one group of
// digits, so positions and rows coincide):
//   X[k] = c[k] sum_j (x[j] c[j]) conj(c[k - j]),   c[j] = exp(-i pi j^2 / bn):
// forward transform of the chirped input (zero beyond the rows), product with
// B = FFT_n(conj c wrapped) at the plan's positions, inverse transform, chirp / n.  The
// inverse DFT is conj(forward(conj x)).  A forward transform has r <= bn data rows and bn
// outputs, an inverse one bn inputs and r wanted rows: k - j takes bn + r - 1 values, from
// 1 - r and from 1 - bn on, so that a free axis (r = bn / 2) needs n >= 1.5 bn - 1 and the
// two directions have a table B each.
template <typename T, typename IO>
__device__ __forceinline__ void lchirp_in(unsigned boff, int n, int LG, const FastDiv &dLG, unsigned coff, int nin, bool conj_in, bool gsrc, const IO &io) {
  typename LineT<T>::V *const buf = line_smem_at<typename LineT<T>::V>(boff);
  const typename cplx_t<typename LineT<T>::R>::type *chirp =
      line_smem_at<typename cplx_t<typename LineT<T>::R>::type>(coff);
  // four values a thread at a time, so that their loads are in flight together
  constexpr int U = 4;
  const unsigned total = (unsigned)n * (unsigned)LG;
  for (unsigned t0 = threadIdx.x; t0 < total; t0 += U * blockDim.x) {
    LV<T> v[U];
    unsigned j[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned t = t0 + u * blockDim.x;
      j[u] = fdiv(t, dLG);
      v[u] = lzero<T>();
      if (t < total && (int)j[u] < nin) v[u] = gsrc ? io.load((int)j[u], (int)(t - j[u] * (unsigned)LG)) : vget(buf[t]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned t = t0 + u * blockDim.x;
      if (t >= total) break;
      if ((int)j[u] < nin) {
        if (conj_in) v[u].im = pneg(v[u].im);
        const auto c = chirp[j[u]];
        v[u] = lmul<T>(v[u], pset(T(), c.x), pset(T(), c.y));
      }
      buf[t] = vput(v[u]);
    }
  }
}
template <typename T>
__device__ __forceinline__ void lchirp_mul(unsigned boff, int n, int LG, const FastDiv &dLG,
                                           const typename cplx_t<typename LineT<T>::R>::type *bpos) {
  typename LineT<T>::V *const buf = line_smem_at<typename LineT<T>::V>(boff);
  const unsigned total = (unsigned)n * (unsigned)LG;
  for (unsigned t = threadIdx.x; t < total; t += blockDim.x) {
    const auto c = bpos[fdiv(t, dLG)];
    buf[t] = vput(lmul<T>(vget(buf[t]), pset(T(), c.x), pset(T(), c.y)));
  }
}
template <typename T, typename IO>
__device__ __forceinline__ void lchirp_out(unsigned boff, int n, int LG, const FastDiv &dLG, unsigned coff, int nout,
                                           bool conj_out, bool gdst, const IO &io) {
  typename LineT<T>::V *const buf = line_smem_at<typename LineT<T>::V>(boff);
  const typename cplx_t<typename LineT<T>::R>::type *chirp =
      line_smem_at<typename cplx_t<typename LineT<T>::R>::type>(coff);
  typedef typename LineT<T>::R R;
  const T sc = pset(T(), R(1) / R(n));
  const unsigned total = (unsigned)nout * (unsigned)LG;
  for (unsigned t = threadIdx.x; t < total; t += blockDim.x) {
    const unsigned k = fdiv(t, dLG);
    const int g = (int)(t - k * (unsigned)LG);
    const auto c = chirp[k];
    LV<T> v = lmul<T>(vget(buf[t]), pset(T(), c.x), pset(T(), c.y));
    v.re = pmulp(v.re, sc);
    v.im = pmulp(v.im, sc);
    if (conj_out) v.im = pneg(v.im);
    if (gdst) io.store((int)k, g, v);
    else buf[t] = vput(v);
  }
}

}  // namespace pmgpu
