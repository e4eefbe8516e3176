// solve.cuh -- the unbounded FFT Poisson solve as five HBM passes.
//
// The reference (source/poisson/pmlib_poisson_solve.f) transforms the complex copy
// of the cuboid vorticity along fft_seq(1) and fft_seq(2), runs the third-axis lines
// (zero-pad, FFT, multiply by the Green's function, spectral curl, iFFT, truncate),
// transforms back and keeps REAL().  The 3-D DFT is separable, so the result does
// not depend on the axis order; here the passes always run x, y, z:
//
//   x_fwd : real cuboid -> X, kx < H = Mx/2+1                 (R2C, zero-pad fused)
//   y_fwd : X -> Y, ky < My                                     (C2C, zero-pad fused)
// (X is stored [z][kx block][y][kx in block][c], Y the same with the ky rows, in blocks of
// spec_block kx; the kx extent is padded to Hp, a multiple of 8)
//   z_pass: Y -> Y (or another buffer): pad, FFT, multiply+curl, iFFT, truncate
//   y_inv : Y -> X (truncate to the pencil extent)
//   x_inv : X -> real cuboid                                     (C2R, truncate fused)
//
// REAL() of the reference's complex inverse equals the C2R inverse of the Hermitian
// part of the spectrum.  The curl's Nyquist wavenumber (-M/(2L), source
// pmlib_poisson_solve.f:268-306) makes i k x w non-Hermitian on the Nyquist planes;
// its Hermitian part is the curl with the Nyquist components of k set to zero, which
// is what z_pass applies (the filter zeta uses |k|^2 and keeps them).
#pragma once

#include "common.cuh"
#include "fft.cuh"
#include "linefft.cuh"

namespace pmgpu {

template <typename R> struct SolveGeom {
  typedef typename cplx_t<R>::type C;
  int ext[3];      // cuboid extents including ghosts (x, y, z)
  int off[3];      // first pencil point inside the cuboid (0 free, nghost periodic)
  int P[3];        // pencil extents (free: N + 2 nghost, periodic: N)
  int M[3];        // FFT lengths (free: 2 P, periodic: P)
  int H;           // Mx / 2 + 1
  int Hp;          // H padded to a multiple of 8 (16-byte aligned tile rows)
  int N2;          // Mx / 2
  FftDesc fx, fy, fz;
  const C *twx, *twy, *twz;
  const R *kxt, *kyt, *kzt;  // wavenumbers (cycles / length), Nyquist index included
  const R *green;            // real octant G(kx, |ky|, |kz|) * dx dy dz / (Mx My Mz), rows of Hp
  int gM1, gM2;              // My / 2 + 1, Mz / 2 + 1
  int kernel2;               // derivative kernel (3 components); green holds its spectrum
  R scale;                   // 1 / (Mx My Mz)
  R eps2pi;                  // 2 pi epsilon (filter argument scale)
  int order;                 // filter order (poisson order or reg_order)
  int allper;                // all axes periodic: spectral Green's function
  // in-place register FFTs (when the lengths factor into register radices, or Bluestein)
  int rx_ok, ry_ok, rz_ok;
  LinePlan lx;               // the half-length complex transform of the x passes
  LinePlan ly, lz;
  const C *rtwx, *rtwy, *rtwz;  // w_n^q, q < n
  const C *rtsx, *rtsy, *rtsz;      // split plans: w_{2n}^q, q < n
  const int *rbx0, *rby0, *rbz0;    // input row of every butterfly of phase 0 at digit 0
  const C *rextx;            // exp(-2 pi i k / Mx), k < H
  const int *xpos;           // frequency -> position of the x transform
  int tky, tkz;              // kx tile of the y / z register passes (0: chosen by shared memory)
  const C *rchx, *rchy, *rchz;  // Bluestein plans: chirp exp(-i pi j^2 / n), j < n
  const C *rbx, *rby, *rbz;     // Bluestein plans: FFT of the wrapped chirp, by position
  const int *yk;             // row of the y spectrum -> ky index (nullptr: natural order)
  const int *zk;             // position of the z transform -> kz index
  // the plain velocity solve's multiplier tables: 2 pi kx (Nyquist component zero, zero
  // from H on, Hp entries), and by z position 2 pi kz (Nyquist component zero) and the
  // offset of the octant plane |kz|
  const R *kxv, *kzv;
  const int *zoff;
};

enum ZMode { Z_VEL = 0, Z_VORT = 1, Z_VECPOT = 2, Z_REGULARISE = 3, Z_FORWARD = 4 };

// zeta(s) = (1 + s^2/2 + s^4/8 + s^6/48 + s^8/384 ...) exp(-s^2/2), truncated by order
// (source/poisson/pmlib_poisson_solve.f:309-334, source/regularise/pmlib_regularise.f:255-282)
template <typename R> __device__ __forceinline__ R zeta_filter(int order, R s) {
  const R s2 = s * s;
  const R e = exp(R(-0.5) * s2);
  R p = R(1);
  if (order >= 4) p += R(0.5) * s2;
  if (order >= 6) p += R(0.125) * s2 * s2;
  if (order >= 8) p += (R(1) / R(48)) * s2 * s2 * s2;
  if (order >= 10) p += (R(1) / R(384)) * s2 * s2 * s2 * s2;
  return order == 0 ? R(1) : p * e;
}

// ---------------------------------------------------------------- common tile machinery
// All passes are persistent: a CTA loops over tiles, and while it transforms tile i
// the rows of tile i+1 stream into a staging buffer with cp.async.  Buffers: S
// (staging), A and B (ping-pong); the first pass reads S, later passes alternate A/B.
constexpr int PASS_THREADS = 512;

template <bool INV, typename R>
__device__ __forceinline__ void vpass_any(const typename Vec<R>::V *src, typename Vec<R>::V *dst, int LG,
                                          const FftDesc &d, int p, const typename cplx_t<R>::type *tw,
                                          const LineMap &lm) {
  const typename cplx_t<R>::type *t = tw + d.twoff[p];
  const int ns = d.ns[p], n = d.n;
  switch (d.rad[p]) {
    case 2: vpass<2, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 3: vpass<3, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 4: vpass<4, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 5: vpass<5, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 7: vpass<7, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 8: vpass<8, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 11: vpass<11, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 13: vpass<13, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 16: vpass<16, INV, R>(src, dst, LG, n, ns, t, lm); break;
    case 17: vpass<17, INV, R>(src, dst, LG, n, ns, t, lm); break;
    default: vpass_generic<INV, R>(src, dst, LG, n, ns, d.rad[p], t, tw + d.rootoff[p], lm); break;
  }
}

// A transform that reads `first` (S or A) and ping-pongs between A and B; `hook`
// runs once after the first pass has finished reading `first` (the prefetch point).
template <bool INV, typename R, typename Hook>
__device__ __forceinline__ typename Vec<R>::V *vfft_chain(typename Vec<R>::V *first, typename Vec<R>::V *A,
                                                          typename Vec<R>::V *B, int LG, const FftDesc &d,
                                                          const typename cplx_t<R>::type *tw, const LineMap &lm,
                                                          Hook hook) {
  typedef typename Vec<R>::V V;
  V *src = first, *dst = (first == A) ? B : A;
  for (int p = 0; p < d.npass; p++) {
    vpass_any<INV, R>(src, dst, LG, d, p, tw, lm);
    __syncthreads();
    if (p == 0) hook();
    V *nsrc = dst;
    V *ndst = (dst == A) ? B : A;
    src = nsrc;
    dst = ndst;
  }
  if (d.npass == 0) hook();
  return src;
}

struct NoHook {
  __device__ void operator()() const {}
};

// ---------------------------------------------------------------- y and z passes
// Tile t = (outer o, kx-tile kt): L = NC * TK lines of n points.  Row r of the tile
// starts at complex offset (spec_off(o * os, kb, kt * TK) + r * rs) * NC and holds L complex.
struct LineTiles {
  int n;          // transform length
  int rows_in;    // rows read (the rest is zero padding)
  int rows_out;   // rows written (truncation)
  long long in_os, in_rs, out_os, out_rs;
  long long in_kb, out_kb;  // strides between kx blocks
  int nouter, nkt, TK;
  int ofast;      // consecutive tiles: outer index fastest (z pass) or kx tile fastest
  // even input of n rows (the Green's function): rows beyond n / 2 are read from their
  // mirror, and z tiles of the mirrored half of ky are left out
  int even;
  FastDiv dLG;    // division by the line vectors per row (register engine)
};
// kx of a block of the spectral arrays: 192 bytes of three components
template <typename R> __host__ __device__ constexpr int spec_block() { return sizeof(R) == 4 ? 8 : 4; }
// tile -> (outer index, first kx)
__device__ __forceinline__ void line_tile_at(const LineTiles &lt, int tile, int TK, int &o, int &k0) {
  if (lt.ofast) {
    const int kt = tile / lt.nouter;
    o = tile - kt * lt.nouter;
    k0 = kt * TK;
  } else {
    o = tile / lt.nkt;
    k0 = (tile - o * lt.nkt) * TK;
  }
}
// complex offset (to be multiplied by the components) of kx index k0 in a row whose
// blocks lie kb apart
template <typename R> __device__ __forceinline__ long long spec_off(long long row, long long kb, int k0) {
  constexpr int B = spec_block<R>();
  return row + (long long)(k0 / B) * kb + (k0 & (B - 1));
}

enum LMode { L_FWD = 0, L_INV = 1, L_Z = 2 };

template <typename R>
__device__ __forceinline__ void tile_rows_load(typename cplx_t<R>::type *S, const typename cplx_t<R>::type *in,
                                               long long base, long long rs, int nrows, int L, int NC) {
  // 16-byte chunks; rows are 16-byte aligned (kx padded to a multiple of 8)
  const int cpr = (L * (int)sizeof(typename cplx_t<R>::type)) / 16;
  const int rsub = threadIdx.x / cpr, c = threadIdx.x - rsub * cpr;
  const int RS = blockDim.x / cpr;
  if (rsub >= RS) return;
  const char *src = reinterpret_cast<const char *>(in + base * NC);
  char *dst = reinterpret_cast<char *>(S);
  const size_t rowb = (size_t)L * sizeof(typename cplx_t<R>::type);
  const size_t strideb = (size_t)rs * NC * sizeof(typename cplx_t<R>::type);
  for (int r = rsub; r < nrows; r += RS) cp_async16(dst + r * rowb + c * 16, src + r * strideb + c * 16);
}

template <typename R>
__device__ __forceinline__ void tile_rows_store(typename cplx_t<R>::type *out, const typename cplx_t<R>::type *Rb,
                                                long long base, long long rs, int nrows, int L, int NC) {
  const int cpr = (L * (int)sizeof(typename cplx_t<R>::type)) / 16;
  const int rsub = threadIdx.x / cpr, c = threadIdx.x - rsub * cpr;
  const int RS = blockDim.x / cpr;
  if (rsub >= RS) return;
  char *dst = reinterpret_cast<char *>(out + base * NC);
  const char *src = reinterpret_cast<const char *>(Rb);
  const size_t rowb = (size_t)L * sizeof(typename cplx_t<R>::type);
  const size_t strideb = (size_t)rs * NC * sizeof(typename cplx_t<R>::type);
  for (int r = rsub; r < nrows; r += RS)
    *reinterpret_cast<float4 *>(dst + r * strideb + c * 16) = *reinterpret_cast<const float4 *>(src + r * rowb + c * 16);
}

// the spectral multiply at one point (kx index kx_i, row y of the y spectrum, kz
// index z): the NC values v of the point in place.  kxp: kx wavenumber, Gp: the
// Green's function value (loaded by the caller for the plain velocity solve)
template <typename R, int NC>
__device__ __forceinline__ void z_point(const SolveGeom<R> &g, typename cplx_t<R>::type *v, int kx_i, R kxp, R Gp,
                                        R ky, R kyc, int y, int iy, int z, R kz, int zmode, int reproj,
                                        int use_zeta) {
  typedef typename cplx_t<R>::type C;
  const R twopi = R(6.283185307179586476925286766559);
  if (kx_i >= g.H) {
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = mk(R(0), R(0));
    return;
  }
  const R kx = kxp;
  const R kxc = (2 * kx_i == g.M[0]) ? R(0) : kx;
  const R kzc = (2 * z == g.M[2]) ? R(0) : kz;
  const R kmag = kx * kx + ky * ky + kz * kz;
  if (zmode == Z_REGULARISE) {
    const R zt = zeta_filter<R>(g.order, g.eps2pi * sqrt(kmag)) * g.scale;
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = cscale(v[c], zt);
    return;
  }
  if constexpr (NC == 3) {
    R zt = R(1);
    if (use_zeta) zt = zeta_filter<R>(g.order, g.eps2pi * sqrt(kmag));
    if (g.kernel2 && !g.allper) {
      // derivative kernel K (pmlib_poisson_solve.f, kernel 2): component c is
      // i S_c + (-1)^(k_c) E_c, S_c odd along axis c and even along the others
      // (stored for |ky|, |kz| with the sign of the odd axis applied here), E_c the
      // spectrum of the kernel's plane at -M_c/2 dx_c
      const size_t noct = (size_t)g.gM2 * g.gM1 * g.Hp;
      const int iz = min(z, g.M[2] - z);
      const size_t oc = ((size_t)iz * g.gM1 + iy) * g.Hp + kx_i;
      const R *E = g.green + 3 * noct;
      R sx = g.green[oc], sy = g.green[noct + oc], sz = g.green[2 * noct + oc];
      if (2 * y > g.M[1]) sy = -sy;
      if (2 * z > g.M[2]) sz = -sz;
      R ex = E[(size_t)iz * g.gM1 + iy];
      R ey = E[(size_t)g.gM2 * g.gM1 + (size_t)iz * g.H + kx_i];
      R ez = E[(size_t)g.gM2 * (g.gM1 + g.H) + (size_t)iy * g.H + kx_i];
      if (kx_i & 1) ex = -ex;
      if (y & 1) ey = -ey;
      if (z & 1) ez = -ez;
      const C Kx = mk(ex, sx), Ky = mk(ey, sy), Kz = mk(ez, sz);
      const C w1 = v[0], w2 = v[1], w3 = v[2];
      if (zmode == Z_VEL) {
        v[0] = csub(cmul(Ky, w3), cmul(Kz, w2));
        v[1] = csub(cmul(Kz, w1), cmul(Kx, w3));
        v[2] = csub(cmul(Kx, w2), cmul(Ky, w1));
      } else {  // Z_VORT: zeta w (+ K 2 pi i (k . w), Nyquist components dropped)
        C o1 = cscale(w1, zt * g.scale), o2 = cscale(w2, zt * g.scale), o3 = cscale(w3, zt * g.scale);
        if (reproj) {
          const C da = cadd(cadd(cscale(w1, kxc), cscale(w2, kyc)), cscale(w3, kzc));
          const C dv = mk(-twopi * da.y, twopi * da.x);
          o1 = cadd(o1, cmul(Kx, dv));
          o2 = cadd(o2, cmul(Ky, dv));
          o3 = cadd(o3, cmul(Kz, dv));
        }
        v[0] = o1;
        v[1] = o2;
        v[2] = o3;
      }
      return;
    }
    R G;
    if (g.allper) {
      G = (kmag > R(0)) ? zt / (twopi * twopi * kmag) * g.scale : R(0);
    } else {
      G = Gp;
    }
    const C w1 = v[0], w2 = v[1], w3 = v[2];
    if (zmode == Z_VEL) {
      const C c1 = csub(cscale(w3, kyc), cscale(w2, kzc));
      const C c2 = csub(cscale(w1, kzc), cscale(w3, kxc));
      const C c3 = csub(cscale(w2, kxc), cscale(w1, kyc));
      const R f = G * twopi;
      v[0] = mk(-f * c1.y, f * c1.x);
      v[1] = mk(-f * c2.y, f * c2.x);
      v[2] = mk(-f * c3.y, f * c3.x);
    } else if (zmode == Z_VECPOT) {
      v[0] = cscale(w1, G);
      v[1] = cscale(w2, G);
      v[2] = cscale(w3, G);
    } else {  // Z_VORT: zeta w (+ reprojection -4 pi^2 G k (k . w), Hermitian part)
      C o1 = cscale(w1, zt * g.scale), o2 = cscale(w2, zt * g.scale), o3 = cscale(w3, zt * g.scale);
      if (reproj) {
        const R nx = kx - kxc, ny = ky - kyc, nz = kz - kzc;
        const C da = cadd(cadd(cscale(w1, kxc), cscale(w2, kyc)), cscale(w3, kzc));
        const C dn = cadd(cadd(cscale(w1, nx), cscale(w2, ny)), cscale(w3, nz));
        const R f = -twopi * twopi * G;
        o1 = cadd(o1, cscale(cadd(cscale(da, kxc), cscale(dn, nx)), f));
        o2 = cadd(o2, cscale(cadd(cscale(da, kyc), cscale(dn, ny)), f));
        o3 = cadd(o3, cscale(cadd(cscale(da, kzc), cscale(dn, nz)), f));
      }
      v[0] = o1;
      v[1] = o2;
      v[2] = o3;
    }
  }
}

// One complex value of a line vector, and back.
__device__ __forceinline__ float2 lane_get(const LV<float2> &a, int h) {
  return h ? make_float2(a.re.y, a.im.y) : make_float2(a.re.x, a.im.x);
}
__device__ __forceinline__ void lane_set(LV<float2> &a, int h, float2 v) {
  if (h) { a.re.y = v.x; a.im.y = v.y; }
  else { a.re.x = v.x; a.im.x = v.y; }
}
__device__ __forceinline__ float2 lane_get(const LV<float> &a, int) { return make_float2(a.re, a.im); }
__device__ __forceinline__ void lane_set(LV<float> &a, int, float2 v) { a.re = v.x; a.im = v.y; }
__device__ __forceinline__ double2 lane_get(const LV<double> &a, int) { return make_double2(a.re, a.im); }
__device__ __forceinline__ void lane_set(LV<double> &a, int, double2 v) { a.re = v.x; a.im = v.y; }

// The spectral multiply (any mode) of a tile of LG vectors per position: TK kx of NC
// components from kx index k0, spectrum row y.  zpos: position -> kz index (nullptr:
// natural order)
template <typename T, int NC>
__device__ __forceinline__ void z_multiply(const SolveGeom<typename LineT<T>::R> &g, typename LineT<T>::V *buf, int LG,
                                           int k0, int y, int zmode, int reproj, int use_zeta, const int *zpos) {
  typedef typename LineT<T>::R R;
  constexpr int G = LineT<T>::G;
  const int N = g.M[2], nk = LG / NC;
  const R ky = g.kyt[y];
  const R kyc = (2 * y == g.M[1]) ? R(0) : ky;  // Nyquist component dropped in the curl
  const int iy = min(y, g.M[1] - y);
  const bool pre = NC == 3 && zmode != Z_REGULARISE && !g.allper && !g.kernel2;
  const int nks = __ffs(nk) - 1;  // a power of two
  for (int t = threadIdx.x; t < N * nk; t += blockDim.x) {
    const int q = t >> nks, kk = t - (q << nks);
    const int z = zpos ? zpos[q] : q;
    typename LineT<T>::V *p = buf + (size_t)q * LG + kk * NC;
    LV<T> a[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) a[c] = vget(p[c]);
#pragma unroll
    for (int h = 0; h < G; h++) {
      const int kx_i = k0 + kk * G + h;
      const R kxp = kx_i < g.H ? g.kxt[kx_i] : R(0);
      const R Gp = pre ? g.green[((size_t)min(z, g.M[2] - z) * g.gM1 + iy) * g.Hp + kx_i] : R(0);
      typename cplx_t<R>::type v[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) v[c] = lane_get(a[c], h);
      z_point<R, NC>(g, v, kx_i, kxp, Gp, ky, kyc, y, iy, z, g.kzt[z], zmode, reproj, use_zeta);
#pragma unroll
      for (int c = 0; c < NC; c++) lane_set(a[c], h, v[c]);
    }
#pragma unroll
    for (int c = 0; c < NC; c++) p[c] = vput(a[c]);
  }
}

// The plain velocity solve's middle of the z pass in registers: a thread takes one block
// of RL consecutive positions of the three component lines of one kx group, runs the
// last forward phase (it has no twiddles), multiplies by i G (k x w) with 2 pi folded into
// k, runs the first inverse phase and writes the block back in place.  A block's vectors
// start RL * LG apart, so with an odd RL (and LG = 12, 6 or 3) the eight lanes of a
// quarter-warp fall in distinct banks; even RL share banks two to four times.
__device__ __forceinline__ float2 ld_lines(const float *p, float2) { return __ldg(reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ float ld_lines(const float *p, float) { return __ldg(p); }
__device__ __forceinline__ double ld_lines(const double *p, double) { return __ldg(p); }
template <int RL, typename T>
__device__ __forceinline__ void z_mid_vel(const SolveGeom<typename LineT<T>::R> &g, typename LineT<T>::V *buf, int LG,
                                          int k0, int y, int npts) {
  typedef typename LineT<T>::R R;
  constexpr int G = LineT<T>::G;
  const int nk = LG / 3, nks = __ffs(nk) - 1;
  const T ky = pset(T(), (2 * y == g.M[1]) ? R(0) : R(6.283185307179586476925286766559) * g.kyt[y]);
  const R *green = g.green + (size_t)min(y, g.M[1] - y) * g.Hp + k0;
  const int total = (npts / RL) << nks;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int beta = t >> nks, kk = t - (beta << nks);
    typename LineT<T>::V *p = buf + (size_t)(beta * RL) * LG + kk * 3;
    const T kx = ld_lines(g.kxv + k0 + kk * G, T());
    T Gv[RL];
    R kzs[RL];
#pragma unroll
    for (int k = 0; k < RL; k++) {
      Gv[k] = ld_lines(green + __ldg(g.zoff + beta * RL + k) + kk * G, T());
      kzs[k] = __ldg(g.kzv + beta * RL + k);
    }
    LV<T> a[3][RL];
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int j = 0; j < RL; j++) a[c][j] = vget(p[j * LG + c]);
      ldft<RL, false, T>(a[c]);
    }
#pragma unroll
    for (int k = 0; k < RL; k++) {
      const T kz = pset(T(), kzs[k]), f = Gv[k], fm = pneg(Gv[k]);
      const LV<T> w1 = a[0][k], w2 = a[1][k], w3 = a[2][k];
      const T c1r = pfmap(w3.re, ky, pneg(pmulp(w2.re, kz))), c1i = pfmap(w3.im, ky, pneg(pmulp(w2.im, kz)));
      const T c2r = pfmap(w1.re, kz, pneg(pmulp(w3.re, kx))), c2i = pfmap(w1.im, kz, pneg(pmulp(w3.im, kx)));
      const T c3r = pfmap(w2.re, kx, pneg(pmulp(w1.re, ky))), c3i = pfmap(w2.im, kx, pneg(pmulp(w1.im, ky)));
      a[0][k] = {pmulp(fm, c1i), pmulp(f, c1r)};
      a[1][k] = {pmulp(fm, c2i), pmulp(f, c2r)};
      a[2][k] = {pmulp(fm, c3i), pmulp(f, c3r)};
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      ldft<RL, true, T>(a[c]);
#pragma unroll
      for (int j = 0; j < RL; j++) p[j * LG + c] = vput(a[c][j]);
    }
  }
}
// the velocity multiplier is G(k) times the curl: kernel 1, or all axes periodic (either
// kernel) unless the filter goes with it
template <typename R> __host__ __device__ inline bool z_plain(const SolveGeom<R> &g, int use_zeta) {
  return g.allper ? !use_zeta : !g.kernel2;
}
// radices of a last phase that z_mid_vel takes
__host__ __device__ constexpr bool z_mid_radix(int r) { return r >= 2 && r <= 6; }
// block of the multiply of a plan whose last radix is r
__host__ __device__ constexpr int z_mid_block(int r) { return z_mid_radix(r) ? r : 1; }
template <typename T>
__device__ __forceinline__ void z_mid_vel_any(const SolveGeom<typename LineT<T>::R> &g, typename LineT<T>::V *buf,
                                              int LG, int k0, int y, int npts, int rl) {
  switch (rl) {
    case 2: z_mid_vel<2, T>(g, buf, LG, k0, y, npts); break;
    case 3: z_mid_vel<3, T>(g, buf, LG, k0, y, npts); break;
    case 4: z_mid_vel<4, T>(g, buf, LG, k0, y, npts); break;
    case 5: z_mid_vel<5, T>(g, buf, LG, k0, y, npts); break;
    case 6: z_mid_vel<6, T>(g, buf, LG, k0, y, npts); break;
    default: z_mid_vel<1, T>(g, buf, LG, k0, y, npts); break;
  }
}

// the Stockham passes' vectors: FP32 pairs, FP64 single lines
template <typename R> struct StockLine;
template <> struct StockLine<float> { typedef float2 T; };
template <> struct StockLine<double> { typedef double T; };

// lines along y (lmode L_FWD / L_INV) or the fused z pass (L_Z, or L_FWD along z
// for the Green's function transform).  axis: 1 = y, 2 = z.
template <typename R, int NC>
__global__ void __launch_bounds__(PASS_THREADS, 1) k_lines(SolveGeom<R> g, LineTiles lt,
                                                            const typename cplx_t<R>::type *in,
                                                            typename cplx_t<R>::type *out, int axis, int lmode,
                                                            int zmode, int reproj, int use_zeta) {
  typedef typename cplx_t<R>::type C;
  typedef typename Vec<R>::V V;
  constexpr int G = Vec<R>::G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftDesc sd;
  if (threadIdx.x == 0) sd = (axis == 1) ? g.fy : g.fz;
  const FftDesc &dsrc = (axis == 1) ? g.fy : g.fz;
  const int ntw = dsrc.ntw;
  C *tw = reinterpret_cast<C *>(smem_raw);
  const int N = lt.n, TK = lt.TK, L = NC * TK, LG = L / G;
  V *S = reinterpret_cast<V *>(tw + ((ntw + 7) & ~7));
  V *A = S + (size_t)LG * N;
  V *B = A + (size_t)LG * N;
  stage_table(tw, axis == 1 ? g.twy : g.twz, ntw);
  {
    C *Sc = reinterpret_cast<C *>(S);
    for (int i = threadIdx.x; i < L * N; i += blockDim.x) Sc[i] = mk(R(0), R(0));
  }
  __syncthreads();
  const LineMap lm = line_map(LG);
  const int ntiles = lt.nouter * lt.nkt;
  auto load = [&](int tile) {
    const int o = tile / lt.nkt, kt = tile - o * lt.nkt;
    tile_rows_load<R>(reinterpret_cast<C *>(S), in, spec_off<R>(o * lt.in_os, lt.in_kb, kt * TK), lt.in_rs, lt.rows_in, L,
                      NC);
    cp_async_commit();
  };
  int tile = blockIdx.x;
  if (tile < ntiles) load(tile);
  for (; tile < ntiles; tile += gridDim.x) {
    cp_async_wait_all();
    __syncthreads();
    const int next = tile + gridDim.x;
    auto hook = [&]() {
      if (next < ntiles) load(next);
    };
    const int o = tile / lt.nkt, kt = tile - o * lt.nkt;
    V *res;
    if (lmode == L_INV) {
      res = vfft_chain<true, R>(S, A, B, LG, sd, tw, lm, hook);
    } else {
      res = vfft_chain<false, R>(S, A, B, LG, sd, tw, lm, hook);
      if (lmode == L_Z) {
        typedef typename StockLine<R>::T T;
        z_multiply<T, NC>(g, reinterpret_cast<typename LineT<T>::V *>(res), LG, kt * TK, g.yk ? g.yk[o] : o, zmode,
                          reproj, use_zeta, nullptr);
        __syncthreads();
        res = vfft_chain<true, R>(res, A, B, LG, sd, tw, lm, NoHook());
      }
    }
    tile_rows_store<R>(out, reinterpret_cast<C *>(res), spec_off<R>(o * lt.out_os, lt.out_kb, kt * TK), lt.out_rs,
                       lt.rows_out, L, NC);
    __syncthreads();
  }
  cp_async_wait_all();
}

// Register-engine line pass (lmode L_FWD along y or z, L_INV along y, L_Z): one tile
// buffer per CTA, transformed in place (linefft.cuh).  The y spectrum rows are stored by
// position (row -> ky through g.yk); the z pass keeps its spectrum by position in shared
// memory (position -> kz through g.zk).  Several CTAs share an SM so that one CTA's loads
// overlap another's transforms.
constexpr int LINE_THREADS_MAX = 256;   // 96 to 256 threads (pass_threads), at most 128 registers
constexpr int LINE_CTAS = 2;

struct LineSmem {
  LineTabs tabs;
  unsigned chirp, bpos;
};
__host__ __device__ inline bool plan_twiddles(const LinePlan &p) {
  bool t = false;
  for (int i = 0; i < p.np; i++) t = t || p.tmul[i] != 0;
  return t;
}
// bytes of the tables of a line pass in shared memory (a direct plan of n points and first
// radix r0); wsize / csize: a twiddle, a complex value
__host__ __device__ constexpr size_t line_tab_bytes(int n, bool twiddles, bool split, int r0, size_t wsize) {
  return (((twiddles + split) * (size_t)n * wsize + 15) & ~(size_t)15) +
         (((size_t)(n / r0) * sizeof(int) + 15) & ~(size_t)15);
}
__host__ __device__ inline size_t line_tab_bytes(const LinePlan &p, size_t wsize, size_t csize) {
  if (!p.bl) return line_tab_bytes(p.n, plan_twiddles(p), p.split != 0, p.rad[0], wsize);
  return (((plan_twiddles(p) + (p.split != 0)) * (size_t)p.n * wsize + 15) & ~(size_t)15) +
         (((size_t)(p.bn + p.n) * csize + 15) & ~(size_t)15);
}

// carves the tables of plan pl out of shared memory and stages them (Bluestein: the product
// table of one direction; the caller
// synchronises before the first tile); tabs.buf: the first byte after them
template <typename T, typename C>
__device__ __forceinline__ LineSmem line_tables(const LinePlan &pl, const C *rtw, const C *rts, const int *rb0,
                                                const C *cg, const C *bg, bool inverse) {
  typedef typename LineT<T>::W W;
  const int n = pl.n;
  LineSmem s;
  unsigned at = 0;
  s.tabs.tw = s.tabs.tws = s.tabs.rbase = s.chirp = s.bpos = 0;
  if (plan_twiddles(pl)) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) line_smem_at<W>(at)[i] = wput<T>(rtw[i]);
    s.tabs.tw = at;
    at += (unsigned)(n * sizeof(W));
  }
  if (pl.split) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) line_smem_at<W>(at)[i] = wput<T>(rts[i]);
    s.tabs.tws = at;
    at += (unsigned)(n * sizeof(W));
  }
  at = (at + 15) & ~15u;
  if (!pl.bl) {
    const int m = n / pl.rad[0];
    for (int i = threadIdx.x; i < m; i += blockDim.x) line_smem_at<int>(at)[i] = rb0[i];
    s.tabs.rbase = at;
    at += ((unsigned)m * sizeof(int) + 15) & ~15u;
  } else {
    s.chirp = at;
    s.bpos = at + (unsigned)(pl.bn * sizeof(C));
    for (int i = threadIdx.x; i < pl.bn; i += blockDim.x) line_smem_at<C>(s.chirp)[i] = cg[i];
    for (int i = threadIdx.x; i < n; i += blockDim.x) line_smem_at<C>(s.bpos)[i] = bg[inverse ? n + i : i];
    at += (unsigned)((pl.bn + n) * sizeof(C) + 15) & ~15u;
  }
  s.tabs.buf = at;
  return s;
}
template <typename T>
__device__ __forceinline__ LineSmem line_setup(const SolveGeom<typename LineT<T>::R> &g, int axis, int lmode) {
  return axis == 1 ? line_tables<T>(g.ly, g.rtwy, g.rtsy, g.rby0, g.rchy, g.rby, lmode == L_INV)
                   : line_tables<T>(g.lz, g.rtwz, g.rtsz, g.rbz0, g.rchz, g.rbz, lmode == L_INV);
}

// rows whose second half mirrors the first (mirror = number of rows; 0: plain rows)
template <typename T> struct EvenIo : LineIo<T> {
  int mirror;
  __device__ __forceinline__ LV<T> load(int row, int g) const {
    return LineIo<T>::load(2 * row > mirror && mirror ? mirror - row : row, g);
  }
};

// the rows of tile (o, k0) of a line pass
template <typename T>
__device__ __forceinline__ LineIo<T> line_io(const LineTiles &lt, const typename cplx_t<typename LineT<T>::R>::type *in,
                                             typename cplx_t<typename LineT<T>::R>::type *out, int nc, int o, int k0) {
  typedef typename LineT<T>::R R;
  typedef typename LineT<T>::V V;
  typedef typename cplx_t<R>::type C;
  constexpr int G = LineT<T>::G;
  LineIo<T> io;
  const long long bi = spec_off<R>(o * lt.in_os, lt.in_kb, k0) * nc, bo = spec_off<R>(o * lt.out_os, lt.out_kb, k0) * nc;
  if constexpr (sizeof(T) == 4) {
    // single FP32 line: the first word of its pair, plus the kx parity
    const int odd = k0 & 1;
    io.in = reinterpret_cast<const V *>(reinterpret_cast<const R *>(in + bi - odd * nc) + odd);
    io.out = reinterpret_cast<V *>(reinterpret_cast<R *>(out + bo - odd * nc) + odd);
  } else {
    io.in = reinterpret_cast<const V *>(in + bi);
    io.out = reinterpret_cast<V *>(out + bo);
  }
  io.rs_in = lt.in_rs * nc / G;
  io.rs_out = lt.out_rs * nc / G;
  io.rows_in = lt.rows_in;
  io.rows_out = lt.rows_out;
  return io;
}

// one tile of a line pass (ends with a barrier)
template <typename T>
__device__ __forceinline__ void line_tile(const SolveGeom<typename LineT<T>::R> &g, const LineTiles &lt,
                                          const typename cplx_t<typename LineT<T>::R>::type *in,
                                          typename cplx_t<typename LineT<T>::R>::type *out, int nc, int axis, int lmode,
                                          int zmode, int reproj, int use_zeta, const LineSmem &s, int tile) {
  typedef typename LineT<T>::V V;
  typedef EvenIo<T> IO;
  const LinePlan &pl = (axis == 1) ? g.ly : g.lz;
  const int LG = nc * lt.TK / LineT<T>::G;
  const RtPlan rp{pl, LG, lt.dLG};
  const bool blue = pl.bl != 0;
  int o, k0;
  line_tile_at(lt, tile, lt.TK, o, k0);
  if (lt.even && axis == 2 && 2 * (g.yk ? g.yk[o] : o) > g.M[1]) return;
  IO io;
  static_cast<LineIo<T> &>(io) = line_io<T>(lt, in, out, nc, o, k0);
  io.mirror = lt.even ? lt.n : 0;
  V *const buf = line_smem_at<V>(s.tabs.buf);
  const int y = g.yk ? g.yk[o] : o;  // z pass: the spectrum row's ky
  const bool zvel = lmode == L_Z && zmode == Z_VEL && nc == 3 && z_plain(g, use_zeta);
  const bool mid = zvel && !blue && pl.np >= 2 && z_mid_radix(pl.rad[pl.np - 1]);
  const int nrep = lmode == L_Z && blue ? 2 : 1;
  for (int rep = 0; rep < nrep; rep++) {
    const bool binv = lmode == L_INV || rep == 1;
    if (blue) {
      lchirp_in<T, IO>(s.tabs.buf, pl.n, LG, lt.dLG, s.chirp, rep == 0 && lmode != L_INV ? lt.rows_in : pl.bn, binv,
                       rep == 0, io);
      __syncthreads();
    }
    if (blue || lmode != L_INV) {
      const int pe = mid ? pl.np - 1 : pl.np;
      for (int p = 0; p < pe; p++) {
        lphase_any<false, true, T, IO>(rp, p, s.tabs, io, !blue, false, !blue && lmode == L_FWD && p == pl.np - 1);
        __syncthreads();
      }
    }
    if (blue) {
      // (the z pass's inverse table stays in global memory)
      typedef typename cplx_t<typename LineT<T>::R>::type C;
      lchirp_mul<T>(s.tabs.buf, pl.n, LG, lt.dLG, rep == 1 ? g.rbz + pl.n : line_smem_at<C>(s.bpos));
      __syncthreads();
    } else if (lmode == L_Z) {
      if (zvel) z_mid_vel_any<T>(g, buf, LG, k0, y, plan_points(pl), mid ? pl.rad[pl.np - 1] : 1);
      else if (nc == 3) z_multiply<T, 3>(g, buf, LG, k0, y, zmode, reproj, use_zeta, g.zk);
      else z_multiply<T, 1>(g, buf, LG, k0, y, zmode, reproj, use_zeta, g.zk);
      __syncthreads();
    }
    if (blue || lmode != L_FWD) {
      for (int p = mid ? pl.np - 2 : pl.np - 1; p >= 0; p--) {
        lphase_any<true, true, T, IO>(rp, p, s.tabs, io, !blue, !blue && lmode == L_INV && p == pl.np - 1, false);
        __syncthreads();
      }
    }
    if (blue) {
      const bool last = rep == nrep - 1;
      lchirp_out<T, IO>(s.tabs.buf, pl.n, LG, lt.dLG, s.chirp, last && lmode != L_FWD ? lt.rows_out : pl.bn, binv,
                        last, io);
      __syncthreads();
      if (!last) {
        if (nc == 3) z_multiply<T, 3>(g, buf, LG, k0, y, zmode, reproj, use_zeta, nullptr);
        else z_multiply<T, 1>(g, buf, LG, k0, y, zmode, reproj, use_zeta, nullptr);
        __syncthreads();
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS)
    k_rlines(SolveGeom<typename LineT<T>::R> g, LineTiles lt, const typename cplx_t<typename LineT<T>::R>::type *in,
             typename cplx_t<typename LineT<T>::R>::type *out, int nc, int axis, int lmode, int zmode, int reproj,
             int use_zeta) {
  const LineSmem s = line_setup<T>(g, axis, lmode);
  __syncthreads();
  const int ntiles = lt.nouter * lt.nkt;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    line_tile<T>(g, lt, in, out, nc, axis, lmode, zmode, reproj, use_zeta, s, tile);
}

// ---------------------------------------------------------------- compile-time line passes
// forward phases P .. PE - 1 and inverse phases P .. 0 of a compile-time plan, each with its
// barrier
template <typename T, typename PL, int P, int PE, bool GOUT>
__device__ __forceinline__ void ct_forward(const LineTabs &tb, const LineIo<T> &io) {
  if constexpr (P < PE) {
    lphase<PL::rad(P), false, T, LineIo<T>, PL>(PL(), P, tb, io, true, false, GOUT && P == PL::NP - 1);
    __syncthreads();
    ct_forward<T, PL, P + 1, PE, GOUT>(tb, io);
  }
}
template <typename T, typename PL, int P, bool GIN>
__device__ __forceinline__ void ct_inverse(const LineTabs &tb, const LineIo<T> &io) {
  if constexpr (P >= 0) {
    lphase<PL::rad(P), true, T, LineIo<T>, PL>(PL(), P, tb, io, true, GIN && P == PL::NP - 1, false);
    __syncthreads();
    ct_inverse<T, PL, P - 1, GIN>(tb, io);
  }
}
// asks for a tile's input rows (`bytes` each) to be brought into L2
template <typename T> __device__ __forceinline__ void line_prefetch(const LineIo<T> &io, int rows, unsigned bytes) {
  for (int r = threadIdx.x; r < rows; r += blockDim.x)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(io.in + (long long)r * io.rs_in)),
                 "r"(bytes)
                 : "memory");
}
// k_rlines for a compile-time plan PL of three-component lines, one mode each (L_Z: the
// plain velocity solve with the last digit in the multiply)
template <typename T, int LMODE, typename PL>
__device__ __forceinline__ void line_tile_ct(const SolveGeom<typename LineT<T>::R> &g, const LineIo<T> &io,
                                             const LineTabs &tb, int o, int k0) {
  typedef typename LineT<T>::V V;
  if constexpr (LMODE == L_FWD) {
    ct_forward<T, PL, 0, PL::NP, true>(tb, io);
  } else if constexpr (LMODE == L_INV) {
    ct_inverse<T, PL, PL::NP - 1, true>(tb, io);
  } else {
    constexpr int RL = PL::NP > 1 ? z_mid_block(PL::rad(PL::NP - 1)) : 1;
    constexpr int PE = RL > 1 ? PL::NP - 1 : PL::NP;
    ct_forward<T, PL, 0, PE, false>(tb, io);
    z_mid_vel<RL, T>(g, line_smem_at<V>(tb.buf), PL::LG(), k0, g.yk ? g.yk[o] : o,
                     PL::split() ? 2 * PL::n() : PL::n());
    __syncthreads();
    ct_inverse<T, PL, PE - 1, false>(tb, io);
  }
}
template <typename T, int LMODE, typename PL>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS)
    k_rlines_ct(SolveGeom<typename LineT<T>::R> g, LineTiles lt, const typename cplx_t<typename LineT<T>::R>::type *in,
                typename cplx_t<typename LineT<T>::R>::type *out, int, int axis, int, int, int, int) {
  constexpr int TK = PL::LG() * LineT<T>::G / 3;
  const LineSmem s = line_setup<T>(g, axis, LMODE);
  __syncthreads();
  const int ntiles = lt.nouter * lt.nkt;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    int o, k0;
    line_tile_at(lt, tile, TK, o, k0);
    const LineIo<T> io = line_io<T>(lt, in, out, 3, o, k0);
    if (LMODE == L_Z && tile + (int)gridDim.x < ntiles) {
      // the next tile's rows on their way to L2 while this one is transformed
      int no, nk;
      line_tile_at(lt, tile + gridDim.x, TK, no, nk);
      line_prefetch<T>(line_io<T>(lt, in, out, 3, no, nk), PL::n(), PL::LG() * 16);
    }
    line_tile_ct<T, LMODE, PL>(g, io, s.tabs, o, k0);
  }
}

// ---------------------------------------------------------------- batches of patches
// A batched pass runs one pass family (x forward, y forward, the fused z pass, y
// inverse or x inverse) of every patch of a batch in one launch.  Every patch has a
// descriptor (its geometry and the pass's tiles and arrays) and a range of work
// items, one per tile.  CTAs take chunks of consecutive items from a counter in
// global memory (zeroed before the launch) and load a patch's descriptor and tables
// into shared memory when the patch changes.  Each tile is transformed by the same
// code as in the pass of a single plan, so a patch's result is bit-identical to
// its solve alone.
template <typename R> struct PassDesc {
  SolveGeom<R> g;
  LineTiles lt;     // line passes: the tiles of this patch's lines
  const void *in;   // pass input (x forward: the patch's vorticity)
  void *out;        // pass output (x inverse: the patch's velocity)
  int RB, cs;       // x passes: rows per tile, component stride of the real field
  int vec16;        // x forward: rows are staged in 16-byte chunks
  int first;        // first work item of the patch
  FastDiv dLG;      // x passes: division by the line vectors of a tile
  int ntiles;
  int patch;        // index into the caller's arrays
  int cls;          // compile-time plan (plan_class), 0: run-time plan
};
// key of a compile-time plan in the batched kernels
__host__ __device__ constexpr int plan_class(int n, int split, int lg) { return n * 4 + split * 2 + (lg == 12 ? 1 : 0); }
struct BatchWork {
  const void *desc;   // PassDesc<R>[npatch]
  int npatch, nitems, chunk, pad;
  unsigned *counter;  // zero at the launch
};
// the caller's arrays of a batched solve, one per patch (x forward: vorticity, x
// inverse and ghost fill: velocity), passed by value with the launch
constexpr int BATCH_MAX = 1024;
struct BatchIo {
  const void *p[BATCH_MAX];
};

// the CTA's next chunk of work items [i0, i1); false when none is left
__device__ __forceinline__ bool batch_next(const BatchWork &bw, int &i0, int &i1) {
  __shared__ int s_next;
  __syncthreads();
  if (threadIdx.x == 0) s_next = (int)atomicAdd(bw.counter, (unsigned)bw.chunk);
  __syncthreads();
  i0 = s_next;
  i1 = min(i0 + bw.chunk, bw.nitems);
  return i0 < bw.nitems;
}

// the patch that holds work item `item`, and a copy of its descriptor in shared
// memory when it is not the current one (all threads; ends with a barrier when it
// loads).  Returns true when the patch changed.
template <typename R>
__device__ __forceinline__ bool batch_patch(const BatchWork &bw, int item, PassDesc<R> &sd, int &cur) {
  const PassDesc<R> *d = reinterpret_cast<const PassDesc<R> *>(bw.desc);
  if (cur >= 0 && item >= sd.first && item < sd.first + sd.ntiles) return false;
  int lo = 0, hi = bw.npatch - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (d[mid].first <= item) lo = mid;
    else hi = mid - 1;
  }
  __syncthreads();  // everyone is done with the previous descriptor
  const unsigned *src = reinterpret_cast<const unsigned *>(d + lo);
  unsigned *dst = reinterpret_cast<unsigned *>(&sd);
  for (int i = threadIdx.x; i < (int)(sizeof(PassDesc<R>) / 4); i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  cur = lo;
  return true;
}

template <typename R>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_lines_batch(BatchWork bw, int axis, int lmode, int zmode) {
  typedef typename cplx_t<R>::type C;
  typedef typename StockLine<R>::T T;
  __shared__ PassDesc<R> sd;
  LineSmem s;
  int cur = -1, i0, i1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (batch_patch<R>(bw, it, sd, cur)) {
        s = line_setup<T>(sd.g, axis, lmode);
        __syncthreads();
      }
      line_tile<T>(sd.g, sd.lt, reinterpret_cast<const C *>(sd.in), reinterpret_cast<C *>(sd.out), 3, axis, lmode,
                   zmode, 0, 0, s, it - sd.first);
    }
  }
}

// ---------------------------------------------------------------- x passes, register engine
// R2C / C2R of real rows through a half-length complex transform: the packed points
// z[m] = x[2m] + i x[2m+1], m < N = Mx/2, give the Mx-point spectrum by
//   X[k] = (Z[k] + conj Z[N-k] - i W^k (Z[k] - conj Z[N-k])) / 2,   W = exp(-2 pi i / Mx),
// and back by Z[k] = X[k] + conj X[N-k] + i W^-k (X[k] - conj X[N-k]).  The lines are
// transformed as line vectors (linefft.cuh): in FP32 a vector holds one component of two
// rows.  A free axis of even length has exactly the second half of its packed points
// zero: a split plan.  A tile is RB rows of NC components, LG = NC RB / G vectors a
// point, vector g = rho NC + c for row group rho.  The forward pass stages its raw rows in
// shared memory (the next tile's rows stream in while this one is transformed) and its first
// phase packs from there; the inverse pass reads the spectrum rows straight into the
// twist and its last phase writes the real rows.
struct XSmem {
  LineTabs tabs;
  unsigned chirp, bpos;
  unsigned ext, xpos;
  unsigned srow;   // first vector of every row of the tile in the spectral array
  unsigned stage;  // forward: raw rows
  unsigned rows;   // inverse: offset of every row of the tile in the real field, -1: none
};

// input of the forward transform: packed point m of the staged rows (rows of P0 NC reals)
template <typename T, int NC> struct XStageIo {
  typedef typename LineT<T>::R R;
  unsigned stage;
  int P0;
  int rows_in, rows_out;
  __device__ __forceinline__ LV<T> load(int m, int g) const {
    const int rho = g / NC, c = g - rho * NC;
    const bool odd = 2 * m + 1 < P0;
    const R *p = line_smem_at<R>(stage) + rho * LineT<T>::G * P0 * NC + 2 * m * NC + c;
    if constexpr (LineT<T>::G == 2) {
      const R *q = p + P0 * NC;
      return {make_float2(p[0], q[0]), make_float2(odd ? p[NC] : R(0), odd ? q[NC] : R(0))};
    } else {
      return {p[0], odd ? p[NC] : R(0)};
    }
  }
  __device__ __forceinline__ void store(int, int, const LV<T> &) const {}
};
// output of the inverse transform: packed point m to the real rows (component stride cs)
template <typename T, int NC> struct XRowIo {
  typedef typename LineT<T>::R R;
  R *out;
  unsigned rows;
  int P0, cs;
  int rows_in, rows_out;
  __device__ __forceinline__ LV<T> load(int, int) const { return lzero<T>(); }
  __device__ __forceinline__ void put(int row, int m, int c, R a, R b) const {
    const long long o = line_smem_at<long long>(rows)[row];
    if (o < 0) return;
    R *p = out + o + (size_t)(2 * m) * cs + c;
    p[0] = a;
    if (2 * m + 1 < P0) p[cs] = b;
  }
  __device__ __forceinline__ void store(int m, int g, const LV<T> &v) const {
    const int rho = g / NC, c = g - rho * NC;
    if constexpr (LineT<T>::G == 2) {
      put(2 * rho, m, c, v.re.x, v.im.x);
      put(2 * rho + 1, m, c, v.re.y, v.im.y);
    } else {
      put(rho, m, c, v.re, v.im);
    }
  }
};

// shared memory of an x pass of RB rows a tile (G rows a vector, wsize bytes a twiddle)
__host__ __device__ inline size_t x_tab_bytes(const LinePlan &p, int N, int H, size_t wsize, size_t csize) {
  return line_tab_bytes(p, wsize, csize) + (((size_t)H * csize + 15) & ~(size_t)15) +
         (((size_t)N * sizeof(int) + 15) & ~(size_t)15);
}

template <typename T, int NC>
__device__ __forceinline__ XSmem x_setup(const SolveGeom<typename LineT<T>::R> &g, int RB, bool inverse) {
  typedef typename LineT<T>::R R;
  typedef typename cplx_t<R>::type C;
  XSmem s;
  const LineSmem l = line_tables<T>(g.lx, g.rtwx, g.rtsx, g.rbx0, g.rchx, g.rbx, inverse);
  s.tabs = l.tabs;
  s.chirp = l.chirp;
  s.bpos = l.bpos;
  unsigned at = l.tabs.buf;
  s.ext = at;
  at += (unsigned)(g.H * sizeof(C) + 15) & ~15u;
  s.xpos = at;
  at += (unsigned)(g.N2 * sizeof(int) + 15) & ~15u;
  for (int i = threadIdx.x; i < g.H; i += blockDim.x) line_smem_at<C>(s.ext)[i] = g.rextx[i];
  for (int i = threadIdx.x; i < g.N2; i += blockDim.x) line_smem_at<int>(s.xpos)[i] = g.xpos[i];
  s.srow = at;
  at += (unsigned)(RB * sizeof(long long) + 15) & ~15u;
  s.stage = s.rows = at;
  if (inverse) at += (unsigned)(RB * sizeof(long long) + 15) & ~15u;
  else at += (unsigned)(RB * g.P[0] * NC * sizeof(R) + 15) & ~15u;
  s.tabs.buf = at;
  return s;
}

// x forward: raw rows of tile `tile` into the stage (cp.async, committed)
template <typename R, int NC>
__device__ __forceinline__ void rxf_load(const SolveGeom<R> &g, const R *__restrict__ in, int RB, int cs, int vec16,
                                         R *stage, int tile) {
  const int P0 = g.P[0];
  const int nrows = g.P[1] * g.P[2];
  const int row0 = tile * RB;
  for (int rr = 0; rr < RB; rr++) {
    const int row = row0 + rr;
    if (row >= nrows) break;
    const int y = row % g.P[1], z = row / g.P[1];
    const R *src = in + (((size_t)(z + g.off[2]) * g.ext[1] + (y + g.off[1])) * g.ext[0] + g.off[0]) * cs;
    R *dst = stage + (size_t)rr * P0 * NC;
    if (vec16) {
      const int nch = (P0 * NC * (int)sizeof(R)) / 16;
      for (int c = threadIdx.x; c < nch; c += blockDim.x)
        cp_async16(reinterpret_cast<char *>(dst) + 16 * c, reinterpret_cast<const char *>(src) + 16 * c);
    } else {
      for (int e = threadIdx.x; e < P0 * NC; e += blockDim.x) {
        const int x = e / NC, c = e - x * NC;
        if (sizeof(R) == 8) cp_async8(dst + e, src + (size_t)x * cs + c);
        else cp_async4(dst + e, src + (size_t)x * cs + c);
      }
    }
  }
  cp_async_commit();
}

// Vector v of spectral row `row` (z P1 + y): the rows of a z plane lie block by block of kx,
// so that a y line tile is contiguous.
template <typename R, int NC>
__device__ __forceinline__ size_t spec_vec(const SolveGeom<R> &g, int row, int v) {
  constexpr int XG = sizeof(R) == 4 ? 2 : 1, BV = spec_block<R>() * NC / XG;  // vectors of a block row
  const int z = row / g.P[1], y = row - z * g.P[1];
  const int kb = v / BV, nkb = g.Hp / spec_block<R>();
  return (((size_t)z * nkb + kb) * g.P[1] + y) * BV + (v - kb * BV);
}

// the first vector of a row's block 0, and the stride between its blocks
template <typename R, int NC> __device__ __forceinline__ long long spec_row0(const SolveGeom<R> &g, int row) {
  return (long long)spec_vec<R, NC>(g, row, 0);
}
template <typename R, int NC> __device__ __forceinline__ long long spec_kb(const SolveGeom<R> &g) {
  return (long long)g.P[1] * (spec_block<R>() * NC / (sizeof(R) == 4 ? 2 : 1));
}

// forward / inverse phases of the x transforms: all in shared memory but the outer end
template <typename T, typename IO, typename PL, bool INV, int P>
__device__ __forceinline__ void x_phase_ct(const LineTabs &tb, const IO &io) {
  lphase<PL::rad(P), INV, T, IO, PL>(PL(), P, tb, io, true, false, false);
  __syncthreads();
}

// row groups of a tile of a compile-time x plan
template <typename PL, int NC> __device__ constexpr int x_groups() {
  if constexpr (PL::RT) return 1;
  else return PL::LG() / NC;
}

// x forward of a staged tile (the caller waited for its copies and synchronised);
// `prefetch` runs once the stage has been read.  Ends with a barrier.  PL: a compile-time
// plan, or RtPlan for the run-time one.
template <typename T, int NC, typename PL, typename Prefetch>
__device__ __forceinline__ void rxf_tile(const SolveGeom<typename LineT<T>::R> &g,
                                         typename cplx_t<typename LineT<T>::R>::type *__restrict__ X, int RB,
                                         const FastDiv &dLG, const XSmem &s, int tile, Prefetch prefetch) {
  typedef typename LineT<T>::R R;
  typedef typename cplx_t<R>::type C;
  constexpr int G = LineT<T>::G;
  constexpr int XG = sizeof(R) == 4 ? 2 : 1;  // kx of a spectral vector
  const LinePlan &pl = g.lx;
  const bool blue = pl.bl != 0;
  const int N = g.N2, LG = NC * RB / G, P0 = g.P[0];
  const RtPlan rp{pl, LG, dLG};
  const int *xpos = line_smem_at<int>(s.xpos);
  const C *ext = line_smem_at<C>(s.ext);
  XStageIo<T, NC> io;
  io.stage = s.stage;
  io.P0 = P0;
  io.rows_in = (P0 + 1) / 2;
  io.rows_out = N;
  const int nrows = g.P[1] * g.P[2], row0 = tile * RB;
  long long *srow = line_smem_at<long long>(s.srow);
  for (int rr = threadIdx.x; rr < RB; rr += blockDim.x)
    srow[rr] = row0 + rr < nrows ? spec_row0<R, NC>(g, row0 + rr) : -1;
  if constexpr (!PL::RT) {
    x_phase_ct<T, XStageIo<T, NC>, PL, false, 0>(s.tabs, io);
    prefetch();
    if constexpr (PL::NP > 1) x_phase_ct<T, XStageIo<T, NC>, PL, false, 1>(s.tabs, io);
    if constexpr (PL::NP > 2) x_phase_ct<T, XStageIo<T, NC>, PL, false, 2>(s.tabs, io);
  } else {
  if (blue) {
    lchirp_in<T>(s.tabs.buf, pl.n, LG, dLG, s.chirp, io.rows_in, false, true, io);
    __syncthreads();
    prefetch();
  }
  for (int p = 0; p < pl.np; p++) {
    lphase_any<false, false, T>(rp, p, s.tabs, io, !blue, false, false);
    __syncthreads();
    if (p == 0 && !blue) prefetch();
  }
  if (blue) {
    lchirp_mul<T>(s.tabs.buf, pl.n, LG, dLG, line_smem_at<C>(s.bpos));
    __syncthreads();
    for (int p = pl.np - 1; p >= 0; p--) {
      lphase_any<true, false, T>(rp, p, s.tabs, io, false, false, false);
      __syncthreads();
    }
    lchirp_out<T>(s.tabs.buf, pl.n, LG, dLG, s.chirp, N, false, false, io);
    __syncthreads();
  }
  }
  // the twist.  Consecutive threads: the vectors of a block row, then the tile's rows, then
  // the next block: RB rows of 192 bytes lie together
  const T half = pset(T(), R(0.5));
  constexpr int BV = spec_block<R>() * NC / XG;
  const int nrg = PL::RT ? RB / G : x_groups<PL, NC>(), nrs = __ffs(nrg) - 1;  // a power of two
  const int nt = g.Hp / XG * NC * nrg;
  const long long kbs = spec_kb<R, NC>(g);
  for (int t = threadIdx.x; t < nt; t += blockDim.x) {
    const int w0 = t / BV, kb = w0 >> nrs, rho = w0 - (kb << nrs), bv = t - w0 * BV;
    const int v = kb * BV + bv;
    if (srow[rho * G] < 0) continue;
    const int kv = v / NC, c = v - kv * NC;
    const typename LineT<T>::V *b = line_smem_at<typename LineT<T>::V>(s.tabs.buf) + rho * NC + c;
    LV<T> o[XG];
#pragma unroll
    for (int h = 0; h < XG; h++) {
      const int k = kv * XG + h;
      o[h] = lzero<T>();
      if (k < g.H) {
        const LV<T> zk = vget(b[xpos[k == N ? 0 : k] * LG]);
        const LV<T> zn = vget(b[xpos[k == 0 || k == N ? 0 : N - k] * LG]);
        const C w = ext[k];
        const LV<T> a = {padd(zk.re, zn.re), psub(zk.im, zn.im)}, d = {psub(zk.re, zn.re), padd(zk.im, zn.im)};
        const LV<T> t2 = lmul<T>(d, pset(T(), w.x), pset(T(), w.y));
        o[h] = lsub_i(a, t2);  // a - i W^k d
        o[h].re = pmulp(o[h].re, half);
        o[h].im = pmulp(o[h].im, half);
      }
    }
    const long long at = kb * kbs + bv;
    if constexpr (G == 2) {
      float4 *x = reinterpret_cast<float4 *>(X) + at;
      x[srow[2 * rho]] = make_float4(o[0].re.x, o[1].re.x, o[0].im.x, o[1].im.x);
      if (srow[2 * rho + 1] >= 0) x[srow[2 * rho + 1]] = make_float4(o[0].re.y, o[1].re.y, o[0].im.y, o[1].im.y);
    } else if constexpr (XG == 2) {
      reinterpret_cast<float4 *>(X)[srow[rho] + at] = make_float4(o[0].re, o[1].re, o[0].im, o[1].im);
    } else {
      X[srow[rho] + at] = vput(o[0]);
    }
  }
  __syncthreads();
}

template <typename T, int NC, typename PL = RtPlan>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS)
    k_rxfwd(SolveGeom<typename LineT<T>::R> g, const typename LineT<T>::R *__restrict__ in,
            typename cplx_t<typename LineT<T>::R>::type *__restrict__ X, int RB, int cs, int vec16, FastDiv dLG) {
  const XSmem s = x_setup<T, NC>(g, RB, false);
  const int nrows = g.P[1] * g.P[2];
  const int ntiles = (nrows + RB - 1) / RB;
  int tile = blockIdx.x;
  if (tile < ntiles) rxf_load<typename LineT<T>::R, NC>(g, in, RB, cs, vec16, line_smem_at<typename LineT<T>::R>(s.stage), tile);
  for (; tile < ntiles; tile += gridDim.x) {
    cp_async_wait_all();
    __syncthreads();
    const int next = tile + gridDim.x;
    rxf_tile<T, NC, PL>(g, X, RB, dLG, s, tile, [&]() {
      if (next < ntiles) rxf_load<typename LineT<T>::R, NC>(g, in, RB, cs, vec16, line_smem_at<typename LineT<T>::R>(s.stage), next);
    });
  }
  cp_async_wait_all();
}

template <typename T, int NC>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_rxfwd_batch(BatchWork bw, BatchIo bio) {
  typedef typename LineT<T>::R R;
  typedef typename cplx_t<R>::type C;
  __shared__ PassDesc<R> sd;
  XSmem s;
  int cur = -1, i0, i1, staged = -1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (cur >= 0 && (it < sd.first || it >= sd.first + sd.ntiles)) {
        cp_async_wait_all();  // no copy into the old layout may still be in flight
        staged = -1;
      }
      if (batch_patch<R>(bw, it, sd, cur)) {
        s = x_setup<T, NC>(sd.g, sd.RB, false);
        __syncthreads();
      }
      const R *in = reinterpret_cast<const R *>(bio.p[sd.patch]);
      if (staged != it) rxf_load<R, NC>(sd.g, in, sd.RB, sd.cs, sd.vec16, line_smem_at<R>(s.stage), it - sd.first);
      cp_async_wait_all();
      __syncthreads();
      const int next = it + 1;
      const bool pre = next < i1 && next < sd.first + sd.ntiles;
      rxf_tile<T, NC, RtPlan>(sd.g, reinterpret_cast<C *>(sd.out), sd.RB, sd.dLG, s, it - sd.first, [&]() {
        if (pre) rxf_load<R, NC>(sd.g, in, sd.RB, sd.cs, sd.vec16, line_smem_at<R>(s.stage), next - sd.first);
      });
      staged = pre ? next : -1;
    }
  }
  cp_async_wait_all();
}

// spectral vector v of a row: the values of its (one or two) kx
__device__ __forceinline__ void spec_row(const float2 *row, size_t v, float2 *o) {
  const float4 q = __ldg(reinterpret_cast<const float4 *>(row) + v);
  o[0] = make_float2(q.x, q.z);
  o[1] = make_float2(q.y, q.w);
}
__device__ __forceinline__ void spec_row(const double2 *row, size_t v, double2 *o) { o[0] = __ldg(row + v); }

// one tile of the x inverse pass (ends with a barrier)
template <typename T, int NC, typename PL>
__device__ __forceinline__ void rxi_tile(const SolveGeom<typename LineT<T>::R> &g,
                                         const typename cplx_t<typename LineT<T>::R>::type *__restrict__ X,
                                         typename LineT<T>::R *__restrict__ outp, int RB, int cs, const FastDiv &dLG,
                                         const XSmem &s, int tile) {
  typedef typename LineT<T>::R R;
  typedef typename cplx_t<R>::type C;
  constexpr int G = LineT<T>::G;
  constexpr int XG = sizeof(R) == 4 ? 2 : 1;
  const LinePlan &pl = g.lx;
  const bool blue = pl.bl != 0;
  const int N = g.N2, LG = NC * RB / G, P0 = g.P[0];
  const RtPlan rp{pl, LG, dLG};
  const int *xpos = line_smem_at<int>(s.xpos);
  const C *ext = line_smem_at<C>(s.ext);
  const int nrows = g.P[1] * g.P[2], row0 = tile * RB;
  long long *srow = line_smem_at<long long>(s.srow);
  for (int rr = threadIdx.x; rr < RB; rr += blockDim.x) {
    const int row = row0 + rr;
    srow[rr] = spec_row0<R, NC>(g, row < nrows ? row : row0);
    const int y = row % g.P[1], z = row / g.P[1];
    line_smem_at<long long>(s.rows)[rr] = row < nrows ? (long long)((((size_t)(z + g.off[2]) * g.ext[1] + (y + g.off[1])) * g.ext[0] + g.off[0]) * cs)
                             : -1;
  }
  // the twist: Z[k] and Z[N-k] from X[k] and X[N-k]; k <= N/2 from this side, k > N/2 from
  // its mirror
  const int nh = N / 2 / XG + 1, nv = nh * NC;
  constexpr int BV = spec_block<R>() * NC / XG;
  const int nrg = PL::RT ? RB / G : x_groups<PL, NC>(), nrs = __ffs(nrg) - 1, nb = (nv + BV - 1) / BV;
  const long long kbs = spec_kb<R, NC>(g);
  __syncthreads();
  {
    for (int t = threadIdx.x; t < nb * nrg * BV; t += blockDim.x) {
      const int w0 = t / BV, kb = w0 >> nrs, rho = w0 - (kb << nrs);
      const int v = kb * BV + (t - w0 * BV);
      if (v >= nv) continue;
      typename LineT<T>::V *b = line_smem_at<typename LineT<T>::V>(s.tabs.buf) + rho * NC;
      const int kv = v / NC, c = v - kv * NC;
      // vector w of the row at base r
      auto at = [&](long long r, int w) { return (size_t)(r + (w / BV) * kbs + w % BV); };
      C xk[G][XG], xn[G][XG];
#pragma unroll
      for (int q = 0; q < G; q++) {
        const long long r = srow[rho * G + q];
        spec_row(X, at(r, v), xk[q]);
        if constexpr (XG == 2) {
          // X[N - 2 kv] is the even, X[N - 2 kv - 1] the odd value of a pair when N is even,
          // both lie in one pair when it is odd
          C m0[XG], m1[XG];
          const int n0 = N - 2 * kv, n1 = max(n0 - 1, 0);
          spec_row(X, at(r, (n0 >> 1) * NC + c), m0);
          spec_row(X, at(r, (n1 >> 1) * NC + c), m1);
          xn[q][0] = (n0 & 1) ? m0[1] : m0[0];
          xn[q][1] = (n1 & 1) ? m1[1] : m1[0];
        } else {
          spec_row(X, at(r, (N - kv) * NC + c), xn[q]);
        }
      }
#pragma unroll
      for (int h = 0; h < XG; h++) {
        const int k = kv * XG + h;
        if (2 * k > N) continue;
        LV<T> a, m;
        if constexpr (G == 2) {
          a = {make_float2(xk[0][h].x, xk[1][h].x), make_float2(xk[0][h].y, xk[1][h].y)};
          m = {make_float2(xn[0][h].x, xn[1][h].x), make_float2(xn[0][h].y, xn[1][h].y)};
        } else {
          a = {xk[0][h].x, xk[0][h].y};
          m = {xn[0][h].x, xn[0][h].y};
        }
        if (k == 0) a.im = m.im = pset(T(), R(0));  // DC and Nyquist are real
        const LV<T> sum = {padd(a.re, m.re), psub(a.im, m.im)}, dif = {psub(a.re, m.re), padd(a.im, m.im)};
        const C w = ext[k];
        const LV<T> t = lmulc<T>(dif, pset(T(), w.x), pset(T(), w.y));  // W^-k (X[k] - conj X[N-k])
        b[xpos[k] * LG + c] = vput(ladd_i(sum, t));
        if (k > 0 && 2 * k < N) {
          const LV<T> z = lsub_i(sum, t);
          b[xpos[N - k] * LG + c] = vput(LV<T>{z.re, pneg(z.im)});
        }
      }
    }
  }
  __syncthreads();
  XRowIo<T, NC> io;
  io.out = outp;
  io.rows = s.rows;
  io.P0 = P0;
  io.cs = cs;
  io.rows_in = N;
  io.rows_out = (P0 + 1) / 2;
  if constexpr (!PL::RT) {
    if constexpr (PL::NP > 2) x_phase_ct<T, XRowIo<T, NC>, PL, true, 2>(s.tabs, io);
    if constexpr (PL::NP > 1) x_phase_ct<T, XRowIo<T, NC>, PL, true, 1>(s.tabs, io);
    x_phase_ct<T, XRowIo<T, NC>, PL, true, 0>(s.tabs, io);
  } else {
  if (blue) {
    lchirp_in<T>(s.tabs.buf, pl.n, LG, dLG, s.chirp, N, true, false, io);
    __syncthreads();
    for (int p = 0; p < pl.np; p++) {
      lphase_any<false, false, T>(rp, p, s.tabs, io, false, false, false);
      __syncthreads();
    }
    lchirp_mul<T>(s.tabs.buf, pl.n, LG, dLG, line_smem_at<C>(s.bpos));
    __syncthreads();
  }
  for (int p = pl.np - 1; p >= 0; p--) {
    lphase_any<true, false, T>(rp, p, s.tabs, io, !blue, false, false);
    __syncthreads();
  }
  if (blue) {
    lchirp_out<T>(s.tabs.buf, pl.n, LG, dLG, s.chirp, io.rows_out, true, true, io);
    __syncthreads();
  }
  }
}

template <typename T, int NC, typename PL = RtPlan>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS)
    k_rxinv(SolveGeom<typename LineT<T>::R> g, const typename cplx_t<typename LineT<T>::R>::type *__restrict__ X,
            typename LineT<T>::R *__restrict__ outp, int RB, int cs, FastDiv dLG) {
  const XSmem s = x_setup<T, NC>(g, RB, true);
  __syncthreads();
  const int ntiles = (g.P[1] * g.P[2] + RB - 1) / RB;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) rxi_tile<T, NC, PL>(g, X, outp, RB, cs, dLG, s, tile);
}

template <typename T, int NC>
__global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_rxinv_batch(BatchWork bw, BatchIo bio) {
  typedef typename LineT<T>::R R;
  typedef typename cplx_t<R>::type C;
  __shared__ PassDesc<R> sd;
  XSmem s;
  int cur = -1, i0, i1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (batch_patch<R>(bw, it, sd, cur)) {
        s = x_setup<T, NC>(sd.g, sd.RB, true);
        __syncthreads();
      }
      rxi_tile<T, NC, RtPlan>(sd.g, reinterpret_cast<const C *>(sd.in), (R *)bio.p[sd.patch], sd.RB, sd.cs, sd.dLG, s,
                      it - sd.first);
    }
  }
}

// Vector v of a spectral row: two neighbouring kx of one component in FP32, as
// (re, re, im, im); one complex value in FP64.
template <typename R>
__device__ __forceinline__ void spec_put(typename cplx_t<R>::type *row, size_t v, typename cplx_t<R>::type a,
                                         typename cplx_t<R>::type b) {
  if constexpr (sizeof(R) == 4) reinterpret_cast<float4 *>(row)[v] = make_float4(a.x, b.x, a.y, b.y);
  else row[v] = a;
}
// component c at kx index m of a spectral row
template <typename R, int NC>
__device__ __forceinline__ typename cplx_t<R>::type spec_get(const typename cplx_t<R>::type *row, int m, int c) {
  if constexpr (sizeof(R) == 4) {
    const float *p = reinterpret_cast<const float *>(row) + 4 * ((m >> 1) * NC + c) + (m & 1);
    return make_float2(p[0], p[2]);
  } else {
    return row[(size_t)m * NC + c];
  }
}

// ---------------------------------------------------------------- x forward (R2C)
// RB rows per tile, L = NC RB real lines packed as N = Mx/2 complex points
// (z[m] = x[2m] + i x[2m+1]); the Mx-point spectrum X[k], k < H follows from Z[k]
// and Z[N-k].  Rows of the real cuboid are staged raw in S.
template <typename R, int NC>
__global__ void __launch_bounds__(PASS_THREADS, 1) k_xfwd(SolveGeom<R> g, const R *__restrict__ in,
                                                           typename cplx_t<R>::type *__restrict__ X, int RB, int cs,
                                                           int vec16) {
  typedef typename cplx_t<R>::type C;
  typedef typename Vec<R>::V V;
  constexpr int G = Vec<R>::G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftDesc sd;
  if (threadIdx.x == 0) sd = g.fx;
  const int ntw = g.fx.ntw + g.fx.next;
  C *tw = reinterpret_cast<C *>(smem_raw);
  const int N = g.N2, L = NC * RB, LG = L / G;
  const int P0 = g.P[0];
  const size_t sreal = (size_t)RB * P0 * NC;  // staged reals
  const size_t sS = ((sreal * sizeof(R) + 15) / 16) * 16 / sizeof(V);
  V *S = reinterpret_cast<V *>(tw + ((ntw + 7) & ~7));
  V *A = S + sS;
  V *B = A + (size_t)LG * N;
  stage_table(tw, g.twx, ntw);
  const LineMap lm = line_map(LG);
  const int nrows = g.P[1] * g.P[2];
  const int ntiles = (nrows + RB - 1) / RB;
  R *Sr = reinterpret_cast<R *>(S);
  auto load = [&](int tile) {
    const int row0 = tile * RB;
    for (int rr = 0; rr < RB; rr++) {
      const int row = row0 + rr;
      if (row >= nrows) break;
      const int y = row % g.P[1], z = row / g.P[1];
      const R *src = in + (((size_t)(z + g.off[2]) * g.ext[1] + (y + g.off[1])) * g.ext[0] + g.off[0]) * cs;
      R *dst = Sr + (size_t)rr * P0 * NC;
      if (vec16) {
        const int nch = (P0 * NC * (int)sizeof(R)) / 16;
        for (int c = threadIdx.x; c < nch; c += blockDim.x)
          cp_async16(reinterpret_cast<char *>(dst) + 16 * c, reinterpret_cast<const char *>(src) + 16 * c);
      } else {
        for (int e = threadIdx.x; e < P0 * NC; e += blockDim.x) {
          const int x = e / NC, c = e - x * NC;
          if (sizeof(R) == 8) cp_async8(dst + e, src + (size_t)x * cs + c);
          else cp_async4(dst + e, src + (size_t)x * cs + c);
        }
      }
    }
    cp_async_commit();
  };
  int tile = blockIdx.x;
  if (tile < ntiles) load(tile);
  for (; tile < ntiles; tile += gridDim.x) {
    cp_async_wait_all();
    __syncthreads();
    const int row0 = tile * RB;
    // pack the staged reals into complex lines
    for (int t = threadIdx.x; t < RB * N; t += blockDim.x) {
      const int rr = t / N, m = t - rr * N;
      const R *xr = Sr + (size_t)rr * P0 * NC;
      const int x0 = 2 * m, x1 = 2 * m + 1;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const R a = (x0 < P0 && row0 + rr < nrows) ? xr[x0 * NC + c] : R(0);
        const R b = (x1 < P0 && row0 + rr < nrows) ? xr[x1 * NC + c] : R(0);
        line_set(A, m * L + rr * NC + c, mk(a, b));
      }
    }
    __syncthreads();
    const int next = tile + gridDim.x;
    if (next < ntiles) load(next);
    V *res = vfft_chain<false, R>(A, A, B, LG, sd, tw, lm, NoHook());
    const C *W = tw + sd.extoff;  // exp(-2 pi i k / Mx), k < H
    constexpr int XG = sizeof(R) == 4 ? 2 : 1;
    const int nkv = g.Hp / XG;
    for (int t = threadIdx.x; t < RB * nkv; t += blockDim.x) {
      const int rr = t / nkv, kv = t - rr * nkv;
      const int row = row0 + rr;
      if (row >= nrows) continue;
      C o[XG][NC];
#pragma unroll
      for (int h = 0; h < XG; h++) {
        const int k = kv * XG + h;
        if (k < g.H) {
          const int kk = (k == N) ? 0 : k;
          const int km = (k == 0 || k == N) ? 0 : N - k;
          const C w = W[k];
#pragma unroll
          for (int c = 0; c < NC; c++) {
            const C zk = line_at(res, kk * L + rr * NC + c);
            const C zn = cconj(line_at(res, km * L + rr * NC + c));
            const C a = cadd(zk, zn), bb = csub(zk, zn);
            const C wb = cmul(w, bb);
            o[h][c] = mk(R(0.5) * (a.x + wb.y), R(0.5) * (a.y - wb.x));  // (a - i W^k b) / 2
          }
        } else {
#pragma unroll
          for (int c = 0; c < NC; c++) o[h][c] = mk(R(0), R(0));
        }
      }
#pragma unroll
      for (int c = 0; c < NC; c++) spec_put<R>(X, spec_vec<R, NC>(g, row, kv * NC + c), o[0][c], o[XG - 1][c]);
    }
    __syncthreads();
  }
  cp_async_wait_all();
}

// ---------------------------------------------------------------- x inverse (C2R)
template <typename R, int NC>
__global__ void __launch_bounds__(PASS_THREADS, 1) k_xinv(SolveGeom<R> g, const typename cplx_t<R>::type *__restrict__ X,
                                                           R *__restrict__ outp, int RB, int cs) {
  typedef typename cplx_t<R>::type C;
  typedef typename Vec<R>::V V;
  constexpr int G = Vec<R>::G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftDesc sd;
  if (threadIdx.x == 0) sd = g.fx;
  const int ntw = g.fx.ntw + g.fx.next;
  C *tw = reinterpret_cast<C *>(smem_raw);
  const int N = g.N2, L = NC * RB, LG = L / G;
  const size_t rowc = (size_t)g.Hp * NC;  // complex per X row
  const size_t sS = (RB * rowc * sizeof(C)) / sizeof(V);
  V *S = reinterpret_cast<V *>(tw + ((ntw + 7) & ~7));
  V *A = S + sS;
  V *B = A + (size_t)LG * N;
  stage_table(tw, g.twx, ntw);
  const LineMap lm = line_map(LG);
  const int nrows = g.P[1] * g.P[2];
  const int ntiles = (nrows + RB - 1) / RB;
  C *Sc = reinterpret_cast<C *>(S);
  auto load = [&](int tile) {
    const int row0 = tile * RB;
    const int nr = min(RB, nrows - row0);
    const int rch = (int)(rowc * sizeof(C) / 16);  // 16-byte vectors of a row
    for (int c = threadIdx.x; c < nr * rch; c += blockDim.x) {
      const int rr = c / rch, v = c - rr * rch;
      cp_async16(reinterpret_cast<char *>(Sc) + 16 * (size_t)c,
                 reinterpret_cast<const char *>(X) + 16 * spec_vec<R, NC>(g, row0 + rr, v));
    }
    cp_async_commit();
  };
  int tile = blockIdx.x;
  if (tile < ntiles) load(tile);
  for (; tile < ntiles; tile += gridDim.x) {
    cp_async_wait_all();
    __syncthreads();
    const int row0 = tile * RB;
    const C *W = tw + sd.extoff;
    for (int t = threadIdx.x; t < RB * N; t += blockDim.x) {
      const int rr = t / N, m = t - rr * N;
      const C w = cconj(W[m]);
      const bool ok = row0 + rr < nrows;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        C z = mk(R(0), R(0));
        if (ok) {
          C xm = spec_get<R, NC>(Sc + rr * rowc, m, c);
          C xn = spec_get<R, NC>(Sc + rr * rowc, N - m, c);
          if (m == 0) {
            xm.y = R(0);
            xn.y = R(0);
          }  // DC and Nyquist are real
          const C a = cadd(xm, cconj(xn));
          const C b = csub(xm, cconj(xn));
          const C wb = cmul(w, b);
          z = mk(a.x - wb.y, a.y + wb.x);  // a + i W^{-m} b
        }
        line_set(A, m * L + rr * NC + c, z);
      }
    }
    __syncthreads();
    const int next = tile + gridDim.x;
    if (next < ntiles) load(next);
    V *res = vfft_chain<true, R>(A, A, B, LG, sd, tw, lm, NoHook());
    for (int t = threadIdx.x; t < RB * N; t += blockDim.x) {
      const int rr = t / N, m = t - rr * N;
      const int row = row0 + rr;
      if (row >= nrows) continue;
      const int y = row % g.P[1], z = row / g.P[1];
      R *dst = outp + (((size_t)(z + g.off[2]) * g.ext[1] + (y + g.off[1])) * g.ext[0] + g.off[0]) * cs;
      const int x0 = 2 * m, x1 = 2 * m + 1;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const C v = line_at(res, m * L + rr * NC + c);
        if (x0 < g.P[0]) dst[(size_t)x0 * cs + c] = v.x;
        if (x1 < g.P[0]) dst[(size_t)x1 * cs + c] = v.y;
      }
    }
    __syncthreads();
  }
  cp_async_wait_all();
}

// ---------------------------------------------------------------- periodic ghosts
// ghost fill after the inverse transform (source/fourier/pmlib_fourier_ifft.f:247-253):
// along a periodic axis the ghosts copy the interior one period away.
// ghost point t of the (ngl + ngh) x e[o1] x e[o2] strips along `axis`
template <typename R>
__device__ __forceinline__ void ghost_fill_point(R *__restrict__ mesh, int ex, int ey, int ez, int nv, int axis, int N,
                                                 int ngl, int ngh, long long t) {
  const int e[3] = {ex, ey, ez};
  const int ng = ngl + ngh;
  const int o1 = axis == 0 ? 1 : 0, o2 = axis == 2 ? 1 : 2;
  const int s = (int)(t % ng);
  const long long r = t / ng;
  const int a = (int)(r % e[o1]), b = (int)(r / e[o1]);
  int dstc = (s < ngl) ? s : ngl + N + (s - ngl);
  int srcc = (s < ngl) ? dstc + N : dstc - N;
  int id[3], is[3];
  id[o1] = a; id[o2] = b; id[axis] = dstc;
  is[o1] = a; is[o2] = b; is[axis] = srcc;
  const size_t di = (((size_t)id[2] * ey + id[1]) * ex + id[0]) * nv;
  const size_t si = (((size_t)is[2] * ey + is[1]) * ex + is[0]) * nv;
  for (int c = 0; c < nv; c++) mesh[di + c] = mesh[si + c];
}

template <typename R>
__global__ void k_ghost_fill(R *__restrict__ mesh, int ex, int ey, int ez, int nv, int axis, int N,
                             int ngl, int ngh) {
  const int e[3] = {ex, ey, ez};
  const int o1 = axis == 0 ? 1 : 0, o2 = axis == 2 ? 1 : 2;
  const long long total = (long long)(ngl + ngh) * e[o1] * e[o2];
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x)
    ghost_fill_point<R>(mesh, ex, ey, ez, nv, axis, N, ngl, ngh, t);
}

// All periodic ghosts of a mesh in one launch: every point of a periodic axis's ghost strips
// copies its image in the interior of all periodic axes, which is what filling the axes in
// turn leaves there (a point in two strips is written twice, with the same value).
struct GhostAll {
  int ext[3], per[3], n[3], ngl[3], ngh[3], nv;
  long long first[4];  // strip points of axes 0, 1, 2 in one index space
};
template <typename R> __global__ void k_ghost_fill_all(GhostAll q, R *__restrict__ mesh) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < q.first[3];
       t += (long long)gridDim.x * blockDim.x) {
    const int axis = t >= q.first[2] ? 2 : t >= q.first[1] ? 1 : 0;
    long long r = t - q.first[axis];
    int id[3];
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const int len = e == axis ? q.ngl[e] + q.ngh[e] : q.ext[e];
      const long long d = r / len;
      id[e] = (int)(r - d * len);
      r = d;
      if (e == axis && id[e] >= q.ngl[e]) id[e] += q.n[e];
    }
    size_t di = 0, si = 0;
#pragma unroll
    for (int e = 2; e >= 0; e--) {
      int i = id[e];
      if (q.per[e]) i += i < q.ngl[e] ? q.n[e] : i >= q.ngl[e] + q.n[e] ? -q.n[e] : 0;
      di = di * q.ext[e] + id[e];
      si = si * q.ext[e] + i;
    }
    for (int c = 0; c < q.nv; c++) mesh[di * q.nv + c] = mesh[si * q.nv + c];
  }
}

// the ghost fill along one axis of every patch of a batch that is periodic there:
// patch i's ghost points are items [first, first + total) of one index space
struct GhostDesc {
  long long first, total;
  int patch, ext[3], nv, N, ngl, ngh;
};
template <typename R>
__global__ void k_ghost_fill_batch(const GhostDesc *__restrict__ d, int npatch, long long total, int axis,
                                   BatchIo io) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = npatch - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (d[mid].first <= t) lo = mid;
      else hi = mid - 1;
    }
    const GhostDesc &q = d[lo];
    ghost_fill_point<R>((R *)io.p[q.patch], q.ext[0], q.ext[1], q.ext[2], q.nv, axis, q.N, q.ngl, q.ngh,
                        t - q.first);
  }
}

}  // namespace pmgpu
