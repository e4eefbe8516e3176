// passes.cuh -- host launchers of the FFT passes of the solve (x forward + y
// forward, the fused z pass, y inverse + x inverse).  Included by the pass units
// passes_*.cu, each of which instantiates them for one precision and component
// count, so the heavy kernels compile in parallel.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>

#include "kernels.cuh"

namespace pmgpu {

template <typename K> static int persistent_grid(K kernel, size_t smem, int ntiles) {
  int per = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, PASS_THREADS, smem) != cudaSuccess || per < 1) per = 1;
  return std::max(1, std::min(ntiles, per * num_sms()));
}


// Tile and CTA of a register-engine line pass along `axis`, within `slack` bytes less than
// the shared memory (tk = 0: the pass takes the Stockham path).
struct LineShape {
  int tk, threads;
};
// Threads of a CTA with sm bytes of shared memory whose phases have `tasks` work items: the
// multiple of 32 that keeps the most threads of an SM busy, counting the idle ones of a
// phase's last round.  An SM holds 512 threads of 128 registers.  Loads pass through the L1
// that the shared memory leaves, so three or more CTAs share at most 196 KB (256^3, y
// forward, tiles of 55 KB: four CTAs of 128 threads 409 us, three of 160 298 us).
static inline int pass_threads(size_t sm, const double *tasks, int n) {
  const size_t cta = sm + 1024;
  int most = (int)(196 * 1024 / cta);
  if (most < 3) most = std::min<int>(2, std::max<int>(1, (int)(228 * 1024 / cta)));
  int best = 256;
  double top = 0.0;
  for (int t = 96; t <= 256; t += 32) {
    const int ctas = std::min(most, 512 / t);
    double work = 0.0, spent = 0.0;
    for (int i = 0; i < n; i++) {
      work += tasks[i];
      spent += std::ceil(tasks[i] / t) * t;
    }
    const double busy = ctas * t * work / spent;
    if (busy > top * 1.001) {
      top = busy;
      best = t;
    }
  }
  return best;
}
// of a line pass of plan pl with lg vectors a position; of an x pass, with its twist
static inline int line_threads(const LinePlan &pl, int lg, size_t sm, double twist = 0.0) {
  double tasks[LP_MAX + 1];
  int n = 0;
  for (int p = 0; p < pl.np; p++)
    tasks[n++] = (double)lg * (p == 0 && pl.split ? pl.n : plan_points(pl)) / pl.rad[p];
  if (twist > 0.0) tasks[n++] = twist;
  return pass_threads(sm, tasks, n);
}
template <typename R, int NC>
static LineShape line_shape(const SolveGeom<R> &g, int axis, size_t slack) {
  if (!(axis == 1 ? g.ry_ok : g.rz_ok)) return LineShape{0, 0};
  const LinePlan &pl = axis == 1 ? g.ly : g.lz;
  const int tuned = axis == 1 ? g.tky : g.tkz;
  const int top = spec_block<R>();  // tiles lie within a kx block
  auto bytes = [&](int tk) { return line_smem(pl, NC, tk, sizeof(R)) + slack; };
  auto shape = [&](int tk) {
    const int lg = NC * tk / (sizeof(R) == 4 && tk > 1 ? 2 : 1);
    return LineShape{tk, line_threads(pl, lg, bytes(tk))};
  };
  if (tuned > 0 && tuned <= top && bytes(tuned) <= PASS_SMEM_BUDGET) return shape(tuned);
  if (line_whole_block(bytes(top), (axis == 2 || pl.bl) && slack == 0)) return shape(top);
  for (size_t budget : {LINE_SMEM_2, PASS_SMEM_BUDGET})
    if (bytes(top / 2) <= budget) return shape(top / 2);
  for (int tk = top / 4; tk >= 1; tk /= 2)
    if (bytes(tk) <= PASS_SMEM_BUDGET) return shape(tk);
  return LineShape{0, 0};
}

// Rows of a tile and CTA of a register-engine x pass (rb = 0: the Stockham path): at most
// 12 vectors a point (as the line tiles), four CTAs of 128 threads an SM if the tile
// fits, else two of 256, else one; single FP32 rows when no pair of rows fits.
struct XShape {
  int rb, threads;
  bool pairs;
};
// rows: all rows of the launch.
template <typename R, int NC>
static XShape x_shape(const SolveGeom<R> &g, bool inverse, size_t slack, long long rows) {
  if (!g.rx_ok) return XShape{0, 0, false};
  auto bytes = [&](int rb, bool pairs) {
    return x_smem(g.lx, g.N2, g.H, g.P[0], NC, rb, sizeof(R), pairs, inverse) + slack;
  };
  const bool f32 = sizeof(R) == 4;
  // rows shorter than those of the compile-time plans: more of them, to fill the CTA, while
  // that leaves two tiles an SM.  Solves in microseconds, always four times the rows / so many:
  // 16^3 fff FP32 50.7 / 40.3, 40 x 40 x 40 ppf 57 / 47, 20 x 48 x 48 pff 61 / 56
  int most = f32 ? 8 : 4;
  for (int i = 0; i < 2 && plan_points(g.lx) < 32 && rows >= 2 * (2 * most) * (long long)num_sms(); i++) most *= 2;
  for (size_t budget : {LINE_SMEM_4, LINE_SMEM_2, PASS_SMEM_BUDGET})
    for (int rb = most; rb >= (budget == PASS_SMEM_BUDGET ? (f32 ? 2 : 1) : most / 2); rb /= 2)
      if (bytes(rb, f32) <= budget)
        return XShape{rb, line_threads(g.lx, NC * rb / (f32 ? 2 : 1), bytes(rb, f32), (double)g.Hp * NC * rb / (f32 ? 4 : 1)),
                      f32};
  if (f32 && bytes(1, false) <= PASS_SMEM_BUDGET) return XShape{1, 256, false};
  return XShape{0, 0, false};
}

// fills the periodic ghosts of a mesh of nv components.  One launch while every periodic
// axis has at least as many cells as ghosts on a side (an image is then an interior
// cell), else one an axis.  Bound by launches and by the strips' short runs: velocity of
// 512 x 512 x 256, two axes periodic, 29.9 us an axis at a time, 23.3 in one; velocity and
// vorticity of a 64^3 reprojection 30.6 / 20.8.
template <typename R>
int ghost_fill_all(const pmgpu_topo *topo, R *mesh, int nv, cudaStream_t st, const char *caller) {
  GhostAll q;
  memset(&q, 0, sizeof(q));
  q.nv = nv;
  bool any = false, one = true;
  for (int e = 0; e < 3; e++) {
    q.n[e] = topo->ncell[e];
    q.ngl[e] = topo->nghost[2 * e];
    q.ngh[e] = topo->nghost[2 * e + 1];
    q.ext[e] = q.n[e] + q.ngl[e] + q.ngh[e];
    q.per[e] = topo->bound_cond[2 * e] != 0 && topo->bound_cond[2 * e + 1] != 0;
    any = any || q.per[e];
    one = one && (!q.per[e] || (q.n[e] >= q.ngl[e] && q.n[e] >= q.ngh[e]));
  }
  if (!any) return 0;
  for (int e = 0; e < 3; e++) {
    const long long strip = q.per[e] ? (long long)(q.ngl[e] + q.ngh[e]) * q.ext[(e + 1) % 3] * q.ext[(e + 2) % 3] : 0;
    q.first[e + 1] = q.first[e] + strip;
    if (one || strip == 0) continue;
    const int nblk = (int)std::min<long long>((strip + 255) / 256, 148 * 16);
    { KTimer kt_(KC_GFILL, st);
      k_ghost_fill<R><<<std::max(nblk, 1), 256, 0, st>>>(mesh, q.ext[0], q.ext[1], q.ext[2], nv, e, q.n[e], q.ngl[e], q.ngh[e]); }
    PM_LAUNCHED();
    CKL(caller);
  }
  if (one && q.first[3] > 0) {
    const int nblk = (int)std::min<long long>((q.first[3] + 255) / 256, 148 * 16);
    KTimer kt_(KC_GFILL, st);
    k_ghost_fill_all<R><<<nblk, 256, 0, st>>>(q, mesh);
    PM_LAUNCHED();
    CKL(caller);
  }
  return 0;
}

// the tiles of a line pass over the spectral arrays X (P1 rows a plane) and Y (M1 rows):
// y forward X -> Y, y inverse Y -> X, and along z (rows_y spectrum rows, rows_out z rows out)
template <typename R> static LineTiles line_tiles(const SolveGeom<R> &g, int axis, int lmode, int rows_y, int rows_out) {
  const long long Hp = g.Hp, B = spec_block<R>(), P1 = g.P[1], M1 = g.M[1];
  LineTiles lt;
  memset(&lt, 0, sizeof(lt));
  lt.n = g.M[axis];
  if (axis == 1) {
    const bool fwd = lmode == L_FWD;
    lt.rows_in = fwd ? g.P[1] : g.M[1];
    lt.rows_out = fwd ? g.M[1] : g.P[1];
    lt.in_os = (fwd ? P1 : M1) * Hp;
    lt.out_os = (fwd ? M1 : P1) * Hp;
    lt.in_kb = (fwd ? P1 : M1) * B;
    lt.out_kb = (fwd ? M1 : P1) * B;
    lt.in_rs = lt.out_rs = B;
    lt.nouter = g.P[2];
  } else {
    lt.rows_in = g.P[2];
    lt.rows_out = rows_out;
    lt.in_os = lt.out_os = B;
    lt.in_kb = lt.out_kb = M1 * B;
    lt.in_rs = lt.out_rs = M1 * Hp;
    lt.nouter = rows_y;
    lt.ofast = 1;  // neighbouring tiles are neighbours in memory
  }
  return lt;
}

// The kernel of a register-engine line pass of shape sh; compiled: one of its plan's own.
template <typename R, int NC>
static LinesKernel<R> pick_lines(const SolveGeom<R> &g, int axis, int lmode, int zmode, int use_zeta, const LineShape &sh,
                                 bool &compiled) {
  const bool pairs = sizeof(R) == 4 && sh.tk > 1;
  LinesKernel<R> kern = nullptr;
  if constexpr (NC == 3) {
    const bool plain = lmode != L_Z || (zmode == Z_VEL && z_plain(g, use_zeta));
    if (g_fft_ct && plain && (pairs || sizeof(R) == 8))
      kern = lines_kernel_ct<R>(lmode, axis == 1 ? g.ly : g.lz, NC * sh.tk / (pairs ? 2 : 1));
  }
  compiled = kern != nullptr;
  return compiled ? kern : lines_kernel<R>(pairs);
}
// The kernels of register-engine x passes, the same way.
template <typename R, int NC> static RxfKernel<R> pick_xfwd(const SolveGeom<R> &g, const XShape &sh, bool &compiled) {
  RxfKernel<R> kern = nullptr;
  if constexpr (NC == 3)
    if (g_fft_ct && (sh.pairs || sizeof(R) == 8)) kern = rxfwd_kernel_ct<R>(g.lx, NC * sh.rb / (sh.pairs ? 2 : 1));
  compiled = kern != nullptr;
  return compiled ? kern : rxfwd_kernel<R, NC>(sh.pairs);
}
template <typename R, int NC> static RxiKernel<R> pick_xinv(const SolveGeom<R> &g, const XShape &sh, bool &compiled) {
  RxiKernel<R> kern = nullptr;
  if constexpr (NC == 3)
    if (g_fft_ct && (sh.pairs || sizeof(R) == 8)) kern = rxinv_kernel_ct<R>(g.lx, NC * sh.rb / (sh.pairs ? 2 : 1));
  compiled = kern != nullptr;
  return compiled ? kern : rxinv_kernel<R, NC>(sh.pairs);
}

template <typename R, int NC> void compiled_passes(const SolveGeom<R> &g, int compiled[5]) {
  const long long rows = (long long)g.P[1] * g.P[2];
  bool c[5] = {false, false, false, false, false};
  for (int inv = 0; inv < 2; inv++) {
    const XShape sh = x_shape<R, NC>(g, inv != 0, 0, rows);
    if (sh.rb > 0 && inv) pick_xinv<R, NC>(g, sh, c[4]);
    else if (sh.rb > 0) pick_xfwd<R, NC>(g, sh, c[0]);
  }
  for (int f = 1; f <= 3; f++) {
    const int axis = f == 2 ? 2 : 1;
    const LineShape sh = line_shape<R, NC>(g, axis, 0);
    if (sh.tk > 0) pick_lines<R, NC>(g, axis, f == 1 ? L_FWD : f == 2 ? L_Z : L_INV, Z_VEL, 0, sh, c[f]);
  }
  for (int f = 0; f < 5; f++) compiled[f] = c[f];
}

template <typename R, int NC>
static int launch_lines(SolveGeom<R> &g, const typename cplx_t<R>::type *in, typename cplx_t<R>::type *out, int axis,
                        int lmode, int zmode, int reproj, int use_zeta, const LineTiles &tiles, cudaStream_t st,
                        const char *caller) {
  typedef typename cplx_t<R>::type C;
  const int n = g.M[axis];
  const LineShape sh = line_shape<R, NC>(g, axis, 0);
  if (sh.tk > 0) {
    const LinePlan &pl = axis == 1 ? g.ly : g.lz;
    const bool pairs = sizeof(R) == 4 && sh.tk > 1;
    LineTiles lt = tiles;
    lt.nkt = g.Hp / sh.tk;
    lt.TK = sh.tk;
    lt.dLG = make_fastdiv((unsigned)(NC * sh.tk / (pairs ? 2 : 1)));
    const size_t sm = line_smem(pl, NC, sh.tk, sizeof(R));
    bool compiled;
    const LinesKernel<R> kern = pick_lines<R, NC>(g, axis, lmode, zmode, use_zeta, sh, compiled);
    if (smem_attr((const void *)kern, sm, caller)) return -1;
    int per = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, sh.threads, sm) != cudaSuccess || per < 1) per = 1;
    const int grid = std::max(1, std::min(lt.nouter * lt.nkt, per * num_sms()));
    kern<<<grid, sh.threads, sm, st>>>(g, lt, in, out, NC, axis, lmode, zmode, reproj, use_zeta);
    PM_LAUNCHED();
    CKL(caller);
    return 0;
  }
  const int ntw = (axis == 1) ? g.fy.ntw : g.fz.ntw;
  const int TK = pick_tk(n, NC, sizeof(C), ntw);
  if (TK == 0) {
    set_error(caller, "FFT length too large for the shared-memory transform.");
    return -1;
  }
  LineTiles lt = tiles;
  lt.nkt = g.Hp / TK;
  lt.TK = TK;
  lt.ofast = 0;
  const size_t sm = lines_smem(n, NC, TK, sizeof(C), ntw);
  if (smem_attr((const void *)k_lines<R, NC>, sm, caller)) return -1;
  const int grid = persistent_grid(k_lines<R, NC>, sm, lt.nouter * lt.nkt);
  k_lines<R, NC><<<grid, PASS_THREADS, sm, st>>>(g, lt, in, out, axis, lmode, zmode, reproj, use_zeta);
  PM_LAUNCHED();
  CKL(caller);
  return 0;
}

// x forward: real cuboid (component stride cs) -> X
template <typename R, int NC>
static int xfwd(SolveGeom<R> &g, const R *in, typename cplx_t<R>::type *X, cudaStream_t st, const char *caller, int cs) {
  typedef typename cplx_t<R>::type C;
  const bool vec16r = cs == NC && ((size_t)g.ext[0] * NC * sizeof(R)) % 16 == 0 &&
                      ((size_t)g.off[0] * NC * sizeof(R)) % 16 == 0 && ((size_t)g.P[0] * NC * sizeof(R)) % 16 == 0;
  const XShape sh = x_shape<R, NC>(g, false, 0, (long long)g.P[1] * g.P[2]);
  if (sh.rb > 0) {
    const size_t sm = x_smem(g.lx, g.N2, g.H, g.P[0], NC, sh.rb, sizeof(R), sh.pairs, false);
    auto launch = [&](auto kern, int G) -> int {
      if (smem_attr((const void *)kern, sm, caller)) return -1;
      const int ntiles = (g.P[1] * g.P[2] + sh.rb - 1) / sh.rb;
      int per = 1;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, sh.threads, sm) != cudaSuccess || per < 1) per = 1;
      const int grid = std::max(1, std::min(ntiles, per * num_sms()));
      KTimer kt_(KC_XFWD, st);
      kern<<<grid, sh.threads, sm, st>>>(g, in, X, sh.rb, cs, vec16r ? 1 : 0, make_fastdiv((unsigned)(NC * sh.rb / G)));
      PM_LAUNCHED();
      CKL(caller);
      return 0;
    };
    bool compiled;
    if (launch(pick_xfwd<R, NC>(g, sh, compiled), sh.pairs ? 2 : 1)) return -1;
    return 0;
  }
  const int ntwx = g.fx.ntw + g.fx.next;
  const int RB = pick_rb(g.N2, g.P[0], g.Hp, NC, sizeof(C), sizeof(R), ntwx, false);
  if (RB == 0) {
    set_error(caller, "FFT length too large for the shared-memory transform.");
    return -1;
  }
  const size_t stage = (((size_t)RB * g.P[0] * NC * sizeof(R) + 15) / 16) * 16;
  const size_t sm = tw_bytes(ntwx, sizeof(C)) + stage + 2 * (size_t)NC * RB * g.N2 * sizeof(C);
  const bool vec16 = cs == NC && ((size_t)g.ext[0] * NC * sizeof(R)) % 16 == 0 &&
                     ((size_t)g.off[0] * NC * sizeof(R)) % 16 == 0 && ((size_t)g.P[0] * NC * sizeof(R)) % 16 == 0;
  if (smem_attr((const void *)k_xfwd<R, NC>, sm, caller)) return -1;
  const int rows = g.P[1] * g.P[2];
  const int ntiles = (rows + RB - 1) / RB;
  { KTimer kt_(KC_XFWD, st);
    k_xfwd<R, NC><<<persistent_grid(k_xfwd<R, NC>, sm, ntiles), PASS_THREADS, sm, st>>>(g, in, X, RB, cs, vec16 ? 1 : 0); }
  PM_LAUNCHED();
  CKL(caller);
  return 0;
}

template <typename R, int NC>
int fwd_xy(SolveGeom<R> &g, const R *in, typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y,
           cudaStream_t st, const char *caller, int cs) {
  if (xfwd<R, NC>(g, in, X, st, caller, cs)) return -1;
  KTimer kt_(KC_YFWD, st);
  return launch_lines<R, NC>(g, X, Y, 1, L_FWD, 0, 0, 0, line_tiles(g, 1, L_FWD, 0, 0), st, caller);
}

// Transform of a real sequence even in y and z (M1 / 2 + 1 rows of M2 / 2 + 1 planes of M0 reals
// in `in`): x on those rows, y on those planes with the other rows read from their mirror
// -> Y, z the same way for the spectrum rows of ky <= M1 / 2 -> Z (M2 planes).  Needs the
// register engine on every axis.
template <typename R, int NC>
int even_forward(SolveGeom<R> &g, const R *in, typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y,
                 typename cplx_t<R>::type *Z, cudaStream_t st, const char *caller) {
  SolveGeom<R> h = g;
  for (int e = 1; e < 3; e++) h.ext[e] = h.P[e] = g.M[e] / 2 + 1;
  if (xfwd<R, NC>(h, in, X, st, caller, NC)) return -1;
  LineTiles ty = line_tiles(h, 1, L_FWD, 0, 0), tz = line_tiles(h, 2, L_Z, g.M[1], g.M[2]);
  ty.rows_in = g.M[1];
  tz.rows_in = g.M[2];
  ty.even = tz.even = 1;
  { KTimer kt_(KC_YFWD, st);
    if (launch_lines<R, NC>(g, X, Y, 1, L_FWD, 0, 0, 0, ty, st, caller)) return -1; }
  KTimer kt_(KC_ZPASS, st);
  return launch_lines<R, NC>(g, Y, Z, 2, L_FWD, Z_FORWARD, 0, 0, tz, st, caller);
}

// one forward (or inverse) pass along y over the X layout -> Y layout, as in fwd_xy
template <typename R, int NC>
int ypass(SolveGeom<R> &g, const typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y, int inverse,
          cudaStream_t st, const char *caller) {
  if (inverse)
    return launch_lines<R, NC>(g, Y, (typename cplx_t<R>::type *)X, 1, L_INV, 0, 0, 0, line_tiles(g, 1, L_INV, 0, 0), st,
                               caller);
  return launch_lines<R, NC>(g, X, Y, 1, L_FWD, 0, 0, 0, line_tiles(g, 1, L_FWD, 0, 0), st, caller);
}

template <typename R, int NC>
int zpass(SolveGeom<R> &g, const typename cplx_t<R>::type *in, typename cplx_t<R>::type *out, int mode,
                 int reproj, int use_zeta, int rows_y, cudaStream_t st, const char *caller) {
  // Z_FORWARD: forward transform only, P rows in (the rest zero), M rows out
  const int rows_out = (mode == Z_FORWARD) ? g.M[2] : g.P[2];
  KTimer kt_(KC_ZPASS, st);
  return launch_lines<R, NC>(g, in, out, 2, mode == Z_FORWARD ? L_FWD : L_Z, mode, reproj, use_zeta,
                             line_tiles(g, 2, L_Z, rows_y, rows_out), st, caller);
}

template <typename R, int NC>
int inv_yx(SolveGeom<R> &g, const pmgpu_topo *topo, typename cplx_t<R>::type *Y,
           typename cplx_t<R>::type *X, R *out, cudaStream_t st, const char *caller, int cs, bool ghosts) {
  typedef typename cplx_t<R>::type C;
  {
    KTimer kt_(KC_YINV, st);
    if (launch_lines<R, NC>(g, Y, X, 1, L_INV, 0, 0, 0, line_tiles(g, 1, L_INV, 0, 0), st, caller))
      return -1;
  }
  const int rows = g.P[1] * g.P[2];
  const XShape sh = x_shape<R, NC>(g, true, 0, rows);
  if (sh.rb > 0) {
    const size_t sm = x_smem(g.lx, g.N2, g.H, g.P[0], NC, sh.rb, sizeof(R), sh.pairs, true);
    auto launch = [&](auto kern, int G) -> int {
      if (smem_attr((const void *)kern, sm, caller)) return -1;
      const int ntiles = (rows + sh.rb - 1) / sh.rb;
      int per = 1;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, sh.threads, sm) != cudaSuccess || per < 1) per = 1;
      const int grid = std::max(1, std::min(ntiles, per * num_sms()));
      KTimer kt_(KC_XINV, st);
      kern<<<grid, sh.threads, sm, st>>>(g, X, out, sh.rb, cs, make_fastdiv((unsigned)(NC * sh.rb / G)));
      PM_LAUNCHED();
      CKL(caller);
      return 0;
    };
    bool compiled;
    if (launch(pick_xinv<R, NC>(g, sh, compiled), sh.pairs ? 2 : 1)) return -1;
  } else {
    const int ntwx = g.fx.ntw + g.fx.next;
    const int RB = pick_rb(g.N2, g.P[0], g.Hp, NC, sizeof(C), sizeof(R), ntwx, true);
    if (RB == 0) {
      set_error(caller, "FFT length too large for the shared-memory transform.");
      return -1;
    }
    const size_t sm =
        tw_bytes(ntwx, sizeof(C)) + (size_t)RB * g.Hp * NC * sizeof(C) + 2 * (size_t)NC * RB * g.N2 * sizeof(C);
    if (smem_attr((const void *)k_xinv<R, NC>, sm, caller)) return -1;
    const int ntiles = (rows + RB - 1) / RB;
    { KTimer kt_(KC_XINV, st);
      k_xinv<R, NC><<<persistent_grid(k_xinv<R, NC>, sm, ntiles), PASS_THREADS, sm, st>>>(g, X, out, RB, cs); }
    PM_LAUNCHED();
    CKL(caller);
  }
  return ghosts ? ghost_fill_all<R>(topo, out, cs, st, caller) : 0;
}


// ---------------------------------------------------------------- batches of patches
template <typename R, int NC>
int batch_layout(int n, const SolveGeom<R> *g, typename cplx_t<R>::type *const *X,
                 typename cplx_t<R>::type *const *Y, const pmgpu_topo *const *topo, std::vector<unsigned char> &desc,
                 BatchLayout &lay, const char *caller) {
  typedef typename cplx_t<R>::type C;
  static_assert(sizeof(PassDesc<R>) + 64 <= BATCH_SMEM_SLACK, "descriptor copy exceeds the reserved shared memory");
  if (n <= 0 || n > BATCH_MAX) return -1;
  lay = BatchLayout();
  lay.npatch = n;
  std::vector<PassDesc<R>> all[5], d[5][2];  // by pass family, and by part of it
  std::vector<size_t> smem[5];
  auto add = [&](int f, int i, int cls, size_t sm, PassDesc<R> &q) {
    q.patch = i;
    q.cls = cls;
    all[f].push_back(q);
    smem[f].push_back(sm);
  };
  long long rows = 0;
  for (int i = 0; i < n; i++) rows += (long long)g[i].P[1] * g[i].P[2];
  std::vector<GhostDesc> gd[3];
  for (int i = 0; i < n; i++) {
    const SolveGeom<R> &gi = g[i];
    if (!gi.rx_ok || !gi.ry_ok || !gi.rz_ok) return -1;
    // x forward and x inverse (rows per tile as the single-plan passes, within the slack)
    for (int inv = 0; inv < 2; inv++) {
      const int f = inv ? 4 : 0;
      const XShape sh = x_shape<R, NC>(gi, inv != 0, BATCH_SMEM_SLACK, rows);
      if (sh.rb <= 0 || sh.pairs != (sizeof(R) == 4)) return -1;
      const int RB = sh.rb;
      const size_t sm = x_smem(gi.lx, gi.N2, gi.H, gi.P[0], NC, RB, sizeof(R), sh.pairs, inv != 0);
      PassDesc<R> q;
      memset(&q, 0, sizeof(q));
      q.g = gi;
      q.RB = RB;
      q.cs = NC;
      q.vec16 = ((size_t)gi.ext[0] * NC * sizeof(R)) % 16 == 0 && ((size_t)gi.off[0] * NC * sizeof(R)) % 16 == 0 &&
                ((size_t)gi.P[0] * NC * sizeof(R)) % 16 == 0;
      q.dLG = make_fastdiv((unsigned)(NC * RB / (sizeof(R) == 4 ? 2 : 1)));
      q.in = inv ? X[i] : nullptr;   // x forward reads the caller's vorticity
      q.out = inv ? nullptr : X[i];  // x inverse writes the caller's velocity
      q.ntiles = (gi.P[1] * gi.P[2] + RB - 1) / RB;
      const int lg = NC * RB / (sizeof(R) == 4 ? 2 : 1);
      add(f, i, g_fft_ct ? rx_batch_class<R>(gi.lx, lg) : 0, sm, q);
    }
    // y forward, z pass, y inverse (run_solve's launch_lines arguments)
    for (int f = 1; f <= 3; f++) {
      const int axis = f == 2 ? 2 : 1;
      const LineShape sh = line_shape<R, NC>(gi, axis, BATCH_SMEM_SLACK);
      const int TK = sh.tk;
      if (TK <= (sizeof(R) == 4 ? 1 : 0)) return -1;
      const LinePlan &pl = axis == 1 ? gi.ly : gi.lz;
      PassDesc<R> q;
      memset(&q, 0, sizeof(q));
      q.g = gi;
      LineTiles &lt = q.lt;
      lt = line_tiles(gi, axis, f == 3 ? L_INV : f == 2 ? L_Z : L_FWD, gi.M[1], gi.P[2]);
      lt.TK = TK;
      lt.nkt = gi.Hp / TK;
      lt.dLG = make_fastdiv((unsigned)(NC * TK / (sizeof(R) == 4 ? 2 : 1)));
      q.in = f == 1 ? X[i] : Y[i];
      q.out = f == 3 ? X[i] : Y[i];
      q.ntiles = lt.nouter * lt.nkt;
      const int lmode = f == 3 ? L_INV : f == 2 ? L_Z : L_FWD, lg = NC * TK / (sizeof(R) == 4 ? 2 : 1);
      const bool plain = f != 2 || z_plain(gi, 0);
      add(f, i, g_fft_ct && plain ? lines_batch_class<R>(lmode, pl, lg) : 0, line_smem(pl, NC, TK, sizeof(R)), q);
    }
    // periodic ghosts of the velocity (x, then y, then z)
    for (int a = 0; a < 3; a++) {
      const pmgpu_topo *t = topo[i];
      if (t->bound_cond[2 * a] == 0 || t->bound_cond[2 * a + 1] == 0) continue;
      GhostDesc q;
      memset(&q, 0, sizeof(q));
      q.patch = i;
      for (int e = 0; e < 3; e++) q.ext[e] = gi.ext[e];
      q.nv = NC;
      q.N = t->ncell[a];
      q.ngl = t->nghost[2 * a];
      q.ngh = t->nghost[2 * a + 1];
      q.total = (long long)(q.ngl + q.ngh) * gi.ext[(a + 1) % 3] * gi.ext[(a + 2) % 3];
      q.first = lay.ghost[a].total;
      lay.ghost[a].total += q.total;
      gd[a].push_back(q);
    }
  }
  // A patch goes to the part of its plan.  A family whose tiles all fit on the GPU at once runs
  // as one part, of run-time plans: its time is that of a tile, and a second launch adds
  // another.  Microseconds, two parts / one: 2 patches of up to 64 cells 84 / 66, of up to 40
  // 93 / 83; with four tiles an SM for the limit 12 patches 224 / 228
  for (int f = 0; f < 5; f++) {
    long long items = 0, compiled = 0;
    for (const PassDesc<R> &q : all[f]) {
      items += q.ntiles;
      if (q.cls) compiled += q.ntiles;
    }
    const bool one = compiled < items && items <= 3ll * num_sms();
    for (size_t k = 0; k < all[f].size(); k++) {
      PassDesc<R> &q = all[f][k];
      if (one) q.cls = 0;
      BatchPart &bp = lay.pass[f].part[q.cls ? 0 : 1];
      q.first = bp.nitems;
      bp.nitems += q.ntiles;
      bp.npatch++;
      bp.smem = std::max(bp.smem, smem[f][k]);
      d[f][q.cls ? 0 : 1].push_back(q);
    }
  }
  // chunks of work items: about eight per CTA slot of the GPU
  size_t off = 0;
  for (int f = 0; f < 5; f++)
    for (int k = 0; k < 2; k++) {
      BatchPart &bp = lay.pass[f].part[k];
      bp.desc_off = off;
      off += sizeof(PassDesc<R>) * bp.npatch;
      off = (off + 255) & ~(size_t)255;
      const int slots = num_sms() * 3;
      bp.chunk = std::max(1, std::min(16, bp.nitems / (8 * slots)));
    }
  for (int a = 0; a < 3; a++) {
    lay.ghost[a].desc_off = off;
    lay.ghost[a].npatch = (int)gd[a].size();
    off += sizeof(GhostDesc) * gd[a].size();
    off = (off + 255) & ~(size_t)255;
  }
  lay.bytes = off;
  desc.assign(off, 0);
  for (int f = 0; f < 5; f++)
    for (int k = 0; k < 2; k++)
      if (!d[f][k].empty())
        memcpy(desc.data() + lay.pass[f].part[k].desc_off, d[f][k].data(), sizeof(PassDesc<R>) * d[f][k].size());
  for (int a = 0; a < 3; a++)
    if (!gd[a].empty()) memcpy(desc.data() + lay.ghost[a].desc_off, gd[a].data(), sizeof(GhostDesc) * gd[a].size());
  return 0;
}

template <typename R, int NC>
int batch_launch(const BatchLayout &lay, const void *d_desc, unsigned *counters, const void *const *vort,
                 void *const *vel, cudaStream_t st, const char *caller) {
  const int n = lay.npatch;
  BatchIo vin, vout;
  memset(&vin, 0, sizeof(vin));
  memset(&vout, 0, sizeof(vout));
  for (int i = 0; i < n; i++) {
    vin.p[i] = vort[i];
    vout.p[i] = vel[i];
  }
  CK(cudaMemsetAsync(counters, 0, BATCH_COUNTERS * sizeof(unsigned), st), caller);
  const char *base = reinterpret_cast<const char *>(d_desc);
  // one part of a pass family; a family's patches differ in their phases: four CTAs of 128
  // threads where they fit
  auto launch = [&](auto kern, int f, int k, auto... args) -> int {
    const BatchPart &bp = lay.pass[f].part[k];
    if (bp.npatch == 0) return 0;
    BatchWork bw;
    bw.desc = base + bp.desc_off;
    bw.npatch = bp.npatch;
    bw.nitems = bp.nitems;
    bw.chunk = bp.chunk;
    bw.pad = 0;
    bw.counter = counters + 2 * f + k;
    const size_t cta = bp.smem + BATCH_SMEM_SLACK + 1024;
    const int threads = 4 * cta <= 196 * 1024 ? 128 : 3 * cta <= 196 * 1024 ? 160 : 256;
    if (smem_attr((const void *)kern, bp.smem, caller)) return -1;
    int per = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, bp.smem) != cudaSuccess || per < 1) per = 1;
    const int grid = std::max(1, std::min(bp.nitems, per * num_sms()));
    kern<<<grid, threads, bp.smem, st>>>(bw, args...);
    PM_LAUNCHED();
    CKL(caller);
    return 0;
  };
  auto lines = [&](int f, int axis, int lmode, int zmode) -> int {
    return launch(lines_batch_ct<R>(lmode), f, 0) || launch(lines_batch_kernel<R>(), f, 1, axis, lmode, zmode) ? -1 : 0;
  };
  auto xpass = [&](int f, bool inverse, const BatchIo &io) -> int {
    return launch(rx_batch_ct<R>(inverse), f, 0, io) || launch(rx_batch_kernel<R>(inverse), f, 1, io) ? -1 : 0;
  };
  { KTimer kt_(KC_XFWD, st); if (xpass(0, false, vin)) return -1; }
  { KTimer kt_(KC_YFWD, st); if (lines(1, 1, L_FWD, 0)) return -1; }
  { KTimer kt_(KC_ZPASS, st); if (lines(2, 2, L_Z, Z_VEL)) return -1; }
  { KTimer kt_(KC_YINV, st); if (lines(3, 1, L_INV, 0)) return -1; }
  { KTimer kt_(KC_XINV, st); if (xpass(4, true, vout)) return -1; }
  for (int a = 0; a < 3; a++) {
    if (lay.ghost[a].npatch == 0) continue;
    const long long total = lay.ghost[a].total;
    const int nblk = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    const GhostDesc *gd = reinterpret_cast<const GhostDesc *>(base + lay.ghost[a].desc_off);
    { KTimer kt_(KC_GFILL, st);
      k_ghost_fill_batch<R><<<std::max(nblk, 1), 256, 0, st>>>(gd, lay.ghost[a].npatch, total, a, vout); }
    PM_LAUNCHED();
    CKL(caller);
  }
  return 0;
}

}  // namespace pmgpu

#define PMGPU_INSTANTIATE_PASSES(R, NC, NAME)                                                                  \
  namespace pmgpu {                                                                                            \
  template int fwd_xy<R, NC>(SolveGeom<R> &, const R *, cplx_t<R>::type *, cplx_t<R>::type *, cudaStream_t,    \
                             const char *, int);                                                               \
  template int zpass<R, NC>(SolveGeom<R> &, const cplx_t<R>::type *, cplx_t<R>::type *, int, int, int, int,    \
                            cudaStream_t, const char *);                                                       \
  template int inv_yx<R, NC>(SolveGeom<R> &, const pmgpu_topo *, cplx_t<R>::type *, cplx_t<R>::type *, R *,    \
                             cudaStream_t, const char *, int, bool);                                           \
  template int even_forward<R, NC>(SolveGeom<R> &, const R *, cplx_t<R>::type *, cplx_t<R>::type *,             \
                                   cplx_t<R>::type *, cudaStream_t, const char *);                              \
  template int ypass<R, NC>(SolveGeom<R> &, const cplx_t<R>::type *, cplx_t<R>::type *, int, cudaStream_t,      \
                            const char *);                                                                     \
  int upload_cs_##NAME(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }                 \
  }

#define PMGPU_INSTANTIATE_BATCH(R, NC)                                                                         \
  namespace pmgpu {                                                                                            \
  template int ghost_fill_all<R>(const pmgpu_topo *, R *, int, cudaStream_t, const char *);                    \
  template void compiled_passes<R, NC>(const SolveGeom<R> &, int[5]);                                          \
  template int batch_layout<R, NC>(int, const SolveGeom<R> *, cplx_t<R>::type *const *,                        \
                                   cplx_t<R>::type *const *, const pmgpu_topo *const *,                        \
                                   std::vector<unsigned char> &, BatchLayout &, const char *);                 \
  template int batch_launch<R, NC>(const BatchLayout &, const void *, unsigned *, const void *const *,          \
                                   void *const *, cudaStream_t, const char *);                                 \
  }
