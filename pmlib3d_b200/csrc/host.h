// host.h -- host-side declarations shared by the library's translation units:
// error reporting, launch accounting and per-kernel timing, and the FFT pass
// launchers that are compiled in their own units (passes_*.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "../../include/pmlib_gpu.h"
#include "common.cuh"
#include "solve.cuh"

namespace pmgpu {

enum KClass { KC_BIN, KC_SCAN, KC_PLACE, KC_FIXUP, KC_DEPOSIT, KC_GADD, KC_XFWD, KC_YFWD, KC_ZPASS, KC_YINV,
              KC_XINV, KC_GFILL, KC_M2P, KC_DERIV, KC_ADVANCE, KC_MAP, KC_OTHER, KC_N };

// brackets one launch with CUDA events on its stream while timing is enabled
struct KTimer {
  int cls;
  cudaStream_t st;
  cudaEvent_t a = nullptr, b = nullptr;
  KTimer(int c, cudaStream_t s);
  ~KTimer();
};

#define CK(expr, caller)                         \
  do {                                           \
    if (!::pmgpu::cuda_ok((expr), (caller))) {   \
      return -1;                                 \
    }                                            \
  } while (0)
#define CKL(caller) CK(cudaGetLastError(), caller)

int num_sms();
// Raises a kernel's maximum dynamic shared memory to `bytes` if it is below: the
// attribute only grows, and it is set at most once per size increase and device, so
// launches of the same kernel on other streams are not held up by setting it again.
int smem_attr(const void *func, size_t bytes, const char *caller);

// shared-memory budget of one persistent pass CTA
constexpr size_t PASS_SMEM_BUDGET = 220 * 1024;

// shared memory of a line-pass CTA with four and with two CTAs on an SM (228 KB an SM, of
// which 1 KB a CTA is the system's)
constexpr size_t LINE_SMEM_4 = 56 * 1024;
constexpr size_t LINE_SMEM_2 = 113 * 1024;
// shared memory the batched kernels keep for their own bookkeeping (the patch
// descriptor copy and the chunk counter), taken off the per-CTA budgets so that as
// many CTAs fit on an SM as in the passes of a single plan
constexpr size_t BATCH_SMEM_SLACK = 3 * 1024;
// A line tile takes its whole kx block (rows of 192 bytes) if its `bytes` of shared memory
// fit: on two CTAs an SM for Bluestein and the z pass of a single plan, which spend their
// time on the transforms, else on four; longer y lines take half of it (three CTAs an SM)
constexpr bool line_whole_block(size_t bytes, bool two_ctas) {
  return bytes <= (two_ctas ? LINE_SMEM_2 : LINE_SMEM_4);
}

static inline size_t tw_bytes(int ntw, size_t csize) { return (size_t)((ntw + 7) & ~7) * csize; }

// kx tile of the Stockham y / z passes: the largest of 8 (FP32), 4, 2, 1 (FP64) whose
// three buffers fit (FP32 vectors hold two neighbouring kx)
static inline int pick_tk(int n, int nc, size_t csize, int ntw) {
  for (int tk = csize == 8 ? 8 : 4; tk >= 1; tk /= 2) {  // within a kx block
    if (csize == 8 && tk % 2) continue;
    if (tw_bytes(ntw, csize) + 3 * (size_t)nc * tk * n * csize <= PASS_SMEM_BUDGET) return tk;
  }
  return 0;
}
static inline size_t lines_smem(int n, int nc, int tk, size_t csize, int ntw) {
  return tw_bytes(ntw, csize) + 3 * (size_t)nc * tk * n * csize;
}
// shared memory of a line pass: the plan's tables and one tile of TK kx lines of nc
// components (FP32: 16-byte vectors of two lines, or single lines for TK = 1)
static inline size_t line_smem(const LinePlan &p, int nc, int tk, size_t rsize) {
  const size_t csize = 2 * rsize, w = rsize == 4 && tk > 1 ? 16 : csize;
  return line_tab_bytes(p, w, csize) + (size_t)nc * tk * plan_points(p) * csize;
}
// shared memory of an x pass of rb rows a tile; pairs: FP32 vectors of two rows
static inline size_t x_smem(const LinePlan &p, int N, int H, int P0, int nc, int rb, size_t rsize, bool pairs,
                            bool inverse) {
  const size_t csize = 2 * rsize, w = pairs ? 16 : csize;
  const size_t rows = ((size_t)rb * 8 + 15) & ~(size_t)15;
  const size_t stage = rows + (inverse ? rows : (((size_t)rb * P0 * nc * rsize + 15) & ~(size_t)15));
  return x_tab_bytes(p, N, H, w, csize) + stage + (size_t)nc * rb * plan_points(p) * csize;
}

// rows per tile of the x passes
static inline int pick_rb(int n2, int P0, int Hp, int nc, size_t csize, size_t rsize, int ntw, bool inverse) {
  for (int rb = 8; rb >= 1; rb--) {
    if (csize == 8 && (nc * rb) % 2) continue;
    const size_t stage = inverse ? (size_t)rb * Hp * nc * csize : (((size_t)rb * P0 * nc * rsize + 15) / 16) * 16;
    if (tw_bytes(ntw, csize) + stage + 2 * (size_t)nc * rb * n2 * csize <= PASS_SMEM_BUDGET) return rb;
  }
  return 0;
}

// ---- batches of patches: one launch per pass family (x forward, y forward, z pass,
// y inverse, x inverse) over the tiles of every patch, then the periodic ghost fill
// per axis.  The descriptors are built on the host once (batch_layout) and live in
// device memory; a solve passes the patches' arrays by value (BatchIo).
struct BatchPart {
  size_t desc_off = 0;  // byte offset of the part's descriptors
  int npatch = 0, nitems = 0, chunk = 1;
  size_t smem = 0;
};
struct BatchPassInfo {
  BatchPart part[2];  // the patches with a compile-time plan, and the others
};
struct BatchGhostInfo {
  size_t desc_off;
  int npatch;
  long long total;
};
struct BatchLayout {
  int npatch = 0;
  BatchPassInfo pass[5];
  BatchGhostInfo ghost[3];
  size_t bytes = 0;  // descriptor bytes
};

// ---- FFT passes (passes.cuh, instantiated per precision and component count)
// x then y forward: real cuboid (component stride cs) -> X -> Y
template <typename R, int NC>
int fwd_xy(SolveGeom<R> &g, const R *in, typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y, cudaStream_t st,
           const char *caller, int cs = NC);
template <typename R, int NC>
int even_forward(SolveGeom<R> &g, const R *in, typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y,
                 typename cplx_t<R>::type *Z, cudaStream_t st, const char *caller);
// periodic ghosts of a mesh of nv components
template <typename R>
int ghost_fill_all(const pmgpu_topo *topo, R *mesh, int nv, cudaStream_t st, const char *caller);
// z pass on rows_y spectrum rows: Z_VEL / Z_VORT / Z_VECPOT / Z_REGULARISE / Z_FORWARD
template <typename R, int NC>
int zpass(SolveGeom<R> &g, const typename cplx_t<R>::type *in, typename cplx_t<R>::type *out, int mode, int reproj,
          int use_zeta, int rows_y, cudaStream_t st, const char *caller);
// y then x inverse into the cuboid (periodic ghosts filled when `ghosts`)
template <typename R, int NC>
int inv_yx(SolveGeom<R> &g, const pmgpu_topo *topo, typename cplx_t<R>::type *Y, typename cplx_t<R>::type *X, R *out,
           cudaStream_t st, const char *caller, int cs = NC, bool ghosts = true);

// fills `desc` (host bytes) and `lay` for the velocity solve of n patches of
// geometries g[i] with work spectra X[i], Y[i] (run_solve's layout); -1 if a patch
// needs a pass the batched kernels do not run (the Stockham fallback)
template <typename R, int NC>
int batch_layout(int n, const SolveGeom<R> *g, typename cplx_t<R>::type *const *X,
                 typename cplx_t<R>::type *const *Y, const pmgpu_topo *const *topo, std::vector<unsigned char> &desc,
                 BatchLayout &lay, const char *caller);
// queues the batched solve: d_desc holds the descriptors; counters: BATCH_COUNTERS words, two
// parts a pass family, cleared here
constexpr int BATCH_COUNTERS = 10;
template <typename R, int NC>
int batch_launch(const BatchLayout &lay, const void *d_desc, unsigned *counters, const void *const *vort,
                 void *const *vel, cudaStream_t st, const char *caller);
// one pass along y (forward X -> Y, or inverse Y -> X)
template <typename R, int NC>
int ypass(SolveGeom<R> &g, const typename cplx_t<R>::type *X, typename cplx_t<R>::type *Y, int inverse,
          cudaStream_t st, const char *caller);

// whether the passes of a plain velocity solve (x forward, y forward, z, y inverse, x inverse)
// run kernels compiled for their plan
template <typename R, int NC> void compiled_passes(const SolveGeom<R> &g, int compiled[5]);

// each pass unit holds its own copy of the DFT constant tables
int upload_cs_f32_1(const void *t32, const void *t64);
int upload_cs_f32_3(const void *t32, const void *t64);
int upload_cs_f64_1(const void *t32, const void *t64);
int upload_cs_f64_3(const void *t32, const void *t64);
int upload_cs_x_f32_3(const void *t32, const void *t64);
int upload_cs_x_f32_1(const void *t32, const void *t64);
int upload_cs_x_f32_s(const void *t32, const void *t64);
int upload_cs_x_f32_b(const void *t32, const void *t64);
int upload_cs_x_f64(const void *t32, const void *t64);
int upload_cs_x_f64_b(const void *t32, const void *t64);
int upload_cs_ct_yf_f32(const void *t32, const void *t64);
int upload_cs_ct_yi_f32(const void *t32, const void *t64);
int upload_cs_ct_z_f32(const void *t32, const void *t64);
int upload_cs_ct_x_f32(const void *t32, const void *t64);
int upload_cs_ct_yf_f64(const void *t32, const void *t64);
int upload_cs_ct_yi_f64(const void *t32, const void *t64);
int upload_cs_ct_z_f64(const void *t32, const void *t64);
int upload_cs_ct_x_f64(const void *t32, const void *t64);
int upload_cs_ct_xb_f32(const void *t32, const void *t64);
int upload_cs_ct_xb_f64(const void *t32, const void *t64);
int upload_cs_lines_f32(const void *t32, const void *t64);
int upload_cs_lines_f32b(const void *t32, const void *t64);
int upload_cs_lines_f64(const void *t32, const void *t64);
int upload_cs_lines_f64b(const void *t32, const void *t64);

// launches of the y / z line passes take a compile-time-plan kernel when one is
// compiled for the plan and kx tile (0: always the run-time engine)
extern int g_fft_ct;

}  // namespace pmgpu
