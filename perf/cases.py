"""The framework's work as timed cases: the particle-mesh vortex step and the calls around it.

A case is one of

* ``step``   -- P2M, unbounded solve with curl, M2P on device particles (``pmlib.step_dev``)
* ``stage``  -- one Runge-Kutta stage of the vortex client (``pmlib.vortex_stage_dev``)
* ``solve``  -- a mesh solve alone, plain or with reprojection (``pmlib.pmlib_poisson_solve_dev``)
* ``batch``  -- independent patches of uneven sizes in one call (``pmlib.Batch``)
* ``setup``  -- a plan for a grid not seen before, one solve with it, and its release (a served
  request of a new grid)
* ``host``   -- the step on host arrays, as the Fortran module calls it (``pmlib.step``)

Sizes follow the configurations of the repository's benchmark and tests: the 64^3 and 256^3 ring
steps, the 512 x 512 x 256 periodic-periodic-free step, 96 patches with 32 to 192 cells a side, and
ragged boxes.  ``adjust`` grows the free axes by ``pmlib_patch_adjust`` as the reference's programs
do; without it the grid is taken as given and its transform lengths may hold large primes.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pmlib3d_b200 import pmlib as P

H = 1.0 / 128  # cell size (a power of two: box sides are exact)
NG = 4         # ghost cells of free faces
DTYPES = {"f32": (torch.float32, P.FP32), "f64": (torch.float64, P.FP64)}


def _step(name, n, bc, dtype, order=6, interp=3, adjust=False, jitter=0.1, fill="all", kind="step"):
    c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "bc": bc, "dtype": dtype, "order": order,
         "interp": interp, "adjust": adjust, "jitter": jitter, "fill": fill}
    return {"name": name, **c} if name else c


def _solve(name, n, bc, dtype, reproj, adjust, order=6, kind="solve"):
    c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "bc": bc, "dtype": dtype, "order": order,
         "reproj": reproj, "adjust": adjust}
    return {"name": name, **c} if name else c


def _batch(name, count, nmin, nmax, sizes):
    c = {"kind": "batch", "count": count, "nmin": nmin, "nmax": nmax, "sizes": sizes}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the 64^3 single-ring step: the smallest grid in use, bound by launches and latency
        _step("step64_f32", (64, 64, 64), "fff", "f32"),
        # the headline 256^3 two-ring step in the FP32 form ...
        _step("step256_f32", (256, 256, 256), "fff", "f32"),
        # ... and on the FP64 plain path, the drop-in
        _step("step256_f64", (256, 256, 256), "fff", "f64"),
        # the large periodic-periodic-free step, 67 M particles
        _step("step_ppf512_f32", (512, 512, 256), "ppf", "f32"),
        # a ragged box taken as given (transform lengths 150, 242 and 190 = 2 5 19), M6*, particles
        # anywhere in their cells as after some steps without remeshing
        _step("step_ragged_m6_f32", (150, 113, 87), "pff", "f32", interp=4, jitter=0.499),
        # after a truncated remeshing only the vortex cores hold particles
        _step("step_cores_f32", (192, 160, 176), "fff", "f32", adjust=True, fill="cores"),
        # one stage of the client's RK3 step on an adjusted grid, double precision
        _step("stage_f64", (96, 96, 128), "fff", "f64", adjust=True, kind="stage"),
        # ... and in FP32 on a larger one
        _step("stage_f32", (184, 184, 184), "fff", "f32", adjust=True, kind="stage"),
        # a solve with reprojection of the vorticity (every remeshing step of the clients)
        _solve("solve_reproj_f32", (160, 96, 128), "ppf", "f32", True, True),
        # 96 uneven patches, the batched workload
        _batch("batch96_f32", 96, 32, 192, 3),
        # a served request of a new grid: its plan, one solve, release
        _solve("new_grid_f32", (120, 88, 72), "fff", "f32", False, True, kind="setup"),
        # the Fortran-side call on host arrays
        _step("host64_f64", (64, 64, 64), "fff", "f64", kind="host"),
    ]


def _cells_drawn(rng, lo, hi, most, bc):
    while True:
        n = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        n = [c + c % 2 if b == "p" else c for c, b in zip(n, bc)]
        if n[0] * n[1] * n[2] <= most:
            return tuple(n)


def draw(rng: random.Random):
    kind = rng.choices(["step", "stage", "solve", "batch", "setup", "host"], [10, 3, 4, 2, 2, 1])[0]
    bc = rng.choice(["fff", "fff", "ppf", "pff", "ppp"])
    dtype = rng.choice(["f32", "f32", "f32", "f64"])
    adjust = rng.random() < 0.6
    order = rng.choice([6, 6, 6, 2, 4, 8, 10])
    most = {"f32": 12_000_000, "f64": 6_000_000}[dtype]
    if kind in ("step", "stage", "host"):
        hi = 96 if kind == "host" else 400
        n = _cells_drawn(rng, 32, hi, most, bc)
        return _step("", n, bc, dtype, order, rng.choice([3, 3, 3, 4]), adjust, rng.choice([0.1, 0.499]),
                     "cores" if kind == "step" and rng.random() < 0.3 else "all", kind)
    if kind == "batch":
        return _batch("", rng.randint(8, 96), 32, rng.randint(64, 192), rng.randrange(1 << 20))
    n = _cells_drawn(rng, 32, 300, most if kind == "solve" else most // 2, bc)
    if kind == "setup":
        bc = rng.choice(["fff", "ppf", "pff"])
        n = tuple(c + c % 2 if b == "p" else c for c, b in zip(n, bc))
        return _solve("", n, bc, dtype, False, True, order, kind="setup")
    return _solve("", n, bc, dtype, rng.random() < 0.5, adjust, order)


# ---------------------------------------------------------------- grids and inputs
def _grid(n, bc, adjust):
    """Cells per axis (grown as pmlib_patch_adjust grows them) and the low corner."""
    n = [c + 16 - (c + 2 * NG) % 16 if adjust and b == "f" else c for c, b in zip(n, bc)]
    return n, [-0.5 * c * H for c in n]


def _case_grid(case):
    return _grid((case["nx"], case["ny"], case["nz"]), case["bc"], case["adjust"])


def _patch(n, bc, adjust, interp):
    """Patch and cuboid topology through the framework's own calls."""
    half = [0.5 * c * H for c in n]
    pa = P.make_patch([-x for x in half], half, (H, H, H), bound_cond=[int(b == "p") for b in bc], nghost=NG)
    if adjust and P.pmlib_patch_adjust(pa) != 0:
        raise RuntimeError(P.last_error())
    ierr, t = P.pmlib_topology_cuboid(pa, interp)
    if ierr != 0:
        raise RuntimeError(P.last_error())
    return pa, t


def _plan(pa, t, order, interp, precision):
    ierr, plan = P.pmlib_poisson_setup(pa, t, P.make_params(order=order, kernel=1, radius=2.0, interp=interp),
                                       precision)
    if ierr != 0:
        raise RuntimeError(P.last_error())
    return plan


def _rings(x, y, z, n, bc):
    """Two coaxial vortex rings of opposite circulation, about z where x and y are periodic, else about x."""
    L = min(n) * H
    R, sigma, off = 0.25 * L, 0.04 * L, 0.1 * L
    out = torch.zeros((*torch.broadcast_shapes(x.shape, y.shape, z.shape), 3), dtype=torch.float64, device="cuda")
    a, b, c = (x, y, z) if bc[:2] == "pp" else (y, z, x)  # the ring axis is c
    rho = torch.sqrt(a * a + b * b)
    rs = torch.where(rho > 0, rho, torch.ones_like(rho))
    ia, ib = (0, 1) if bc[:2] == "pp" else (1, 2)
    for s, c0 in ((1.0, -off), (-1.0, off)):
        d2 = (rho - R) ** 2 + (c - c0) ** 2
        w = torch.where(d2 < 16 * sigma * sigma, s * torch.exp(-d2 / (sigma * sigma)), torch.zeros_like(d2))
        out[..., ia] -= w * b / rs
        out[..., ib] += w * a / rs
    return out


def _particles(case, seed):
    """One particle a cell in remeshing order (x fastest), jittered; rings and 1 % noise (FP64)."""
    n, lo = _case_grid(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    ax = [lo[e] + (torch.arange(n[e], dtype=torch.float64, device="cuda") + 0.5) * H for e in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    pos = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], -1)
    del x, y, z
    if case["fill"] == "cores":
        w = _rings(pos[:, 0], pos[:, 1], pos[:, 2], n, case["bc"])
        pos = pos[w.square().sum(-1) > 1e-6].contiguous()
        del w
    pos += (2.0 * torch.rand(pos.shape, dtype=torch.float64, device="cuda", generator=g) - 1.0) * (case["jitter"] * H)
    vort = _rings(pos[:, 0], pos[:, 1], pos[:, 2], n, case["bc"])
    vort += 0.01 * torch.randn(vort.shape, dtype=torch.float64, device="cuda", generator=g)
    dt = DTYPES[case["dtype"]][0]
    return pos.to(dt).contiguous(), vort.to(dt).contiguous()


def _mesh_field(n, lo, bc, seed, dtype, interp=3):
    """A smooth random vorticity with 1 % noise on the cuboid (ghosts included), (nz', ny', nx', 3); the periodic
    ghosts repeat the interior."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    gp = 2 if interp == 3 else 3
    gh = [gp if b == "p" else NG for b in bc]
    idx = [torch.arange(-gh[e], n[e] + gh[e], device="cuda") for e in range(3)]
    idx = [torch.remainder(i, n[e]) if bc[e] == "p" else i + gh[e] for e, i in enumerate(idx)]
    m = [n[e] if bc[e] == "p" else n[e] + 2 * NG for e in range(3)]
    x, y, z = (lo[e] + (torch.arange(m[e], device="cuda", dtype=torch.float64) + (0.5 if bc[e] == "p" else 0.5 - NG)) * H
               for e in range(3))
    w = _rings(x[None, None, :], y[None, :, None], z[:, None, None], n, bc)
    amp = 0.5 + torch.rand(3, dtype=torch.float64, device="cuda", generator=g)
    w = w * amp + 0.01 * torch.randn(w.shape, dtype=torch.float64, device="cuda", generator=g)
    w = w[idx[2]][:, idx[1]][:, :, idx[0]]
    return w.to(dtype).contiguous()


def _batch_specs(case):
    """(cells, boundary types, blob axis) of the batch's patches: cells log-uniform, even where periodic."""
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case["count"]):
        bc = r.choice(["fff", "ppf", "pff"])
        n = [int(round(math.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]))))) for _ in range(3)]
        out.append(([c + c % 2 if b == "p" else c for c, b in zip(n, bc)], bc, r.randrange(3)))
    return out


def _blobs(case, seed):
    """The batch's vorticity fields in one flat array (a blob a patch, scaled from the seed) and their slices."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    specs = _batch_specs(case)
    amp = 0.5 + torch.rand(len(specs), dtype=torch.float64, device="cuda", generator=g)
    parts, where, at = [], [], 0
    for i, (n0, bc, axis) in enumerate(specs):
        n, lo = _grid(n0, bc, True)
        gh = [2 if b == "p" else NG for b in bc]
        x, y, z = (lo[e] + (torch.arange(-gh[e], n[e] + gh[e], device="cuda", dtype=torch.float64) + 0.5) * H
                   for e in range(3))
        r2 = x[None, None, :] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2
        f = torch.zeros((*r2.shape, 3), dtype=torch.float32, device="cuda")
        f[..., axis] = (amp[i] * torch.exp(-r2 / (0.2 * max(n) * H) ** 2)).float()
        size = -(-f.numel() // 64) * 64  # 256-byte aligned slices
        parts.append(torch.nn.functional.pad(f.reshape(-1), (0, size - f.numel())))
        where.append((at, tuple(f.shape)))
        at += size
    return torch.cat(parts), where


def prepare(case, seed):
    k = case["kind"]
    if k == "batch":
        vort, where = _blobs(case, seed)
        vel = torch.zeros_like(vort)
        pts = [_patch(n, bc, True, 3) for n, bc, _ in _batch_specs(case)]
        b = P.Batch([p for p, _ in pts], [t for _, t in pts], P.make_params(order=6, kernel=1, radius=2.0, interp=3),
                    P.FP32)
        return {"kind": k, "batch": b, "vort": vort, "vel": vel, "stream": torch.cuda.Stream(),
                "wp": [vort.data_ptr() + 4 * at for at, _ in where], "up": [vel.data_ptr() + 4 * at for at, _ in where]}
    dt, prec = DTYPES[case["dtype"]]
    n, lo = _case_grid(case)
    interp = case.get("interp", 3)
    pa, t = _patch((case["nx"], case["ny"], case["nz"]), case["bc"], case["adjust"], interp)
    s = {"kind": k, "order": case["order"], "prec": prec, "patch": pa, "topo": t, "interp": interp}
    if k in ("solve", "setup"):
        s["vort"] = _mesh_field(n, lo, case["bc"], seed, dt, interp)
        s["vel"] = torch.zeros_like(s["vort"])
        s["reproj"] = case["reproj"]
        if k == "solve":
            s["plan"] = _plan(pa, t, case["order"], interp, prec)
        return s
    s["plan"] = _plan(pa, t, case["order"], interp, prec)
    pos, vort = _particles(case, seed)
    if k == "host":
        s["pos"], s["vort"] = pos.cpu().numpy(), vort.cpu().numpy()
        s["vel"] = np.zeros_like(s["pos"])
        return s
    s["n"] = pos.shape[0]
    s["pos"], s["vort"], s["vel"] = pos, vort, torch.zeros_like(pos)
    if k == "stage":
        s["dvort"], s["vel_rk"], s["dvort_rk"] = (torch.zeros_like(pos) for _ in range(3))
    return s


STAGE_DT, STAGE_VISC = 0.02, 1e-4  # CFL about 0.02 for these rings


def _ok(ierr):
    if ierr != 0:
        raise RuntimeError(P.last_error())


def run(s):
    k = s["kind"]
    if k == "step":
        _ok(P.step_dev(s["plan"], s["pos"].data_ptr(), s["vort"].data_ptr(), s["n"], s["vel"].data_ptr()))
        return s["vel"]
    if k == "stage":
        ierr, s["n"] = P.vortex_stage_dev(s["plan"], 3, 1, STAGE_DT, 4, STAGE_VISC, s["pos"].data_ptr(),
                                          s["vort"].data_ptr(), s["vel_rk"].data_ptr(), s["dvort_rk"].data_ptr(),
                                          s["n"], s["vel"].data_ptr(), s["dvort"].data_ptr())
        _ok(ierr)
        return {"npart": s["n"], **{a: s[a] for a in ("pos", "vort", "vel_rk", "dvort_rk", "vel", "dvort")}}
    if k == "solve":
        _ok(P.pmlib_poisson_solve_dev(s["plan"], s["vort"].data_ptr(), s["vel"].data_ptr(), reproj=s["reproj"]))
        return {"vel": s["vel"], "vort": s["vort"]} if s["reproj"] else s["vel"]
    if k == "batch":
        _ok(s["batch"].solve(s["wp"], s["up"], s["stream"].cuda_stream))
        return s["vel"]
    if k == "setup":
        plan = _plan(s["patch"], s["topo"], s["order"], s["interp"], s["prec"])
        _ok(P.pmlib_poisson_solve_dev(plan, s["vort"].data_ptr(), s["vel"].data_ptr()))
        plan.close()
        return s["vel"]
    _ok(P.step(s["plan"], s["pos"], s["vort"], s["vel"]))
    return s["vel"]


# ---------------------------------------------------------------- what a pass cannot do without
def _fft_flops(n, bc, fields):
    """Real transforms of `fields` scalar fields on the doubled grid."""
    M = [c if b == "p" else 2 * (c + 2 * NG) for c, b in zip(n, bc)]
    N = M[0] * M[1] * M[2]
    return fields * 2.5 * N * math.log2(N), N


def work(case):
    k = case["kind"]
    if k == "batch":
        by = fl = 0.0
        for n0, bc, _ in _batch_specs(case):
            n, _ = _grid(n0, bc, True)
            gh = [2 if b == "p" else NG for b in bc]
            cells = math.prod(c + 2 * g for c, g in zip(n, gh))
            f, N = _fft_flops(n, bc, 6)
            by += 6 * 4 * cells + 4 * N / 8
            fl += f
        return {"bytes": by, "flops": fl}
    w = 4 if case["dtype"] == "f32" else 8
    n, _ = _case_grid(case)
    bc = case["bc"]
    cells = math.prod(n)
    f, N = _fft_flops(n, bc, 6)
    green = 0 if bc == "ppp" or k == "setup" else w * N / 8
    if k in ("solve", "setup"):
        extra = 2 if case["reproj"] else 1
        return {"bytes": 3 * w * cells * (1 + extra) + green, "flops": f * (1 + extra) / 2}
    # the particles: lattice cells, or those of the cores (a tube of about 2.6 sigma around either ring)
    np_ = cells
    if case["fill"] == "cores":
        L = min(n) * H
        np_ = min(cells, 2 * (2 * math.pi * 0.25 * L) * math.pi * (2.63 * 0.04 * L) ** 2 / H ** 3)
    W = 4 if case["interp"] == 3 else 6
    if k == "stage":  # position, vorticity and both stage arrays in and out, velocity and right-hand side out
        return {"bytes": w * np_ * (4 * 6 + 6) + green, "flops": f + np_ * 18 * W ** 3 + cells * 90}
    return {"bytes": 9 * w * np_ + green, "flops": f + np_ * 12 * W ** 3}


# ---------------------------------------------------------------- the same in 64 bits, by torch alone
def _weights(d, interp):
    if interp == 3:
        a, b = d + 1, 2 - d
        inner = lambda t: 1 - 2.5 * t ** 2 + 1.5 * t ** 3  # noqa: E731
        outer = lambda t: 0.5 * (2 - t) ** 2 * (1 - t)  # noqa: E731
        return [outer(a), inner(d), inner(1 - d), outer(b)]
    w0 = lambda t: -(t - 1) * (25 * t ** 4 - 38 * t ** 3 - 3 * t ** 2 + 12 * t + 12) / 12  # noqa: E731
    w1 = lambda t: (t - 1) * (t - 2) * (25 * t ** 3 - 114 * t ** 2 + 153 * t - 48) / 24  # noqa: E731
    w2 = lambda t: -(t - 2) * (t - 3) ** 3 * (5 * t - 8) / 24  # noqa: E731
    return [w2(d + 2), w1(d + 1), w0(d), w0(1 - d), w1(2 - d), w2(3 - d)]


def _stencil(pos, n, lo, bc, interp):
    """Per axis: the cells (on the transform's input grid) and weights of every particle's stencil."""
    out = []
    for e in range(3):
        t = (pos[:, e].double() - lo[e]) / H
        b = torch.floor(t + 0.5)
        w = _weights(t - (b - 0.5), interp)
        off = 1 if interp == 3 else 2
        idx = []
        for s in range(len(w)):
            i = b.long() - off + s - 1  # cell 0 is the first interior one
            if bc[e] == "p":
                i = torch.remainder(i, n[e])
            else:
                i = i + NG
                m = n[e] + 2 * NG
                w[s] = torch.where((i >= 0) & (i < m), w[s], torch.zeros_like(w[s]))
                i = i.clamp(0, m - 1)
            idx.append(i)
        out.append((idx, w))
    return out


def _in_shape(n, bc):
    return [n[e] if bc[e] == "p" else n[e] + 2 * NG for e in (2, 1, 0)]


def _deposit(st, vort, shape):
    mesh = torch.zeros((shape[0] * shape[1] * shape[2], 3), dtype=torch.float64, device="cuda")
    v = vort.double()
    for kz, wz in zip(*st[2]):
        for ky, wy in zip(*st[1]):
            row, wyz = (kz * shape[1] + ky) * shape[2], wz * wy
            for kx, wx in zip(*st[0]):
                mesh.index_add_(0, row + kx, v * (wyz * wx)[:, None])
    return mesh.reshape(*shape, 3)


def _interpolate(st, mesh):
    shape, f = mesh.shape, mesh.reshape(-1, 3)
    out = torch.zeros((st[0][0][0].numel(), 3), dtype=torch.float64, device="cuda")
    for kz, wz in zip(*st[2]):
        for ky, wy in zip(*st[1]):
            row, wyz = (kz * shape[1] + ky) * shape[2], wz * wy
            for kx, wx in zip(*st[0]):
                out += f[row + kx] * (wyz * wx)[:, None]
    return out


def _green(n, bc, order, M):
    """Spectrum of the regularised Green's function (cell volume included), rfftn layout (z, y, x)."""
    eps = 2.0 * H
    ax = [torch.fft.fftfreq(M[e], 1.0 / M[e], dtype=torch.float64, device="cuda") * H for e in range(3)]
    poly = {2: [0.0], 4: [1.0], 6: [1.75, -0.25], 8: [2.375, -2.0 / 3, 1.0 / 24],
            10: [2.921875, -233.0 / 192, 29.0 / 192, -1.0 / 192]}[order]
    at0 = {2: 1.0, 4: 1.5, 6: 1.875, 8: 2.1875, 10: 2.4609375}[order] * math.sqrt(2.0) / (4 * math.pi ** 1.5 * eps)
    g = torch.zeros((M[2], M[1], M[0]), dtype=torch.float64, device="cuda")
    img = [(-1, 0, 1) if b == "p" else (0,) for b in bc]
    for iz in img[2]:
        for iy in img[1]:
            for ix in img[0]:
                for z0 in range(0, M[2], 64):
                    z = ax[2][z0:z0 + 64, None, None] + iz * n[2] * H
                    r = torch.sqrt((ax[0] + ix * n[0] * H) ** 2 + (ax[1][:, None] + iy * n[1] * H) ** 2 + z * z)
                    rho = r / eps
                    q = sum(c * rho ** (2 * i + 1) for i, c in enumerate(poly))
                    v = (q * torch.exp(-0.5 * rho * rho) / math.sqrt(2 * math.pi) +
                         torch.erf(rho / math.sqrt(2.0))) / (4 * math.pi * r)
                    g[z0:z0 + 64] += torch.where(r == 0, torch.full_like(v, at0), v)
    return torch.fft.rfftn(g).real * H ** 3


def _solve_exact(w, n, bc, order, reproj):
    """Velocity (and reprojected vorticity) of w (z, y, x, 3) on the transform's input grid."""
    M = [n[e] if bc[e] == "p" else 2 * (n[e] + 2 * NG) for e in range(3)]
    s = w.shape[:3]
    k = [torch.fft.rfftfreq(M[0], H, dtype=torch.float64, device="cuda")[None, None, :],
         torch.fft.fftfreq(M[1], H, dtype=torch.float64, device="cuda")[None, :, None],
         torch.fft.fftfreq(M[2], H, dtype=torch.float64, device="cuda")[:, None, None]]
    nyq = 0.5 / H * (1 - 1e-12)
    kc = [torch.where(a.abs() >= nyq, torch.zeros_like(a), a) for a in k]
    kn = [a - b for a, b in zip(k, kc)]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    zeta = None
    if reproj:
        s2 = (2 * math.pi * 2.0 * H) ** 2 * k2
        co = [1.0, 0.5, 0.125, 1.0 / 48, 1.0 / 384][:max(1, order // 2)]
        zeta = sum(c * s2 ** i for i, c in enumerate(co)) * torch.exp(-0.5 * s2)
    if bc == "ppp":
        one = torch.ones_like(k2) if zeta is None else zeta
        G = torch.where(k2 > 0, one / (4 * math.pi ** 2 * torch.where(k2 > 0, k2, torch.ones_like(k2))),
                        torch.zeros_like(k2))
    else:
        G = _green(n, bc, order, M)
    wh = [torch.fft.rfftn(w[..., c], s=(M[2], M[1], M[0])) for c in range(3)]
    back = lambda a: torch.fft.irfftn(a, s=(M[2], M[1], M[0]))[:s[0], :s[1], :s[2]]  # noqa: E731
    vel = torch.stack([back(2j * math.pi * G * (kc[(c + 1) % 3] * wh[(c + 2) % 3] - kc[(c + 2) % 3] * wh[(c + 1) % 3]))
                       for c in range(3)], -1)
    if not reproj:
        return vel, None
    d = sum(kc[c] * wh[c] for c in range(3))
    dn = sum(kn[c] * wh[c] for c in range(3))
    new = torch.stack([back(zeta * wh[c] - 4 * math.pi ** 2 * G * (kc[c] * d + kn[c] * dn)) for c in range(3)], -1)
    return vel, new


def _ghosts(f, n, bc, interp=3):
    """A field of the transform's input grid on the cuboid: periodic axes get their ghosts."""
    gp = 2 if interp == 3 else 3
    for e, dim in ((0, 2), (1, 1), (2, 0)):
        if bc[e] == "p":
            f = f.index_select(dim, torch.remainder(torch.arange(-gp, n[e] + gp, device="cuda"), n[e]))
    return f


def _rhs(w, u, bc):
    """visc lap(w) + (w . grad) u by fourth-order differences, zero outside the interior cells of free axes."""
    out = torch.zeros_like(w)
    for e, dim in ((0, 2), (1, 1), (2, 0)):
        sh = lambda f, m: torch.roll(f, -m, dim)  # noqa: E731
        out += STAGE_VISC * (-(sh(w, 2) + sh(w, -2)) / 12 + 4.0 / 3 * (sh(w, 1) + sh(w, -1)) - 2.5 * w) / H ** 2
        out += w[..., e:e + 1] * ((sh(u, -2) - sh(u, 2)) / 6 + 4.0 / 3 * (sh(u, 1) - sh(u, -1))) / (2 * H)
    for e, dim in ((0, 2), (1, 1), (2, 0)):
        if bc[e] == "f":
            out.narrow(dim, 0, NG).zero_()
            out.narrow(dim, out.shape[dim] - NG, NG).zero_()
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        vort, where = _blobs(case, seed)
        out = torch.zeros(vort.numel(), dtype=torch.float64, device="cuda")
        for (at, shape), (n0, bc, _) in zip(where, _batch_specs(case)):
            n, _ = _grid(n0, bc, True)
            size = math.prod(shape)
            w = vort[at:at + size].reshape(shape).double()
            for e, dim in ((0, 2), (1, 1), (2, 0)):
                if bc[e] == "p":
                    w = w.narrow(dim, 2, n[e])
            out[at:at + size] = _ghosts(_solve_exact(w, n, bc, 6, False)[0], n, bc).reshape(-1)
        return out
    n, lo = _case_grid(case)
    bc, interp = case["bc"], case.get("interp", 3)
    if k in ("solve", "setup"):
        w = _mesh_field(n, lo, bc, seed, DTYPES[case["dtype"]][0], interp).double()
        for e, dim in ((0, 2), (1, 1), (2, 0)):
            if bc[e] == "p":
                w = w.narrow(dim, 2 if interp == 3 else 3, n[e])
        vel, new = _solve_exact(w, n, bc, case["order"], case["reproj"])
        vel = _ghosts(vel, n, bc, interp)
        return vel if new is None else {"vel": vel, "vort": _ghosts(new, n, bc, interp)}
    pos, vort = _particles(case, seed)
    st = _stencil(pos, n, lo, bc, interp)
    w = _deposit(st, vort, _in_shape(n, bc))
    u, _ = _solve_exact(w, n, bc, case["order"], False)
    vel = _interpolate(st, u)
    if k != "stage":
        return vel.cpu().numpy() if k == "host" else vel
    dv = _interpolate(st, _rhs(w, u, bc))
    vrk, drk = STAGE_DT * vel, STAGE_DT * dv
    return {"npart": None, "pos": pos.double() + vrk / 3, "vort": vort.double() + drk / 3, "vel_rk": vrk, "dvort_rk": drk,
            "vel": vel, "dvort": dv}
