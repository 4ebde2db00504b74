"""The measured work of the framework: calls of its public entry points over the range its users meet.

A case names a padded grid (``nx, ny, nz`` voxels and absorbing layers of ``layer`` voxels per side on the axes in
``absorb``), a precision, a linear solver and a number of right-hand sides.  Inputs follow the framework's own
configurations: beads of index 1.36 to 1.60 in water, 500 nm light, 50 nm voxels, illumination directions inside an
NA 1.2 cone snapped to the lattice of the grid.  Kinds:

  operator  DevicePlan.apply_operator on host arrays: the seam an outer solver calls once per iteration
  green     fm_green_apply_noalloc on device buffers the caller owns
  solve     solve / solve_batch from a host permittivity to host fields
  serve     the slot engine: requests with their own phantoms share launches (continuous batching)

The forms that store complex64 keep their fields as complex64, as a program that chose them for memory does.
"""
import ctypes
import math
import os
import sys
import warnings

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "frequencymaxwell.jl_b200"))

import fmcuda as F  # noqa: E402
from fmcuda import _lib, serving  # noqa: E402

RES, WL, EPS_BG = 50e-9, 500e-9, 1.33 ** 2
ITERATIONS = 100  # what max(2*Bornmax, 100) gives when the tolerance is not met before


def _case(kind, nx, ny, nz, absorb="z", layer=0, precision="float64", solver="gmres", rhs=1, beads=1, radius=8.0,
          tolerance=1e-6, oblique=False, device_phantom=False):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, absorb=absorb, layer=layer, precision=precision, solver=solver,
                rhs=rhs, beads=beads, radius=radius, tolerance=tolerance, oblique=oblique,
                device_phantom=device_phantom)


def listed():
    return [dict(c, name=name) for name, c in (
        # one operator application for an outer solver on a small grid: latency
        ("operator_32", _case("operator", 32, 32, 16, layer=8, radius=4.0)),
        # the Green convolution on the caller's device buffers, one complex64 field of the batching grid
        ("green_128", _case("green", 128, 128, 64, layer=32, precision="float32")),
        # the plain method on the reference's smallest configuration: one bead, double precision, launch-bound
        ("plain_64", _case("solve", 64, 64, 32, layer=16)),
        # the plain method on the batching grid: double precision, 12 beads, one oblique wave
        ("plain_128", _case("solve", 128, 128, 64, layer=32, beads=12, oblique=True)),
        # the precision configuration in single precision: one bead of 16 px, x-polarised wave along +z
        ("precision_128", _case("solve", 128, 128, 64, layer=32, precision="float32", radius=16.0)),
        # many illuminations of one phantom: the headline workload at the batch a third of the memory holds
        ("batch_128", _case("solve", 128, 128, 64, layer=32, precision="float32-math64", solver="block", rhs=6,
                            beads=12, oblique=True)),
        # the largest grid of the serving mix as one solve with restarts
        ("restart_256", _case("solve", 256, 256, 128, layer=64, precision="float32-math64", solver="restart20",
                              beads=40, radius=16.0)),
        # the longest axes (512 on x and z), as the large single configuration has them, one slab of it
        ("long_512", _case("solve", 512, 64, 256, layer=128, precision="float32-math64", solver="restart20",
                           beads=12, radius=12.0)),
        # the reference's first example: 3 um absorbing layers give z = 124, not a power of two; loose tolerance
        ("example_124", _case("solve", 128, 128, 64, layer=30, radius=10.0, tolerance=1e-2, device_phantom=True)),
        # the grid of the reference's two-beam example (201 x 201 x 197 padded): two coherent waves, BiCGStab
        ("beams_201", _case("solve", 201, 201, 191, layer=3, solver="bicgstab", radius=10.0, tolerance=1e-1)),
        # an open domain: absorbing layers on all axes, the two shifted branches differ on every axis
        ("open_128", _case("solve", 96, 96, 96, absorb="xyz", layer=16, precision="float32-math64", solver="block",
                           rhs=2, beads=6, radius=10.0, oblique=True)),
        # small requests served together: three phantoms, four illuminations each, eight slots
        ("serve_64", _case("serve", 64, 64, 32, layer=16, precision="float32-math64", solver="block", rhs=12,
                           beads=4, radius=6.0, tolerance=1e-5, oblique=True)),
    )]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: half on axes the fused passes take, half on any length (odd ones too)."""
    while True:
        what = rng.choice(["operator", "green", "plain", "single", "batch", "restart", "loose", "beams", "open", "serve"])
        tiles = rng.random() < 0.5 or what in ("green", "serve")

        def axes(lo, hi):
            pool = [n for n in (32, 64, 96, 128, 256, 512) if lo <= n <= hi]
            return [rng.choice(pool) if tiles else _spread(rng, lo, min(hi, 220)) for _ in range(3)]
        bx, by, pz = axes(32, 128)
        if what in ("green", "serve") or tiles:
            pz = rng.choice([32, 64, 128])
            if what == "green":
                bx, by = [n if n != 96 else 64 for n in (bx, by)]
        layer = pz // 4 if tiles and what != "green" else rng.randint(3, pz // 3)
        nz = pz - 2 * layer
        radius = rng.uniform(2.0, min(16.0, bx / 6, by / 6, nz / 5))
        if radius < 1.0 or nz < 8:
            continue
        if what == "operator":
            c = _case("operator", bx, by, nz, layer=layer, radius=radius,
                      precision=rng.choice(["float64", "float32", "float32-math64"]))
        elif what == "green":
            c = _case("green", bx, by, nz, layer=layer, precision="float32")
        elif what == "plain":
            c = _case("solve", bx, by, nz, layer=layer, radius=radius, beads=rng.randint(1, 4), oblique=True)
        elif what == "single":
            c = _case("solve", bx, by, nz, layer=layer, radius=radius, precision="float32")
        elif what == "batch":
            c = _case("solve", bx, by, nz, layer=layer, radius=radius, precision="float32-math64", solver="block",
                      rhs=rng.randint(1, 6), beads=rng.randint(1, 4), oblique=True)
            if (3 * bx * by * pz) % 4:
                continue
        elif what == "restart":
            bx, by, pz = axes(64, 512)
            layer = pz // 4 if tiles else rng.randint(3, pz // 3)
            c = _case("solve", bx, by, pz - 2 * layer, layer=layer, precision="float32-math64", solver="restart20",
                      radius=rng.uniform(4.0, 8.0), beads=4)
            if tiles and pz == 96 or bx * by * pz > (16 << 20) / (1 if tiles else 8) or bx * by * pz < 1 << 20:
                continue
        elif what == "loose":
            c = _case("solve", bx, by, nz, layer=layer, radius=radius, tolerance=1e-2, device_phantom=True)
        elif what == "beams":
            c = _case("solve", bx, by, nz, layer=layer, solver="bicgstab", radius=radius, tolerance=1e-1)
        elif what == "open":
            n = rng.choice([32, 64, 128]) if tiles else _spread(rng, 40, 100)
            layer = n // 8
            c = _case("solve", n - 2 * layer, n - 2 * layer, n - 2 * layer, absorb="xyz", layer=layer,
                      precision="float32-math64", solver="gmres", radius=rng.uniform(2.0, n / 12), oblique=True)
        else:
            c = _case("serve", bx if bx < 128 else 64, by if by < 128 else 64, 16, layer=8,
                      precision="float32-math64", solver="block", rhs=rng.randint(3, 12), beads=2, radius=3.0,
                      tolerance=1e-5, oblique=True)
        if what in ("plain", "batch") and not tiles and c["rhs"] * math.prod(_padded(c)) > 1 << 20:
            continue
        if all(any(c[k] != d[k] for k in c) for d in listed()):
            return c


# ---- inputs ----------------------------------------------------------------------------------------------------

def _grid(c):
    return c["nx"], c["ny"], c["nz"]


def _pad(c):
    return tuple(c["layer"] if a in c["absorb"] else 0 for a in "xyz")


def _padded(c):
    return tuple(n + 2 * p for n, p in zip(_grid(c), _pad(c)))


def _beads(c, rng):
    """(centre, radius, index) of non-overlapping beads; one bead sits at the centre, as phantom_bead puts it."""
    g, out = _grid(c), []
    if c["beads"] == 1:
        return [([(n + 1) / 2 for n in g], c["radius"], rng.uniform(1.36, 1.60))]
    for _ in range(20000):
        r = rng.uniform(0.4, 1.0) * c["radius"]
        p = [rng.uniform(1 + r, n - r) for n in g]
        if all(math.dist(p, q) >= r + s + 1 for q, s, _ in out):
            out.append((p, r, rng.uniform(1.36, 1.60)))
            if len(out) == c["beads"]:
                break
    return out


def _paint(c, beads):
    eps = np.full(_grid(c), complex(EPS_BG), order="F")
    for p, r, n in beads:
        lo = [max(1, round(x - r)) for x in p]
        hi = [min(m, round(x + r)) for x, m in zip(p, _grid(c))]
        i, j, k = np.ogrid[lo[0]:hi[0] + 1, lo[1]:hi[1] + 1, lo[2]:hi[2] + 1]
        inside = (i - p[0]) ** 2 + (j - p[1]) ** 2 + (k - p[2]) ** 2 <= r ** 2
        eps[lo[0] - 1:hi[0], lo[1] - 1:hi[1], lo[2] - 1:hi[2]][inside] = n * n
    return eps


def _waves(c, rng):
    """rhs waves of (k, polarisation, phase); two per right-hand side for BiCGStab's coherent pair."""
    kbg = 2 * math.pi * math.sqrt(EPS_BG) / WL
    out = []
    for b in range(c["rhs"] * (2 if c["solver"] == "bicgstab" else 1)):
        if c["oblique"]:
            while True:
                q = [round(rng.uniform(-1, 1) * kbg * 0.9 / d) * d / kbg
                     for d in (2 * math.pi / (n * RES) for n in (c["nx"], c["ny"]))]
                if math.hypot(*q) <= 1.2 / 1.33:
                    break
        else:
            m = 0.0 if c["solver"] != "bicgstab" else (3 if b else -3)
            q = [m * 2 * math.pi / (c["nx"] * RES) / kbg, 0.0]
        k = np.array([q[0], q[1], math.sqrt(1 - q[0] ** 2 - q[1] ** 2)])
        s = np.cross([0.0, 1.0, 0.0] if b % 2 == 0 or not c["oblique"] else [1.0, 0.0, 0.0], k)
        out.append((k / np.linalg.norm(k), s / np.linalg.norm(s), rng.uniform(0, 2 * math.pi)))
    return out


def _requests(c):
    """Phantoms of one pass: one, or (serve) three that share the right-hand sides out."""
    return 3 if c["kind"] == "serve" else 1


def _inputs(c, seed):
    rng = np.random.default_rng(seed)
    return [_beads(c, rng) for _ in range(_requests(c))], _waves(c, rng)


def _field(c, seed, dtype):
    """A random field on the padded grid, x fastest: torch layout (3, z, y, x)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = _padded(c)
    return torch.view_as_complex(torch.randn(3, nz, ny, nx, 2, generator=gen, device="cuda", dtype=dtype))


def _solver(c):
    bcs = [F.AbsorbingBoundaryCondition(2 * c["layer"] * RES, 2 * c["layer"] * RES, 1.0, F.TanhProfile)
           if a in c["absorb"] else F.PeriodicBoundaryCondition() for a in "xyz"]
    linear = {"gmres": F.KrylovJL_GMRES(), "block": F.KrylovJL_GMRES(ortho="block"),
              "restart20": F.KrylovJL_GMRES(gmres_restart=20), "bicgstab": F.KrylovJL_BICGSTAB()}[c["solver"]]
    return F.ConvergentBornSolver(resolution=(RES,) * 3, grid_size=_grid(c), boundary_conditions=bcs,
                                  iterations_max=ITERATIONS // 2, tolerance=c["tolerance"], linear_solver=linear,
                                  precision=c["precision"], max_rhs=max(1, c["rhs"]))


class _Engine(serving.Engine):
    """An engine that gives its slots back when the program lets go of it."""

    def __del__(self):
        self.close()


def prepare(case, seed):
    c = case
    phantoms, waves = _inputs(c, seed)
    if c["kind"] == "green":
        desc = _lib.fm_plan_desc()
        desc.grid[:], desc.pad[:] = _grid(c), _pad(c)
        desc.resolution[:], desc.absorbing[:] = (RES,) * 3, [int(a in c["absorb"]) for a in "xyz"]
        desc.precision, desc.max_rhs = _lib.FM_PREC_F32, 1
        x = _field(c, seed, torch.float32)
        return {"kind": "green", "desc": desc, "x": x, "y": torch.empty_like(x), "scalars": _scalars(c, phantoms[0])}
    solver = _solver(c)
    sources = [F.PlaneWaveSource(wavelength=WL, polarization=e, k_vector=k, phase=ph) for k, e, ph in waves]
    if c["kind"] == "operator":
        plan = solver.plan()
        plan.build_potential(_paint(c, phantoms[0]), EPS_BG, WL, solver.attenuation_filters(), -1)
        x = _field(c, seed, torch.float64).permute(3, 2, 1, 0).cpu().numpy()
        return {"kind": "operator", "single": c["precision"] != "float64", "solver": solver, "plan": plan,
                "x": np.asfortranarray(x)}
    if c["kind"] == "serve":
        media = [F.Medium(_paint(c, p), EPS_BG) for p in phantoms]
        engine = _Engine(solver, min(8, c["rhs"]), basis=112, wavelength=WL, permittivity_bg=EPS_BG,
                         ortho="block")
        return {"kind": "serve", "single": True, "engine": engine, "media": media,
                "sources": [sources[i::3] for i in range(3)], "tolerance": c["tolerance"]}
    if c["device_phantom"]:
        (p, r, n), = phantoms[0]
        medium = F.DevicePhantom(_grid(c), [F.Shape(0, tuple(p), complex(n * n), radius=r)], EPS_BG)
    else:
        medium = F.Medium(_paint(c, phantoms[0]), EPS_BG)
    return {"kind": "solve", "single": c["precision"] != "float64", "solver": solver, "medium": medium,
            "coherent": c["solver"] == "bicgstab", "sources": sources}


def _keep(a, single):
    """The field a program keeps: complex64 where the solver stores complex64."""
    t = torch.from_numpy(a)
    return t.to(torch.complex64) if single else t


def run(state):
    s = state
    if s["kind"] == "green":
        k_bg, eps_imag = s["scalars"]
        status = _lib.lib().fm_green_apply_noalloc(
            ctypes.byref(s["desc"]), k_bg, eps_imag, 1, ctypes.c_void_p(s["x"].data_ptr()),
            ctypes.c_void_p(s["y"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.check(status)
        return s["y"]
    if s["kind"] == "operator":
        return _keep(s["plan"].apply_operator(s["x"]), s["single"])
    if s["kind"] == "serve":
        requests = [serving.Request(req_id=i, medium=m, sources=src, tolerance=s["tolerance"])
                    for i, (m, src) in enumerate(zip(s["media"], s["sources"]))]
        for r in requests:
            s["engine"].submit(r)
        s["engine"].drain(requests)
        return [_keep(a, True) for r in requests for a in (r.E, r.H)]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)  # the iteration limit is reached by intention
        if s["coherent"] or len(s["sources"]) == 1:
            fields = [F.solve(s["solver"], s["sources"], s["medium"])]
        else:
            fields = F.solve_batch(s["solver"], [[w] for w in s["sources"]], s["medium"])
    return [_keep(a, s["single"]) for f in fields for a in (f.E, f.H)]


def work(case):
    """Bytes: inputs and outputs once, per iteration one read and one write of a field and a read of the potential,
    and each Krylov vector once per orthogonalisation (once per eight for the block form).  Flops: six transforms a
    branch pair, the Green product, and two multiply-adds per vector element of the orthogonalisation."""
    c = case
    n, g = math.prod(_padded(c)), math.prod(_grid(c))
    esz = 16 if c["precision"] == "float64" else 8
    transforms = 2 * 3 * 5 * n * math.log2(n) * (2 if c["absorb"] == "xyz" else 1)
    apply_flops = transforms + 60 * n
    if c["kind"] == "green":
        return {"bytes": 2 * 3 * n * esz, "flops": apply_flops}
    if c["kind"] == "operator":
        return {"bytes": 2 * 3 * n * 16 + n * esz, "flops": apply_flops + 60 * n}
    loose = {1e-1: 10, 1e-2: 22}.get(c["tolerance"], ITERATIONS)
    applies = c["rhs"] * (loose * (2 if c["solver"] == "bicgstab" else 1) + 2)
    depth = {"bicgstab": 6, "restart20": 11}.get(c["solver"], loose / 2) / (8 if c["solver"] == "block" else 1)
    vectors = c["rhs"] * loose * depth
    return {"bytes": applies * (2 * 3 * n + n) * esz + vectors * 3 * n * esz
            + g * 16 * _requests(c) + c["rhs"] * 2 * 3 * g * 16,
            "flops": applies * apply_flops + c["rhs"] * loose * depth * (8 if c["solver"] == "block" else 1) * 16 * 3 * n}


# ---- the same results from plain torch, in 64 bits ----------------------------------------------------------------

def _scalars(c, beads):
    k_bg = 2 * math.pi * math.sqrt(EPS_BG) / WL
    vmax = max((abs(k_bg ** 2 * (n * n / EPS_BG - 1)) for _, _, n in beads), default=0.0)
    return k_bg, max(2.0 ** -20, 1.01 * vmax)


class _Exact:
    """The solve of one phantom in FP64: fields are (3, z, y, x)."""

    def __init__(self, c, beads):
        self.c, self.dev = c, "cuda" if torch.cuda.is_available() else "cpu"
        self.k_bg, self.eps = _scalars(c, beads)
        self.ksq = complex(self.k_bg ** 2, self.eps)
        self.shape = _padded(c)
        pad, grid = _pad(c), _grid(c)
        v = torch.zeros(self.shape, dtype=torch.complex128, device=self.dev)
        self.roi = tuple(slice(p, p + n) for p, n in zip(pad, grid))
        v[self.roi] = self.k_bg ** 2 * (torch.from_numpy(_paint(c, beads)).to(self.dev) / EPS_BG - 1)
        v -= 1j * self.eps
        for d in range(3):
            if pad[d]:
                t = np.tanh(np.linspace(-2.5, 2.5, pad[d]))
                w = (t / math.tanh(2.5) - math.tanh(-2.5)) / 2
                f = torch.from_numpy(np.concatenate([w, np.ones(grid[d]), w[::-1]])).to(self.dev)
                v *= f.reshape([-1 if a == d else 1 for a in range(3)])
        self.v = v.permute(2, 1, 0).contiguous()

    def _axis(self, d, values):
        return torch.as_tensor(values, dtype=torch.float64, device=self.dev).reshape([-1 if a == 2 - d else 1 for a in range(3)])

    def _branch(self, x, sign):
        n, k, ramp = self.shape, [], 1.0
        for d in range(3):
            s = sign * 0.25 if "xyz"[d] in self.c["absorb"] else 0.0
            i = np.arange(n[d])
            k.append(self._axis(d, 2 * math.pi / (n[d] * RES) * ((i + n[d] // 2) % n[d] - n[d] // 2 + s)))
            if s:
                ramp = ramp * torch.exp(-2j * math.pi * self._axis(d, i * s / n[d]))
        f = torch.fft.fftn(x * ramp, dim=(1, 2, 3))
        ke = (k[0] * f[0] + k[1] * f[1] + k[2] * f[2]) / self.ksq
        den = k[0] ** 2 + k[1] ** 2 + k[2] ** 2 - self.ksq
        for d in range(3):
            f[d] = (f[d] - k[d] * ke) / den
        f = torch.fft.ifftn(f, dim=(1, 2, 3))
        return f * ramp.conj() if torch.is_tensor(ramp) else f

    def green(self, x):
        if not self.c["absorb"]:
            return self._branch(x, 1)
        return (self._branch(x, 1) + self._branch(x, -1)) / 2

    def operator(self, x):
        return x - self.green(self.v * x)

    def precondition(self, x):
        return (1j / self.eps) * self.v * x

    def incident(self, waves):
        pad, grid = _pad(self.c), _grid(self.c)
        E = torch.zeros((3,) + self.shape[::-1], dtype=torch.complex128, device=self.dev)
        H = torch.zeros_like(E)
        for k, e, phase in waves:
            a = 1.0
            for d in range(3):
                r = (np.arange(self.shape[d]) - pad[d]) * RES - (grid[d] - 1) * RES / 2
                a = a * torch.exp(1j * self._axis(d, self.k_bg * k[d] * r))
            a = a * complex(math.cos(phase), math.sin(phase))
            h = np.cross(k, e) / (377 / math.sqrt(EPS_BG))
            for d in range(3):
                E[d] += a * e[d]
                H[d] += a * h[d]
        return E, H

    def curl(self, x):
        n = self.shape
        k = [self._axis(d, 2 * math.pi / (n[d] * RES) * np.where(np.arange(n[d]) < n[d] // 2, np.arange(n[d]), np.arange(n[d]) - n[d]))
             for d in range(3)]
        f = torch.fft.fftn(x, dim=(1, 2, 3))
        out = torch.stack([k[1] * f[2] - k[2] * f[1], k[2] * f[0] - k[0] * f[2], k[0] * f[1] - k[1] * f[0]])
        return torch.fft.ifftn(1j * out, dim=(1, 2, 3))

    def solve(self, waves, restart, method, tolerance):
        E, H = self.incident(waves)
        b = self.green(self.v * E + 1j * self.eps * E)
        step = _bicgstab if method == "bicgstab" else _gmres
        x = step(lambda u: self.precondition(self.operator(u)), lambda u: self.precondition(b - self.operator(u)), b,
                 tolerance, restart)
        h = -1j * WL / (2 * math.pi * 377) * self.curl(x)
        return [f.permute(3, 2, 1, 0)[self.roi].contiguous() for f in (x + E, h + H)]


def _gmres(op, residual, b, tolerance, restart):
    """Left-preconditioned GMRES from x = b with Givens rotations, stopping as Krylov.jl does."""
    x, done, limit = b, 0, None
    while True:
        r = residual(x).reshape(-1)
        beta = float(torch.linalg.vector_norm(r))
        limit = tolerance * 1e-2 + tolerance * beta if limit is None else limit
        if beta <= limit and done == 0:
            return x
        m = min(restart or ITERATIONS, ITERATIONS)
        V = torch.empty((m + 1, r.numel()), dtype=r.dtype, device=r.device)
        V[0] = r / beta
        R, z, rot = np.zeros((m, m), complex), [complex(beta)], []
        for j in range(m):
            w = op(V[j].reshape(b.shape)).reshape(-1)
            h = torch.zeros(j + 1, dtype=w.dtype, device=w.device)
            for _ in range(2):  # classical Gram-Schmidt twice
                p = torch.stack([torch.vdot(V[i], w) for i in range(j + 1)])
                w = w - V[:j + 1].T @ p
                h += p
            norm = float(torch.linalg.vector_norm(w))
            col = list(h.cpu().numpy()) + [norm]
            for i, (cs, sn) in enumerate(rot):
                col[i], col[i + 1] = cs * col[i] + sn * col[i + 1], np.conj(sn) * col[i] - cs * col[i + 1]
            rho = math.hypot(abs(col[j]), norm)
            ph = col[j] / abs(col[j])
            rot.append((abs(col[j]) / rho, ph * norm / rho))
            R[:j, j], R[j, j] = col[:j], ph * rho
            z[j:] = [rot[j][0] * z[j], np.conj(rot[j][1]) * z[j]]
            done += 1
            if abs(z[j + 1]) <= limit or done >= ITERATIONS or j + 1 == m:
                break
            V[j + 1] = w / norm
        y = np.linalg.solve(R[:j + 1, :j + 1], np.array(z[:j + 1]))
        x = x + (V[:j + 1].T @ torch.from_numpy(y).to(x.device)).reshape(b.shape)
        del V
        if abs(z[j + 1]) <= limit or done >= ITERATIONS:
            return x


def _bicgstab(op, residual, b, tolerance, restart):
    """Left-preconditioned BiCGStab with shadow vector b, from x = b."""
    dot = lambda u, v: complex(torch.vdot(u.reshape(-1), v.reshape(-1)))  # noqa: E731
    x, r = b.clone(), residual(b)
    p, norm = r.clone(), float(torch.linalg.vector_norm(r))
    limit, rho = tolerance * 1e-2 + tolerance * norm, dot(b, r)
    for _ in range(ITERATIONS):
        if norm <= limit:
            break
        v = op(p)
        alpha = rho / dot(b, v)
        s = r - alpha * v
        t = op(s)
        omega = dot(t, s) / dot(t, t)
        x = x + alpha * p + omega * s
        r = s - omega * t
        rho, old = dot(b, r), rho
        p = r + (rho / old) * (alpha / omega) * (p - omega * v)
        norm = float(torch.linalg.vector_norm(r))
    return x


def exact(case, seed):
    c = case
    phantoms, waves = _inputs(c, seed)
    if c["kind"] == "green":
        return _Exact(c, phantoms[0]).green(_field(c, seed, torch.float32).to(torch.complex128))
    if c["kind"] == "operator":
        return _Exact(c, phantoms[0]).operator(_field(c, seed, torch.float64)).permute(3, 2, 1, 0).contiguous()
    out, restart = [], 20 if c["solver"] == "restart20" else 0
    for i, beads in enumerate(phantoms):
        e = _Exact(c, beads)
        mine = waves[i::3] if c["kind"] == "serve" else waves
        if c["solver"] == "bicgstab":
            mine = [mine]
        else:
            mine = [[w] for w in mine]
        fields = [e.solve(w, restart, c["solver"], c["tolerance"]) for w in mine]
        if c["kind"] == "serve":
            out += [torch.stack([f[a] for f in fields], dim=-1) for a in (0, 1)]
        else:
            out += [a for f in fields for a in f]
    return out
