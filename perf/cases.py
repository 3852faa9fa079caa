"""The workloads whose speed this repository is measured by.

A case is one implicit timestep of the heat-conduction solve, from the state at time zero, as
a program that embeds the library takes it: the chunk is painted and set up beforehand
(:func:`prepare`); a pass (:func:`run`) copies energy0 into energy, solves, forms the field
summary and reads the new energy field back into the program's own pinned host buffer.  The
solve is the whole-solve entry point (``ext_tea_leaf_solve_``) or, for ``path = "calls"``, the
sequence of per-call ``ext_*`` entry points that an unchanged Fortran driver makes.

Every case has the seeded synthetic layout of the benchmark and the tests (domain 10 x 10 or
10 x 10 x 10, dt 0.004 unless the case says otherwise, density log-uniform in [0.1, 100], energy uniform in [1, 25]); the
seed of :func:`prepare` chooses the layout.  The learned warm start is not among the cases:
it is off unless a program attaches a trained network, and at the sizes it was made for it
saves no time.
"""
from __future__ import annotations

import ctypes
import math
import weakref

import numpy as np
import torch

import __graft_entry__

tea = __graft_entry__.load_package()

DOMAIN = 10.0
ENERGY, U0 = tea.FIELD_IDS["energy1"], tea.FIELD_IDS["u0"]


def _case(name, dim, nx, ny, nz, solver, *, states, eps_rel=1e-10, eps=1e-15, dt=0.004, precond=False, density=False,
          precision="fp64", inner="deck", path="solve", presteps=30, inner_steps=10, max_iters=20000):
    case = dict(name=name, dim=dim, nx=nx, ny=ny, nz=nz, solver=solver, states=states, eps=eps, eps_rel=eps_rel, dt=dt,
                precond=precond, density=density, precision=precision, inner=inner, path=path, presteps=presteps,
                inner_steps=inner_steps, max_iters=max_iters)
    if not name:
        del case["name"]
    return case


def listed():
    return [
        # The reference's default deck is this small: what counts is the time per launch.
        _case("cg_2d_10", 2, 10, 10, 1, "cg", states=6, eps_rel=0.0),
        # Small ragged grids, as in regression decks.
        _case("cheby_2d_97x41", 2, 97, 41, 1, "chebyshev", states=6, eps_rel=0.0, presteps=20),
        # Jacobi, the method a deck gets that names none, on a small tall grid.
        _case("jacobi_2d_33x150", 2, 33, 150, 1, "jacobi", states=6, eps_rel=0.0),
        # The 512 x 512 configuration: plain CG to an absolute 1e-15.
        _case("cg_2d_512", 2, 512, 512, 1, "cg", states=6, eps_rel=0.0, max_iters=10000),
        # The same through the per-call entry points (the drop-in for the Fortran driver).
        _case("calls_cg_2d_512", 2, 512, 512, 1, "cg", states=6, eps_rel=0.0, max_iters=10000, path="calls"),
        # A mid-sized grid, PPCG to 1e-8 (PPCG stalls below that on large 2D grids, on the
        # reference too).
        _case("ppcg_2d_1024", 2, 1024, 1024, 1, "ppcg", states=16, eps_rel=1e-8),
        # An ordinary large grid with odd sides, Chebyshev.
        _case("cheby_2d_2047x2049", 2, 2047, 2049, 1, "chebyshev", states=16),
        # The benchmark's 4096 x 4096 Chebyshev grid, with a tenth of its timestep: from a cold
        # start the full one takes over two seconds.
        _case("cheby_2d_4096", 2, 4096, 4096, 1, "chebyshev", states=16, dt=0.0004),
        # A small 3D grid, CG with the diagonal preconditioner.
        _case("cg_3d_48_precond", 3, 48, 48, 48, "cg", states=12, eps_rel=0.0, precond=True),
        # The 256^3 configuration: PPCG in FP64, CG with FP32 inner sweeps.
        _case("ppcg_3d_256", 3, 256, 256, 256, "ppcg", states=12),
        _case("cg32_3d_256", 3, 256, 256, 256, "cg", states=12, precision="fp32"),
        # The 512^3 grid in its fastest form, a PPCG deck with FP32 Chebyshev corrections; again
        # with a tenth of the configuration's timestep.
        _case("ppcg32_3d_512", 3, 512, 512, 512, "ppcg", states=24, precision="fp32", inner="chebyshev", dt=0.0004),
    ]


def draw(rng):
    def side(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    dim = rng.choice((2, 2, 3))
    precision = rng.choice(("fp64", "fp64", "fp32"))
    solver = rng.choice(("cg", "chebyshev", "ppcg"))
    path = "solve"
    if dim == 2:
        nx, nz = side(10, 4096), 1
        ny = side(max(10, nx // 4), min(4096, 4 * nx))
    else:
        nx = side(8, 256)
        ny = side(max(8, nx // 2), min(256, 2 * nx))
        nz = side(max(8, nx // 2), min(256, 2 * nx))
    cells = nx * ny * nz
    small, large = cells <= 300000, dim == 2 and cells > 2048 * 2048
    if dim == 2 and cells <= 40000 and rng.random() < 0.3:
        solver, precision = "jacobi", "fp64"
    elif dim == 2 and small and solver == "cg" and rng.random() < 0.4:
        path, precision = "calls", "fp64"
    elif dim == 2 and solver == "ppcg" and cells > 1500000:
        solver = "chebyshev"
    elif large and solver == "cg":
        solver = "chebyshev"
    eps_rel = 0.0 if small and rng.random() < 0.5 else (1e-8 if dim == 2 and solver == "ppcg" else 1e-10)
    return _case("", dim, nx, ny, nz, solver, states=rng.choice((6, 12, 16)), eps_rel=eps_rel,
                 dt=0.0004 if large else 0.004,
                 precond=precision == "fp64" and small and solver == "cg" and rng.random() < 0.3,
                 density=small and rng.random() < 0.2, precision=precision,
                 inner=rng.choice(("deck", "chebyshev")) if dim == 3 and not small else "deck",
                 path=path, presteps=rng.choice((20, 30)), inner_steps=rng.choice((6, 10)))


# ----------------------------------------------------------------------------- the program

def _layout(case, seed):
    """The seeded states as the deck reader hands them on: extents moved by dx/100."""
    spec = tea.DeckSpec(dim=case["dim"], cells=8, states=case["states"], seed=int(seed) & 0x7FFFFFFF, domain=DOMAIN)
    d = {"x": DOMAIN / case["nx"], "y": DOMAIN / case["ny"], "z": DOMAIN / case["nz"]}
    states = []
    for line in tea.seeded_deck(spec).splitlines():
        words = line.replace("=", " ").split()
        if words and words[0] == "state":
            s = dict.fromkeys(("density", "energy", "xmin", "xmax", "ymin", "ymax", "zmin", "zmax", "radius"), 0.0)
            s["geometry"] = 1
            for key, value in zip(words[2::2], words[3::2]):
                s[key] = {"rectangle": 1, "cuboid": 1, "circle": 2}[value] if key == "geometry" else float(value)
            if int(words[1]) > 1:
                for axis in "xyz"[:case["dim"]]:
                    s[axis + "min"] += d[axis] / 100.0
                    s[axis + "max"] -= d[axis] / 100.0
            states.append(s)
    return states, d


# Chunks whose program has ended, with their pinned buffers, for the next one of that size:
# the library frees chunks all at once only (ext_finalise_).  A chunk's coordinates are set
# once: the reference's set-up reads the values that an earlier call left.
_idle, _used = {}, {"n": 0, "key": None}


def _take(key):
    if not _used["n"] and _used["key"] not in (None, key):
        _idle.clear()
        tea.cuda_library(_used["key"][0]).ext_finalise_()
    _used["n"] += 1
    _used["key"] = key
    if _idle.get(key):
        return _idle[key].pop()
    dim, nx, ny, nz = key
    chunk = tea.ExtChunk(tea.cuda_library(dim), dim, nx, ny, nz)
    chunk.initialise(0.0, 0.0, DOMAIN / nx, DOMAIN / ny, 0.0, DOMAIN / nz)
    return chunk, torch.empty((chunk.Z, chunk.Y, chunk.X), dtype=torch.float64, pin_memory=True)


def _give(key, chunk, host):
    _used["n"] -= 1
    _idle.setdefault(key, []).append((chunk, host))


class _Program:
    """One set-up chunk, the parameters of its solve and the buffer its energy is read into."""

    def __init__(self, case, seed):
        key = (case["dim"], case["nx"], case["ny"], case["nz"])
        self.case = case
        self.chunk, self.host = _take(key)
        weakref.finalize(self, _give, key, self.chunk, self.host)
        chunk, dim = self.chunk, case["dim"]
        states, _ = _layout(case, seed)
        names = ["density", "energy", "xmin", "xmax", "ymin", "ymax"] + (["zmin", "zmax"] if dim == 3 else []) + ["radius"]
        tables = [np.array([s[k] for s in states]) for k in names]
        geometry = np.array([s["geometry"] for s in states], dtype=np.int32)
        chunk.call("ext_generate_chunk_", ctypes.byref(ctypes.c_int(len(states))),
                   *[t.ctypes.data_as(ctypes.c_void_p) for t in tables], geometry.ctypes.data_as(ctypes.c_void_p),
                   *[ctypes.byref(ctypes.c_int(k)) for k in (1, 2, 3)])
        chunk.update_halo({1, 2}, 2)
        p = self.params = tea.SolveParams()
        p.solver = tea.SOLVERS[case["solver"]]
        p.coefficient = 1 if case["density"] else 2
        p.preconditioner = int(case["precond"])
        p.max_iters, p.ch_cg_presteps = case["max_iters"], case["presteps"]
        p.ppcg_inner_steps = case["inner_steps"]
        p.dt, p.eps, p.eps_rel = case["dt"], case["eps"], case["eps_rel"]
        p.ch_cg_epslim = float(np.float32(1e-5))
        p.precision = tea.PRECISION_FP32_REFINED if case["precision"] == "fp32" else tea.PRECISION_FP64
        p.inner_solver = int(case["inner"] == "chebyshev")

    def halo(self, ids, depth):
        external = (ctypes.c_int * 6)(*[-1] * 6)
        fields = (ctypes.c_int * 6)(*[int(k + 1 in ids) for k in range(6)])
        one = ctypes.c_int(depth)
        return lambda: self.chunk.lib.ext_update_halo_kernel_(self.chunk.cid, external, fields, ctypes.byref(one))

    def cg_by_calls(self):
        """tea_leaf()'s CG branch through the per-call entry points."""
        lib, cid, p, ref = self.chunk.lib, self.chunk.cid, self.params, ctypes.byref
        coefficient, precond = ctypes.c_int(p.coefficient), ctypes.c_int(p.preconditioner)
        dt, rro, pw, rrn = ctypes.c_double(p.dt), ctypes.c_double(), ctypes.c_double(), ctypes.c_double()
        alpha, beta, bb, u0 = ctypes.c_double(), ctypes.c_double(), ctypes.c_double(), ctypes.c_int(0)
        update = self.halo({4, 5}, 1)
        self.halo({1, 3}, 2)()
        lib.ext_cg_solver_init_(cid, ref(coefficient), ref(precond), ref(dt), ref(rro))
        update()
        lib.ext_solver_copy_u_(cid)
        eps = p.eps
        if p.eps_rel > 0.0:
            lib.ext_calculate_2norm_(cid, ref(bb), ref(u0))
            eps = p.eps_rel * p.eps_rel * bb.value
        for _ in range(p.max_iters):
            lib.ext_cg_calc_w_(cid, ref(pw))
            alpha.value = rro.value / pw.value
            lib.ext_cg_calc_ur_(cid, ref(alpha), ref(rrn))
            beta.value = rrn.value / rro.value
            lib.ext_cg_calc_p_(cid, ref(beta))
            update()
            rro.value = rrn.value
            if abs(rrn.value) < eps:
                break
        lib.ext_solver_finalise_(cid)
        self.halo({3}, 1)()

    def timestep(self):
        chunk = self.chunk
        chunk.lib.ext_set_field_kernel_(chunk.cid)
        if self.case["path"] == "calls":
            self.cg_by_calls()
        else:
            chunk.solve(self.params)
        summary = chunk.field_summary()
        if chunk.lib.tea_read_field_(chunk.cid, ctypes.byref(ctypes.c_int(ENERGY)), ctypes.c_void_p(self.host.data_ptr())):
            raise RuntimeError("the energy field could not be read")
        energy = self.host[2:-2, 2:-2, 2:-2] if self.case["dim"] == 3 else self.host[0, 2:-2, 2:-2]
        return {"energy": energy, "summary": np.array(summary)}


def prepare(case, seed):
    return _Program(case, seed)


def run(state):
    return state.timestep()


# ----------------------------------------------------------------------------- work and values

def _iterations(case):
    """About how many operator applications such a solve takes (it grows as the square root
    of the condition number; the factors are from runs of the seeded layouts)."""
    h = DOMAIN / max(case["nx"], case["ny"], case["nz"])
    kappa = 1.0 + 4.0 * case["dim"] * (10.0 if case["density"] else 100.0) * case["dt"] / (h * h)
    if case["solver"] == "jacobi":
        return 5.5 * kappa
    digits = 1.0 if case["eps_rel"] != 1e-8 else 0.8
    return digits * (2.0 + 14.0 * math.sqrt(kappa))


def work(case):
    """A timestep reads density, energy0 and energy and writes energy and u.  Where the five (six)
    arrays that an iteration needs -- u, r, p and the face coefficients -- are more than the
    126 MB of L2, each iteration also has to stream them: read u, r, p and K, write u, r and p.
    An iteration is about 13 (17) operations for the operator and 8 for the vectors."""
    dim, cells = case["dim"], case["nx"] * case["ny"] * case["nz"]
    iterations = _iterations(case)
    word = 4 if case["precision"] == "fp32" else 8
    streamed = cells * word * (3 + dim)
    moved = iterations * cells * word * (6 + dim) if streamed > 126e6 else 0.0
    return {"bytes": 5.0 * 8 * cells + moved, "flops": iterations * cells * (5.0 + 4 * dim + 8)}


def exact(case, seed):
    """The same timestep in plain torch: the painted fields, the operator, and CG with the
    diagonal preconditioner until the residual no longer falls."""
    dim = case["dim"]
    n = [case[k] for k in ("nx", "ny", "nz")[:dim]]
    if max(n) * math.prod(n) > 1.5e10:
        return None  # tens of thousands of passes over large arrays
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    states, d = _layout(case, seed)
    h = [d[a] for a in "xyz"[:dim]]
    longest = max(n) + 4
    shape = [k + 4 for k in reversed(n)]
    # Vertices, and cell centres as the reference's one-thread set-up leaves them: half of the
    # cell's own vertex plus half of the next one, which is still zero -- or, at the end of the
    # axis, was never set.
    vertex, centre = [], []
    for a in range(dim):
        v = h[a] * (torch.arange(n[a] + 5, dtype=torch.float64, device=dev) - 2)
        if n[a] + 4 == longest:
            v[-1] = 0.0
        view = [1] * dim
        view[dim - 1 - a] = -1
        vertex.append((v[:-1].view(view), v[1:].view(view)))
        centre.append((0.5 * v[:-1]).view(view))
    density = torch.full(shape, states[0]["density"], dtype=torch.float64, device=dev)
    energy = torch.full(shape, states[0]["energy"], dtype=torch.float64, device=dev)
    for s in states[1:]:
        if s["geometry"] == 1:
            inside = torch.ones([1] * dim, dtype=torch.bool, device=dev)
            for a in range(dim):
                inside = inside & (vertex[a][1] >= s["xyz"[a] + "min"]) & (vertex[a][0] < s["xyz"[a] + "max"])
        else:
            inside = sum((centre[a] - s["xyz"[a] + "min"]) ** 2 for a in range(dim)).sqrt() <= s["radius"]
        inside = inside.expand(shape)
        density[inside] = s["density"]
        energy[inside] = s["energy"]
    inner = (slice(2, -2),) * dim
    density, energy = density[inner].contiguous(), energy[inner].contiguous()
    w = density if case["density"] else 1.0 / density
    faces, diagonal = [], torch.ones_like(w)
    for a in range(dim):
        axis = dim - 1 - a
        lo, hi = w.narrow(axis, 0, n[a] - 1), w.narrow(axis, 1, n[a] - 1)
        k = case["dt"] / (h[a] * h[a]) * (lo + hi) / (2.0 * lo * hi)
        faces.append((axis, k))
        diagonal.narrow(axis, 0, n[a] - 1).add_(k)
        diagonal.narrow(axis, 1, n[a] - 1).add_(k)

    def apply(x):
        y = x.clone()
        for axis, k in faces:
            m = x.shape[axis] - 1
            flux = k * (x.narrow(axis, 1, m) - x.narrow(axis, 0, m))
            y.narrow(axis, 0, m).sub_(flux)
            y.narrow(axis, 1, m).add_(flux)
        return y

    b = density * energy
    u = b.clone()
    best = None
    for _ in range(3):  # CG, restarted on the true residual
        r = b - apply(u)
        norm = float(r.norm())
        if best is not None and norm >= 0.1 * best:
            break
        best = norm
        z = r / diagonal
        p, rz = z.clone(), torch.dot(r.flatten(), z.flatten())
        x = torch.zeros_like(u)
        stop = 1e-13 * rz
        for it in range(40000):
            q = apply(p)
            alpha = rz / torch.dot(p.flatten(), q.flatten())
            x.add_(alpha * p)
            r.sub_(alpha * q)
            z = r / diagonal
            new = torch.dot(r.flatten(), z.flatten())
            if it % 20 == 19 and float(new) <= float(stop) * 1e-3:
                break
            p.mul_(new / rz).add_(z)
            rz = new
        u += x
    volume = math.prod(h)
    summary = [volume * b.numel(), volume * density.sum(), volume * (density * energy).sum(), volume * (density * u).sum()]
    return {"energy": u / density, "summary": np.array([float(s) for s in summary])}
