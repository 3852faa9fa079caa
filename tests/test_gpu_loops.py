"""The one-launch loops of the whole-solve path against the per-call ext_* sequence, bit for bit:
the on-chip loops of grids that fit the SMs and the streaming CG loop of those that do not.

Sizes sit where the split can go wrong: fewer cells than a warp, one past a 64-cell strip,
one block and many, every number of rows a warp may own, tiles cut unevenly along every axis,
and the largest grids that fit.  The FP32 inner solves are compared with the same solve run
one launch per sweep.  Both paths do the same operations per cell and their sums are rounded
from twice the working precision, so nothing may differ."""
import ctypes
import os

import numpy as np
import pytest

from conftest import same, tea

pytestmark = pytest.mark.gpu

FIELDS = ("iterations", "error", "exact_error", "vol", "mass", "ie", "temp")
# Too large for the chip: the streaming CG loop, on ragged sides and on few and many work units.
STREAM_SHAPES = {2: [(1101, 1003), (4099, 300), (300, 4100)], 3: [(101, 99, 97), (3, 200, 100), (257, 66, 65)]}
SHAPES = {2: [(7, 5), (65, 16), (64, 17), (131, 33), (700, 37), (257, 515), (701, 699), (860, 850), (1023, 1009)],
          3: [(5, 4, 3), (65, 9, 8), (31, 30, 29), (48, 48, 48), (66, 52, 77), (80, 77, 76)]}
# One cluster: cut along each axis and along two, into few blocks and into sixteen, odd tiles.
CLUSTER_SHAPES = {2: [(2, 33), (129, 11), (131, 35), (33, 150), (127, 128)],
                  3: [(17, 7, 9), (33, 16, 5), (66, 5, 24), (30, 2, 61), (63, 15, 16)]}


def _deck(dim, shape, solver, precond):
    # A timestep at which the coefficients stay below about 40, so that every loop converges soon.
    dt = 0.4 * (10.0 / max(shape)) ** 2
    spec = tea.DeckSpec(dim=dim, cells=8, states=6, seed=sum(shape), solver=solver, end_step=2, dt=dt, eps=1e-12,
                        max_iters=400, presteps=10, inner_steps=5 if sum(shape) % 2 else 6, preconditioner=precond,
                        summary_frequency=1)
    deck = tea.seeded_deck(spec)
    for axis, n in zip("xyz", shape):
        deck = deck.replace(f"{axis}_cells=8\n", f"{axis}_cells={n}\n")
    return deck


def _run(deck, dim, **kw):
    """The run's records and its final u and energy1."""
    lib = tea.cuda_library(dim)
    try:
        _, records = tea.run_deck(deck, dim, summary_every_step=True, keep_chunk=True, **kw)
        dims = (ctypes.c_int * 3)()
        assert lib.tea_chunk_dims_(ctypes.byref(ctypes.c_int(1)), dims) == 0
        chunk = tea.ExtChunk.__new__(tea.ExtChunk)
        chunk.lib, chunk.dim, chunk.id = lib, dim, 1
        chunk.X, chunk.Y, chunk.Z = dims
        return records, {f: chunk.read(f) for f in ("u", "energy1")}
    finally:
        lib.ext_finalise_()


def _same(a, b):
    assert len(a[0]) == len(b[0]) == 2
    for x, y in zip(a[0], b[0]):
        for k in FIELDS:
            assert same(x[k], y[k]), (x["step"], k, x[k], y[k])
    for f in a[1]:
        assert np.array_equal(a[1][f], b[1][f], equal_nan=True), (f, np.argwhere(a[1][f] != b[1][f])[:3].tolist())


@pytest.mark.parametrize("solver,precond", [("cg", False), ("cg", True), ("chebyshev", False), ("ppcg", False),
                                            ("jacobi", False)])
@pytest.mark.parametrize("dim,shape", [(d, s) for d in (2, 3) for s in SHAPES[d]])
def test_on_chip_loops_equal_per_call(dim, shape, solver, precond):
    deck = _deck(dim, shape, solver, precond)
    _same(_run(deck, dim, fused=True), _run(deck, dim))


@pytest.mark.parametrize("solver,precond", [("cg", True), ("chebyshev", False), ("ppcg", False), ("jacobi", False)])
@pytest.mark.parametrize("dim,shape", [(d, s) for d in (2, 3) for s in CLUSTER_SHAPES[d]])
def test_cluster_loops_equal_per_call(dim, shape, solver, precond):
    deck = _deck(dim, shape, solver, precond)
    _same(_run(deck, dim, fused=True), _run(deck, dim))


@pytest.mark.parametrize("solver", ["chebyshev", "ppcg"])
@pytest.mark.parametrize("shape", [(1021, 1019), (900, 1100), (1039, 1024)])  # 7 and 8 rows a warp, wide and narrow tiles
def test_in_place_loops_equal_per_call(shape, solver):
    deck = _deck(2, shape, solver, False)
    _same(_run(deck, 2, fused=True), _run(deck, 2))


@pytest.mark.parametrize("precond", [False, True])
@pytest.mark.parametrize("dim,shape", [(d, s) for d in (2, 3) for s in STREAM_SHAPES[d]])
def test_streaming_cg_equals_per_call(dim, shape, precond):
    deck = _deck(dim, shape, "cg", precond)
    _same(_run(deck, dim, fused=True), _run(deck, dim))


@pytest.mark.parametrize("solver", ["cg", "chebyshev", "ppcg"])
@pytest.mark.parametrize("dim,shape", [(d, s) for d in (2, 3) for s in SHAPES[d][1::2] + CLUSTER_SHAPES[d][::2] + STREAM_SHAPES[d][::2]])
def test_one_launch_fp32_loops_equal_single_launches(dim, shape, solver):
    deck = _deck(dim, shape, solver, False)
    kw = {"fused": True, "precision": tea.PRECISION_FP32_REFINED}
    on_chip = _run(deck, dim, **kw)
    os.environ["TEA_B200_NO_GRAPH"] = "1"
    try:
        single = _run(deck, dim, **kw)
    finally:
        del os.environ["TEA_B200_NO_GRAPH"]
    assert all(r["corrections"] >= 1 for r in on_chip[0])
    _same(on_chip, single)


def _spec_deck(dim, shape, states=6, **kw):
    deck = tea.seeded_deck(tea.DeckSpec(dim=dim, cells=8, states=states, end_step=1, summary_frequency=1, **kw))
    for axis, n in zip("xyz", shape):
        deck = deck.replace(f"{axis}_cells=8\n", f"{axis}_cells={n}\n")
    return deck


def _same_step(a, b, what):
    for k in FIELDS:
        assert same(a[0][0][k], b[0][0][k]), (what, k, a[0][0][k], b[0][0][k])
    for f in a[1]:
        assert np.array_equal(a[1][f], b[1][f], equal_nan=True), (what, f)


@pytest.mark.parametrize("solver", ["chebyshev", "ppcg"])
@pytest.mark.parametrize("dim,shape", [(2, (10, 10)), (2, (131, 33)), (2, (300, 200)), (2, (1101, 1003)), (3, (17, 7, 9))])
def test_solve_that_ends_in_its_cg_phase_equals_per_call(dim, shape, solver):
    # Converged from above the switch's error of 1, or out of iterations where it would switch: no switch follows.
    dt = 4.0 * (10.0 / max(shape)) ** 2
    for eps, iters in ((0.9, (400,)), (1e-12, range(3, 30))):
        for max_iters in iters:
            deck = _spec_deck(dim, shape, seed=5, solver=solver, dt=dt, eps=eps, max_iters=max_iters, presteps=3,
                              inner_steps=4)
            _same_step(_run(deck, dim, fused=True), _run(deck, dim), (eps, max_iters))


# ------------------------------------------------------------- sums that cancel or collapse

def _outcome(deck, dim, **kw):
    """The run's records and fields, or the error that it ended with."""
    try:
        return _run(deck, dim, **kw)
    except RuntimeError as e:
        return str(e)


def _same_outcome(a, b, what):
    if isinstance(a, str) or isinstance(b, str):
        # Only the eigenvalue estimate of a Chebyshev or PPCG solve may fail, and then on both paths.
        assert isinstance(a, str) and isinstance(b, str) and "status 5" in a and ("status 5" in b or "eigenvalues" in b), \
            (what, a, b)
        return
    _same_step(a, b, what)


def _single(deck, dim, **kw):
    os.environ["TEA_B200_NO_GRAPH"] = "1"
    try:
        return _outcome(deck, dim, **kw)
    finally:
        del os.environ["TEA_B200_NO_GRAPH"]


# One block, a cluster, and many blocks with one, four and seven rows a warp.
STIFF_SHAPES = [(2, (5, 5)), (2, (10, 10)), (2, (16, 16)), (2, (33, 20)), (2, (23, 2)), (3, (6, 5, 7)), (2, (131, 97)),
                (2, (300, 200)), (3, (31, 30, 29))]


@pytest.mark.parametrize("dt", [1e5, 1e6, 1e7])
@pytest.mark.parametrize("dim,shape", STIFF_SHAPES)
def test_sums_with_cancelling_terms_equal_per_call(dim, shape, dt):
    # Stiff steps: the terms of p.w are far larger than p.w.
    for seed in range(4):
        for solver, precond in (("cg", False), ("cg", True), ("chebyshev", True), ("ppcg", False)):
            deck = _spec_deck(dim, shape, seed=seed, solver=solver, dt=dt, eps=1e-6, max_iters=150, presteps=20,
                              inner_steps=5, preconditioner=precond)
            _same_outcome(_outcome(deck, dim, fused=True), _outcome(deck, dim), (seed, solver, precond))


@pytest.mark.parametrize("dim,shape", [(2, (700, 650)), (2, (1023, 1009)), (2, (1500, 1400)), (3, (101, 99, 97))])
def test_large_sums_with_cancelling_terms_equal_per_call(dim, shape):
    for precond in (False, True):
        deck = _spec_deck(dim, shape, seed=3, solver="cg", dt=1e5, eps=1e-6, max_iters=60, preconditioner=precond)
        _same_outcome(_outcome(deck, dim, fused=True), _outcome(deck, dim), precond)


@pytest.mark.parametrize("dt", [1e3, 1e5])
@pytest.mark.parametrize("dim,shape", STIFF_SHAPES + [(2, (1500, 1400))])
def test_fp32_sums_with_cancelling_terms_equal_single_launches(dim, shape, dt):
    for solver in ("cg", "chebyshev", "ppcg"):
        deck = _spec_deck(dim, shape, seed=1, solver=solver, dt=dt, eps=1e-6, max_iters=100, presteps=20, inner_steps=6)
        kw = {"fused": True, "precision": tea.PRECISION_FP32_REFINED}
        _same_outcome(_outcome(deck, dim, **kw), _single(deck, dim, **kw), solver)


@pytest.mark.parametrize("dt", [0.004, 0.35, 30.0])
@pytest.mark.parametrize("dim,shape", [(2, (2, 2)), (2, (2, 3)), (2, (3, 3)), (2, (6, 2)), (2, (17, 2)), (3, (2, 2, 2)),
                                       (3, (2, 3, 2))])
def test_sums_that_collapse_equal_per_call(dim, shape, dt):
    # CG ends in as many iterations as the operator has eigenvalues, with a fall of r.r by 100 bits in one of
    # them; Jacobi's first sum is far below the error that the loop starts from.
    for seed in range(4):
        for solver, precond in (("cg", False), ("cg", True), ("chebyshev", False), ("jacobi", False)):
            deck = _spec_deck(dim, shape, states=4, seed=seed, solver=solver, dt=dt, eps=1e-60, max_iters=40, presteps=3,
                              preconditioner=precond)
            _same_outcome(_outcome(deck, dim, fused=True), _outcome(deck, dim), (seed, solver, precond))


@pytest.mark.parametrize("inner_steps", [0, -4, -8])
@pytest.mark.parametrize("dim,shape", [(2, (300, 200)), (3, (48, 48, 48))])
def test_chebyshev_solves_do_not_depend_on_inner_steps(dim, shape, inner_steps):
    # Only a PPCG solve has inner steps: the rim words' epochs grow by the exchanges of the loop that runs.
    deck = _deck(dim, shape, "chebyshev", False).replace("end_step=2", "end_step=6")
    own = [ln for ln in deck.splitlines() if ln.startswith("tl_ppcg_inner_steps")][0]
    a = _run(deck.replace(own, f"tl_ppcg_inner_steps={inner_steps}"), dim, fused=True)
    b = _run(deck, dim)
    for x, y in zip(a[0], b[0], strict=True):
        for k in FIELDS:
            assert same(x[k], y[k]), (x["step"], k, x[k], y[k])
    for f in a[1]:
        assert np.array_equal(a[1][f], b[1][f]), f


def _chunk(dim, shape):
    """A chunk with random density and energy."""
    lib = tea.cuda_library(dim)
    chunk = tea.ExtChunk(lib, dim, *shape)
    chunk.initialise(0.0, 0.0, 10.0 / shape[0], 10.0 / shape[1], 0.0, 10.0 / (shape[2] if dim == 3 else 1))
    rng = np.random.default_rng(7)
    chunk.write("density", rng.uniform(0.5, 20.0, (chunk.Z, chunk.Y, chunk.X)))
    chunk.write("energy1", rng.uniform(1.0, 25.0, (chunk.Z, chunk.Y, chunk.X)))
    return lib, chunk


@pytest.mark.parametrize("dim,shape", [(2, (40, 30)), (2, (1101, 1003)), (3, (20, 20, 20))])
def test_cg_loop_timing_is_zero_without_a_loop(dim, shape):
    def timing():
        lib, chunk = _chunk(dim, shape)
        try:
            ms = ctypes.c_double(-1.0)
            lib.tea_kernel_timing_(chunk.cid, ctypes.byref(ctypes.c_int(14)), ctypes.byref(ctypes.c_int(5)), ctypes.byref(ms))
            return ms.value
        finally:
            lib.ext_finalise_()

    assert timing() > 0.0
    os.environ["TEA_B200_NO_GRAPH"] = "1"
    try:
        assert timing() == 0.0
    finally:
        del os.environ["TEA_B200_NO_GRAPH"]


@pytest.mark.parametrize("solver", ["cg", "chebyshev", "ppcg", "jacobi"])
@pytest.mark.parametrize("dim,shape", [(2, (300, 200)), (2, (1500, 1400)), (3, (48, 48, 48))])
def test_waits_that_run_out_end_in_an_error_status(dim, shape, solver):
    # The first block to arrive at a sum waits for the others: with no patience, the loop gives up.
    lib, chunk = _chunk(dim, shape)
    try:
        energy = chunk.read("energy1")
        p = tea.SolveParams()
        p.solver, p.coefficient, p.max_iters, p.ch_cg_presteps, p.ppcg_inner_steps = tea.SOLVERS[solver], 1, 200, 10, 5
        p.dt, p.eps = 0.4 * (10.0 / max(shape)) ** 2, 1e-10

        def solve():
            chunk.write("energy1", energy)
            record = chunk.solve(p)
            return {k: v for k, v in record.items() if k != "reserved"}, chunk.read("u"), chunk.read("energy1")

        first = solve()
        lib.tea_poll_limit_(chunk.cid, ctypes.byref(ctypes.c_int(0)))
        if dim == 2 and shape[0] > 1000 and solver == "jacobi":
            assert solve()[0] == first[0]  # beyond the chip only CG loops are one launch
        else:
            with pytest.raises(RuntimeError, match="status 3: .*lost one another"):
                solve()
        lib.tea_poll_limit_(chunk.cid, ctypes.byref(ctypes.c_int(-1)))
        again = solve()
        assert again[0] == first[0]
        assert np.array_equal(again[1], first[1]) and np.array_equal(again[2], first[2])
    finally:
        lib.ext_finalise_()

@pytest.mark.parametrize("dim,shape", [(2, (131, 33)), (2, (127, 128)), (2, (257, 515)), (2, (860, 850)), (2, (900, 1000)),
                                       (3, (33, 16, 5)), (3, (48, 48, 48)), (3, (66, 52, 77))])
def test_preconditioned_chebyshev_loops_equal_per_call(dim, shape):
    deck = _deck(dim, shape, "chebyshev", True)
    _same(_run(deck, dim, fused=True), _run(deck, dim))


@pytest.mark.parametrize("solver", ["chebyshev", "ppcg"])
@pytest.mark.parametrize("dim,shape", [(2, (10, 10)), (2, (131, 33)), (2, (300, 200)), (2, (1023, 1009)), (2, (1500, 1400)),
                                       (3, (17, 7, 9)), (3, (48, 48, 48)), (3, (101, 99, 97))])
def test_solves_that_fall_back_to_cg_equal_per_call(dim, shape, solver):
    # Too few CG iterations for the spectrum's bounds: the error rises above 1 again and CG goes on from the
    # last residual.  As one launch and, without graphs, as single passes.
    for seed, precond in ((1, False), (2, True), (3, False)):
        deck = _spec_deck(dim, shape, seed=seed, solver=solver, dt=4.0 * (10.0 / max(shape)) ** 2, eps=1e-10,
                          max_iters=120, presteps=4, inner_steps=4, preconditioner=precond)
        b = _outcome(deck, dim)
        _same_outcome(_outcome(deck, dim, fused=True), b, (seed, precond))
        _same_outcome(_single(deck, dim, fused=True), b, (seed, precond, "single"))


@pytest.mark.parametrize("shape", [(10, 10), (131, 33), (300, 200)])
def test_more_inner_steps_than_iterations(shape):
    # The FP64 solve refuses inner steps beyond the iterations that are left, on both paths; no array is
    # shorter than the steps.  The FP32 inner solve takes them all.
    deck = _spec_deck(2, shape, seed=5, solver="ppcg", dt=0.0005 * (10.0 / max(shape)) ** 2, eps=1e-40, max_iters=14,
                      presteps=3, inner_steps=300)
    for kw in ({}, {"fused": True}):
        outcome = _outcome(deck, 2, **kw)
        assert isinstance(outcome, str) and "status 2" in outcome, outcome
    kw = {"fused": True, "precision": tea.PRECISION_FP32_REFINED}
    _same_outcome(_outcome(deck, 2, **kw), _single(deck, 2, **kw), shape)
