"""The coarse correction of the IC(0) preconditioner (coarse.cuh): the corrected PCG solves the same
systems as IC(0) alone, in fewer iterations, over the shapes of its grid: one cell, cells without nodes,
thin plates and bars, sweep tiles of 64 unknowns that are not full, fixed components, parts that a
cell holds together, and load cases on one factor."""
import numpy as np
import pytest

import maille_b200 as mb
from maille_b200 import meshgen as mg
from maille_b200._lib import MAILLE_FP64, MAILLE_MIXED, MAILLE_ORDER_MULTICOLOR

import cases

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def box(cells, size, quadratic):
    p = mg.clamped_cube(cells, quadratic, 50000.0 + 150000.0 * mg.uniform(21, 6 * int(np.prod(cells))), size=size)
    rollers = np.nonzero(np.abs(p.coords[:, 0]) < 1e-12)[0]
    p.fixed[3 * rollers] = 1  # rows with one fixed component
    return p


def frame():
    """Two separate blocks with empty cells between them."""
    return cases.two_blocks(5)


SHAPES = {
    "cube_below_the_limit": lambda: box((4, 4, 4), (1.0, 1.0, 1.0), False),
    "cube": lambda: box((9, 9, 9), (1.0, 1.0, 1.0), False),
    "plate": lambda: box((24, 18, 1), (2.4, 1.8, 0.1), False),
    "bar": lambda: box((2, 2, 60), (0.1, 0.1, 3.0), False),
    "ragged_tet10": lambda: box((7, 4, 5), (1.3, 0.7, 1.0), True),
    "two_blocks": frame,
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_the_corrected_pcg_solves_the_same_system(gpu, oracle_lib, monkeypatch, shape):
    # 1e-10 of the oracle at 1e-13, the tolerance of the parity tests
    p = SHAPES[shape]()
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-13)
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                             (p.p_elem, p.p_face, p.p_value))
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(1e-13)
    iterations = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        f = m.solve()
        assert rel(f.displacements, ref["u"]) < 1e-10
        assert rel(f.reactions, ref["reactions"]) < 1e-10
        iterations[knob] = f.info["iterations"]
    # fewer wherever the mesh is several cells from its supports (the plate is clamped on its whole
    # face: there is nothing for a coarse grid to carry)
    if shape in ("cube", "bar", "ragged_tet10"):
        assert iterations["1"] < iterations["0"]


@pytest.mark.parametrize("precision,tol,err", [(MAILLE_FP64, 1e-13, 1e-10), (MAILLE_MIXED, 1e-10, 1e-8)])
def test_new_moduli_renew_the_correction(gpu, oracle_lib, precision, tol, err):
    p = box((8, 6, 7), (1.0, 0.8, 0.9), True)
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                             (p.p_elem, p.p_face, p.p_value))
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(tol).with_precision(precision)
    m.ordering = MAILLE_ORDER_MULTICOLOR
    with mb.SolverHandle(m) as h:
        first = h.solve()
        p.young = 210000.0 * (0.01 + 0.99 * mg.uniform(22, p.n_elems)) ** 3
        h.refactor(young=p.young)
        a, b = h.solve(), h.solve()
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-14)
    assert rel(a.displacements, ref["u"]) < err
    assert np.array_equal(a.displacements, b.displacements)
    assert a.info["iterations"] < 3 * first.info["iterations"]


@pytest.mark.parametrize("quadratic,cells,precision", [(False, 5, MAILLE_FP64), (False, 13, MAILLE_FP64),
                                                       (True, 7, MAILLE_FP64), (True, 7, MAILLE_MIXED)])
def test_the_thermal_step_takes_the_correction(gpu, oracle_lib, monkeypatch, quadratic, cells, precision):
    # 1e-9 of the largest temperature, as the thermal parity tests; fewer iterations where the diffusion
    # length of an increment spans many nodes, the same on the small cube, where the step leaves it out
    from maille_b200 import thermal as th
    p = mg.thermal_cube(cells, quadratic, increments=3, time_period=0.6, theta=0.75)
    ref = oracle_lib.thermal_transient(p, solver=2)
    iterations = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        s, out = th.solve_problem(p, f=ref["f"], precision=precision)
        assert s == 0
        assert np.abs(out["temps"] - ref["temps"]).max() < 1e-9 * np.abs(ref["temps"]).max()
        iterations[knob] = int(out["iterations"].sum())
    assert iterations["1"] < iterations["0"] if cells > 5 else iterations["1"] == iterations["0"]


@pytest.mark.parametrize("rhs,precision,tol,err", [(1, MAILLE_FP64, 1e-13, 1e-10), (3, MAILLE_FP64, 1e-13, 1e-10),
                                                   (8, MAILLE_FP64, 1e-13, 1e-10), (8, MAILLE_MIXED, 1e-10, 1e-8),
                                                   (2, MAILLE_MIXED, 1e-10, 1e-8)])
@pytest.mark.parametrize("threads", ["128", "256"])
def test_a_batch_takes_the_correction(gpu, monkeypatch, rhs, precision, tol, err, threads):
    # instances of 12 to 1331 rows (one cell to 5 a side), every load-case layout, against the same batch
    # with IC(0) alone
    probs, loads = mg.batched_tet4(count=5, lo=2, hi=11, load_cases=rhs)
    monkeypatch.setenv("MAILLE_BATCH_Q", {1: "2", 2: "1", 3: "2", 8: "4"}[rhs])
    monkeypatch.setenv("MAILLE_BATCH_THREADS", threads)
    out = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        with mb.BatchSolver(probs, loads, tol=tol, precision=precision) as b:
            out[knob] = b.solve()
            again = b.solve()
        assert out[knob].info["status_code"] == 0
        assert all(np.array_equal(x, y) for x, y in zip(out[knob].displacements, again.displacements))
    for a, b in zip(out["0"].displacements, out["1"].displacements):
        assert rel(b, a) < 2 * err
    assert out["1"].iterations.max() < out["0"].iterations.max()


@pytest.mark.parametrize("increments", [1, 2, 9, 12])
@pytest.mark.parametrize("theta,precision", [(1.0, MAILLE_FP64), (0.5, MAILLE_FP64), (1.0, MAILLE_MIXED)])
def test_increments_start_from_the_earlier_ones(gpu, oracle_lib, increments, theta, precision):
    # one, two, as many as are kept plus one, and more than that: the oracle's history (1e-9 of the largest
    # temperature, as the thermal parity tests), and never more iterations than the first increment's
    from maille_b200 import thermal as th
    p = mg.thermal_cube(6, True, increments=increments, time_period=0.02 * increments, theta=theta)
    ref = oracle_lib.thermal_transient(p, solver=2)
    s, out = th.solve_problem(p, f=ref["f"], precision=precision)
    assert s == 0
    assert np.abs(out["temps"] - ref["temps"]).max() < 1e-9 * np.abs(ref["temps"]).max()
    assert np.abs(out["reactions"] - ref["reactions"]).max() < 1e-8 * np.abs(ref["reactions"]).max()
    assert (out["iterations"] <= out["iterations"][0]).all()


@pytest.mark.parametrize("cells,precision,tol", [((33, 35, 36), MAILLE_FP64, 1e-12), ((36, 35, 36), MAILLE_FP64, 1e-12),
                                                 ((36, 35, 36), MAILLE_MIXED, 1e-10)])
@pytest.mark.parametrize("blocks", [None, "1", "500"])
def test_the_team_beside_the_sweeps_at_both_block_sizes(gpu, monkeypatch, cells, precision, tol, blocks):
    # either side of 45000 rows, with one sweeping block and with more than fit, against IC(0) alone: two
    # solutions at relative residual tol differ by at most 2 cond(K) tol, cond < 1e5 (about 4 n^2 = 5e3
    # times the moduli's ratio of 4)
    p = box(cells, tuple(0.1 * c for c in cells), False)
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                             (p.p_elem, p.p_face, p.p_value))
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(tol).with_precision(precision)
    m.ordering = MAILLE_ORDER_MULTICOLOR
    if blocks:
        monkeypatch.setenv("MAILLE_PERSIST_GRID", blocks)
    u = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        u[knob] = m.solve()
    assert rel(u["1"].displacements, u["0"].displacements) < 2e5 * tol
    assert u["1"].info["iterations"] < u["0"].info["iterations"]


def test_increments_without_load_stay_zero(gpu):
    # imposed and initial temperatures 0 and no loads: every right-hand side is 0, so is every start
    from maille_b200 import thermal as th
    p = mg.thermal_cube(5, False, increments=4, time_period=0.1, theta=1.0)
    p.imposed[:] = 0.0
    p.initial[:] = 0.0
    s, out = th.solve_problem(p, f=np.zeros(p.n_nodes))
    assert s == 0
    assert not out["temps"].any() and not out["iterations"].any()
