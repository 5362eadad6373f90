"""Nodes that no element names (construction points, left-over nodes of an exported mesh), far from the part and
fixed: they take no part in the system, and none in the grid of its coarse correction either. The same
iterations and bits as without them."""
import copy

import numpy as np
import pytest

import maille_b200 as mb
from maille_b200 import meshgen as mg, thermal as th
from maille_b200._lib import MAILLE_FP64, MAILLE_MIXED

pytestmark = pytest.mark.gpu

FAR = np.array([[-3e4, 50.0, 2e3], [1e4, -7e3, 1e5]])


def with_far_nodes(p):
    q = copy.copy(p)
    q.coords = np.concatenate([p.coords, FAR])
    per = p.fixed.size // p.n_nodes
    q.fixed = np.concatenate([p.fixed, np.ones(2 * per, np.uint8)])
    for name in ("imposed", "loads", "initial"):
        if hasattr(p, name):
            setattr(q, name, np.concatenate([getattr(p, name), np.zeros(2 * per)]))
    return q


@pytest.mark.parametrize("precision,tol", [(MAILLE_FP64, 1e-12), (MAILLE_MIXED, 1e-10)])
def test_a_solve_ignores_unused_nodes(gpu, precision, tol):
    out = []
    p = mg.mixed_tet10(8)
    for q in (p, with_far_nodes(p)):
        m = mb.Model.from_arrays(q.coords, q.conn, q.young, q.poisson, q.fixed, q.imposed, q.loads,
                                 (q.p_elem, q.p_face, q.p_value))
        out.append(m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(tol).with_precision(precision).solve())
    assert out[1].info["iterations"] == out[0].info["iterations"]
    assert np.array_equal(out[1].displacements[:-6], out[0].displacements)
    assert not out[1].displacements[-6:].any()


def test_a_batch_ignores_unused_nodes(gpu, monkeypatch):
    monkeypatch.setenv("MAILLE_BATCH_Q", "2")  # one lane layout: the same order of every sum
    probs, loads = mg.batched_tet4(count=3, lo=8, hi=10, load_cases=2)
    far = [probs[0], with_far_nodes(probs[1]), probs[2]]
    far_loads = [loads[0], np.concatenate([loads[1], np.zeros((6, 2))]), loads[2]]
    out = []
    for pr, l in ((probs, loads), (far, far_loads)):
        with mb.BatchSolver(pr, l, tol=1e-12) as b:
            out.append(b.solve())
    assert np.array_equal(out[0].iterations, out[1].iterations)
    assert np.array_equal(out[1].displacements[1][:-6], out[0].displacements[1])


def test_a_thermal_step_ignores_unused_nodes(gpu):
    p = mg.thermal_cube(12, False, increments=2, time_period=1.0)
    f = th.thermal_loads(p.coords, p.conn, list(zip(p.s_elem, p.s_value)),
                         list(zip(p.c_elem, p.c_face, p.c_film, p.c_sink)))
    s, a = th.solve_problem(p, f=f)
    q = with_far_nodes(p)
    t, b = th.solve_problem(q, f=np.concatenate([f, np.zeros(2)]))
    assert s == 0 and t == 0
    assert np.array_equal(a["iterations"], b["iterations"])
    assert np.array_equal(b["temps"].reshape(3, -1)[:, :-2], a["temps"].reshape(3, -1))
