"""AUTO's ordering (greedy colouring by node index, one pass of iterated greedy) computed on the device and by
the host analysis (MAILLE_HOST_ORDERING=1): the same algorithm on the same graph, hence the same levels,
iterations and results bit for bit, with node ids as generated and permuted."""
import copy

import numpy as np
import pytest

import maille_b200 as mb
from maille_b200 import meshgen as mg, thermal as th

import cases

pytestmark = pytest.mark.gpu


def permuted(p):
    """The same mesh with its node ids permuted at random."""
    q, n = copy.copy(p), p.n_nodes
    old = np.argsort(mg.uniform(47, n))  # new id -> old id
    new = np.empty(n, np.int64)
    new[old] = np.arange(n)
    q.coords, q.conn = np.ascontiguousarray(p.coords[old]), new[p.conn]
    for name in ("fixed", "imposed", "loads", "initial"):
        if hasattr(p, name):
            setattr(q, name, np.ascontiguousarray(getattr(p, name).reshape(n, -1)[old]).ravel())
    return q


def elastic():
    p5 = mg.mixed_tet10(5)
    p5.fixed[3 * 40 + 1] = 1  # a node with one fixed DOF stays in the system
    return [mg.plain_tet4(8), p5, cases.two_blocks(3), cases.two_blocks(2, quadratic=True)]


@pytest.mark.parametrize("ids", ["generated", "permuted"])
def test_the_elastic_default(gpu, monkeypatch, ids):
    for p in elastic():
        p = permuted(p) if ids == "permuted" else p
        m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                                 (p.p_elem, p.p_face, p.p_value))
        m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(1e-12)
        monkeypatch.setenv("MAILLE_HOST_ORDERING", "1")
        a = m.solve()
        monkeypatch.delenv("MAILLE_HOST_ORDERING")
        b = m.solve()
        assert a.info["levels"] == b.info["levels"], p.name
        assert a.info["iterations"] == b.info["iterations"], p.name
        assert np.array_equal(a.displacements, b.displacements), p.name


@pytest.mark.parametrize("ids", ["generated", "permuted"])
def test_the_thermal_default(gpu, monkeypatch, ids):
    p = mg.thermal_cube(5, True, increments=2, time_period=0.02)
    p = permuted(p) if ids == "permuted" else p
    monkeypatch.setenv("MAILLE_HOST_ORDERING", "1")
    s1, a = th.solve_problem(p, fluxes=False)
    monkeypatch.delenv("MAILLE_HOST_ORDERING")
    s2, b = th.solve_problem(p, fluxes=False)
    assert s1 == 0 and s2 == 0
    assert a["info"]["levels"] == b["info"]["levels"]
    assert np.array_equal(a["iterations"], b["iterations"])
    assert np.array_equal(a["temps"], b["temps"])
