"""Parts on which hats of the coarse grid depend on one another: fewer layers of nodes across than the grid has
lines, cells that a bent part touches with a corner. The coarse matrix is singular there, and the
correction has to stay positive definite: fewer iterations than IC(0) alone, at the oracle's field.

Tolerance: the uniform load excites the lowest mode by at least 0.3 of its norm, so that the relative error
is below 4 times the relative residual: 1e-12 and 1e-10 are far inside 1e-10 and 1e-8 (the parity tests')."""
import copy

import numpy as np
import pytest

import maille_b200 as mb
from maille_b200 import meshgen as mg
from maille_b200._lib import MAILLE_FP64, MAILLE_MIXED

pytestmark = pytest.mark.gpu


def part(cells, size, clamped, young, poisson, bend=None):
    """Box of `cells`, clamped on the face 0 of axis `clamped`; bend (radius, angle): x becomes an arc."""
    nodes, conn = mg.box_grid(cells, size)
    root = nodes[:, clamped] < 1e-9
    if bend:
        t, r = nodes[:, 0] / size[0] * bend[1], bend[0] + nodes[:, 1]
        nodes = np.stack([r * np.cos(t), r * np.sin(t), nodes[:, 2]], 1)
        if (mg._signed_volume6(nodes, conn) < 0).all():
            conn = conn[:, [0, 2, 1, 3]]
    n, ne = nodes.shape[0], conn.shape[0]
    fixed = np.repeat(root, 3).astype(np.uint8)
    loads = np.tile([1.0, 0.7, 0.5], n) * (fixed == 0)
    return mg.Problem(coords=nodes, conn=conn, young=young(ne), poisson=np.full(ne, poisson), fixed=fixed,
                      imposed=np.zeros(3 * n), loads=loads)


def uniform(ne):
    return 50000.0 + 200000.0 * mg.uniform(53, ne)


PARTS = {
    "strip": lambda: part((4, 1, 19), (2.561, 2.708, 7.557), 0, uniform, 0.0, (10.49, 0.6005)),
    "arch": lambda: part((2, 10, 7), (2.0, 8.947, 7.0), 0, uniform, 0.0, (64.4, 2.452)),
    "fin": lambda: part((2, 50, 8), (2.552, 26.44, 4.56), 1,
                        lambda ne: 200000.0 * (0.01 + 0.99 * mg.uniform(59, ne)) ** 3, 0.3, (111.2, 1.144)),
    "flat_cells": lambda: part((3, 7, 6), (1.309, 7.0, 2.214), 1,
                               lambda ne: 200000.0 * np.exp(mg.normal(61, ne)), 0.49),
}


@pytest.mark.parametrize("precision,tol,err", [(MAILLE_FP64, 1e-12, 1e-10), (MAILLE_MIXED, 1e-10, 1e-8)])
@pytest.mark.parametrize("name", sorted(PARTS))
def test_dependent_hats(gpu, oracle_lib, monkeypatch, name, precision, tol, err):
    p = PARTS[name]()
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads)
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(tol).with_precision(precision)
    monkeypatch.setenv("MAILLE_COARSE", "0")
    alone = m.solve().info["iterations"]
    monkeypatch.setenv("MAILLE_COARSE", "1")
    f = m.solve()
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-14)
    assert np.linalg.norm(f.displacements - ref["u"]) < err * np.linalg.norm(ref["u"])
    assert f.info["iterations"] < alone


@pytest.mark.parametrize("precision,tol", [(MAILLE_FP64, 1e-12), (MAILLE_MIXED, 1e-10)])
def test_dependent_hats_in_a_batch(gpu, oracle_lib, monkeypatch, precision, tol):
    probs = [PARTS[k]() for k in sorted(PARTS)]
    loads = [p.loads[:, None] for p in probs]
    iterations = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        with mb.BatchSolver(probs, loads, tol=tol, precision=precision) as b:
            f = b.solve()
        assert f.info["status_code"] == 0
        iterations[knob] = f.iterations
    err = 1e-10 if precision == MAILLE_FP64 else 1e-8
    for p, u in zip(probs, f.displacements):
        ref = oracle_lib.model_solve(copy.copy(p), solver=2, tol=1e-14)["u"]
        assert np.linalg.norm(u[:, 0] - ref) < err * np.linalg.norm(ref)
    assert (iterations["1"] < iterations["0"]).all()


@pytest.mark.parametrize("precision", [MAILLE_FP64, MAILLE_MIXED])
@pytest.mark.parametrize("name", ["strip", "fin"])
def test_dependent_hats_of_the_thermal_step(gpu, oracle_lib, monkeypatch, name, precision):
    # near-steady increments, for which the step takes the correction; 1e-9 of the largest temperature as the
    # thermal parity tests
    from maille_b200 import thermal as th
    e = PARTS[name]()
    n, ne = e.n_nodes, e.n_elems
    fixed = e.fixed[::3].copy()
    p = mg.ThermalProblem(coords=e.coords, conn=e.conn, conductivity=e.young / 1e5, rho_c=np.ones(ne), fixed=fixed,
                          imposed=np.where(fixed != 0, 100.0, 0.0), loads=np.zeros(n), initial=np.full(n, 20.0),
                          time_period=1e5, increments=2, s_elem=np.arange(ne, dtype=np.int64),
                          s_value=np.full(ne, 0.5))
    ref = oracle_lib.thermal_transient(p, solver=2)
    s, out = th.solve_problem(p, f=ref["f"], precision=precision)
    assert s == 0
    assert np.abs(out["temps"] - ref["temps"]).max() < 1e-9 * np.abs(ref["temps"]).max()
