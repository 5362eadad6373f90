"""The mixed form on bending parts: bars, a plate and a curved shell loaded at their end, where the FP32
residual rises by decades before it falls and its recurrence leaves the true one. Against the oracle's
field, in no more than twice the FP64 form's iterations, in single and batched solves.

Tolerance: u - u* = K^-1 r with ||r|| <= 1e-10 ||b||, and an end load on S sections excites the lowest mode
by at least 2 / sqrt(S) of its norm, so that the relative error is below 1e-10 sqrt(S) / 2 times the load's
share along the bending direction (1.05): under 1e-9 for 60 sections. 1e-8 is asked, as in the other mixed
tests."""
import copy

import numpy as np
import pytest

import maille_b200 as mb
from maille_b200 import meshgen as mg
from maille_b200._lib import MAILLE_FP64, MAILLE_MIXED

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def end_loaded(nodes, conn, root, end, load, draw):
    n, ne = nodes.shape[0], conn.shape[0]
    fixed = np.zeros(3 * n, np.uint8)
    loads = np.zeros(3 * n)
    for c in range(3):
        fixed[3 * np.nonzero(root)[0] + c] = 1
        loads[3 * np.nonzero(end)[0] + c] = load[c] / np.count_nonzero(end)
    return mg.Problem(coords=nodes, conn=conn, young=50000.0 + 200000.0 * mg.uniform(31 + draw, ne),
                      poisson=np.full(ne, 0.3), fixed=fixed, imposed=np.zeros(3 * n), loads=loads)


def bar(cells, quadratic=False, draw=0):
    nodes, conn = mg.box_grid(cells, tuple(map(float, cells)))
    if quadratic:
        nodes, conn = mg.to_quadratic_tet(nodes, conn)
    z = nodes[:, 2]
    return end_loaded(nodes, conn, z < 1e-9, z > cells[2] - 1e-9, (1.0, 0.3, 0.0), draw)


def shell(around, through, along, radius, draw=0):
    """A quarter of a cylinder, clamped on one straight edge's section and loaded on the other."""
    h = radius * np.pi / 2 / around
    nodes, conn = mg.box_grid((around, through, along), (np.pi / 2, through * h, along * h))
    t, r = nodes[:, 0], radius + nodes[:, 1]
    xyz = np.stack([r * np.cos(t), r * np.sin(t), nodes[:, 2]], 1)
    conn = conn[:, [0, 2, 1, 3]] if (mg._signed_volume6(xyz, conn) < 0).all() else conn
    return end_loaded(xyz, conn, t < 1e-9, t > np.pi / 2 - 1e-9, (1.0, 1.0, 0.3), draw)


PARTS = {
    "bar_6_to_1": lambda d: bar((10, 10, 60), draw=d),
    "bar_8_to_1": lambda d: bar((6, 6, 48), draw=d),
    "bar_10_to_1": lambda d: bar((4, 4, 40), draw=d),
    "bar_8_to_1_tet10": lambda d: bar((3, 3, 24), True, draw=d),
    "plate_20_to_1": lambda d: bar((40, 2, 40), draw=d),
    "shell": lambda d: shell(30, 2, 30, 10.0, draw=d),
}


@pytest.mark.parametrize("draw", [0, 1])
@pytest.mark.parametrize("part", sorted(PARTS))
def test_the_mixed_form_converges_on_bending_parts(gpu, oracle_lib, part, draw):
    p = PARTS[part](draw)
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-13)
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads)
    m.with_solver(mb.SolverKind.ITERATIVE)
    plain = m.with_precision(MAILLE_FP64).with_tolerance(1e-12).solve()
    f = m.with_precision(MAILLE_MIXED).with_tolerance(1e-10).solve()
    assert rel(f.displacements, ref["u"]) < 1e-8
    assert f.info["iterations"] <= 2 * plain.info["iterations"]


def test_the_mixed_batch_converges_on_bending_parts(gpu, oracle_lib):
    probs = [PARTS[k](2) for k in ("bar_8_to_1", "bar_10_to_1", "shell")]
    turn = np.array([[1.0, 0.0, 0.0], [0.3, 1.0, 0.2], [-0.5, 0.8, 0.0]])  # load cases: other directions
    loads = []
    for p in probs:
        share = np.abs(p.loads).reshape(-1, 3).max(axis=1)
        loads.append(np.stack([(share[:, None] * d).ravel() * (p.fixed == 0) for d in turn], 1))
    with mb.BatchSolver(probs, loads, tol=1e-12, precision=MAILLE_FP64) as b:
        plain = b.solve()
    with mb.BatchSolver(probs, loads, tol=1e-10, precision=MAILLE_MIXED) as b:
        f = b.solve()
    assert f.info["status_code"] == 0
    for k, (p, l) in enumerate(zip(probs, loads)):
        for j in range(3):
            q = copy.copy(p)
            q.loads = np.ascontiguousarray(l[:, j])
            assert rel(f.displacements[k][:, j], oracle_lib.model_solve(q, solver=2, tol=1e-13)["u"]) < 1e-8
    assert (f.iterations <= 2 * plain.iterations).all()


def test_the_mixed_thermal_step_along_a_bar(gpu, oracle_lib):
    # heat along a 20:1 bar with conductivities over two decades, long increments: 1e-9 of the largest
    # temperature as the thermal parity tests, in no more than twice the FP64 form's iterations
    from maille_b200 import thermal as th
    nodes, conn = mg.box_grid((4, 4, 80), (4.0, 4.0, 80.0))
    n, ne = nodes.shape[0], conn.shape[0]
    fixed = (nodes[:, 2] < 1e-9).astype(np.uint8)
    p = mg.ThermalProblem(coords=nodes, conn=conn, conductivity=0.1 * 100.0 ** mg.uniform(37, ne), rho_c=np.ones(ne),
                          fixed=fixed, imposed=np.where(fixed != 0, 100.0, 0.0), loads=np.zeros(n),
                          initial=np.full(n, 20.0), time_period=3e4, increments=3, theta=1.0,
                          s_elem=np.arange(ne, dtype=np.int64), s_value=np.full(ne, 0.05))
    ref = oracle_lib.thermal_transient(p, solver=2)
    s, plain = th.solve_problem(p, f=ref["f"], precision=MAILLE_FP64)
    assert s == 0
    s, out = th.solve_problem(p, f=ref["f"], precision=MAILLE_MIXED)
    assert s == 0
    assert np.abs(out["temps"] - ref["temps"]).max() < 1e-9 * np.abs(ref["temps"]).max()
    assert (out["iterations"] <= 2 * plain["iterations"]).all()


@pytest.mark.parametrize("threads", ["64", "192"])
def test_a_batch_in_blocks_without_the_correction_is_ic0s(gpu, monkeypatch, threads):
    # the correction's product works in groups of 4 warps: other block sizes run IC(0) alone, with its own
    # threshold of the reliable updates, so the same bits as with the correction switched off
    probs = [bar((3, 3, 18)), bar((4, 4, 16), draw=1)]
    loads = [np.stack([p.loads, np.roll(p.loads, -1)], 1) for p in probs]
    for k, v in (("Q", "2"), ("SUB", "1"), ("TASK", "4"), ("THREADS", threads)):
        monkeypatch.setenv("MAILLE_BATCH_" + k, v)
    out = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("MAILLE_COARSE", knob)
        with mb.BatchSolver(probs, loads, tol=1e-10, precision=MAILLE_MIXED) as b:
            out[knob] = b.solve()
    assert out["0"].info["status_code"] == 0
    assert np.array_equal(out["0"].iterations, out["1"].iterations)
    assert all(np.array_equal(x, y) for x, y in zip(out["0"].displacements, out["1"].displacements))
