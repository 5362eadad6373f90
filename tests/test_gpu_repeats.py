"""Elements that name a node twice, through the C ABI (Model refuses them: their edges are not straight): a
Tet10 whose mid nodes of two edges are one node. Its blocks of that node meet in one place of the matrix,
and all of them count, as in the oracle's assembly."""
import ctypes

import numpy as np
import pytest

from maille_b200 import _lib, meshgen as mg
from maille_b200.batch import BatchSolver
from maille_b200.model import _result_struct, problem_struct
from maille_b200.thermal import solve_problem

gpu_only = pytest.mark.gpu


def collapse(conn, every):
    """Every `every`-th element takes its last mid node for the one of its fourth edge too; also the nodes
    that no element names any more. At its Gauss points the Jacobian's determinant is 0.17 to 0.72 of the
    straight element's in size."""
    conn = conn.copy()
    conn[::every, 7] = conn[::every, 9]
    return conn, np.setdiff1d(np.arange(conn.max() + 1), conn)


def elastic(every=7):
    p = mg.clamped_cube((4, 3, 3), True, 50000.0 + 150000.0 * mg.uniform(41, 6 * 36), size=(1.2, 0.9, 1.0))
    p.conn, unused = collapse(p.conn, every)
    p.fixed.reshape(-1, 3)[unused] = 1
    p.loads = 0.01 * (mg.uniform(43, 3 * p.n_nodes) - 0.5) * (p.fixed == 0)
    p.p_elem, p.p_face, p.p_value = (a[:0] for a in (p.p_elem, p.p_face, p.p_value))
    return p


def test_the_collapsed_elements_have_a_volume():
    p = elastic()
    a, b = (5.0 + 3.0 * np.sqrt(5.0)) / 20.0, (5.0 - np.sqrt(5.0)) / 20.0
    dl = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    straight, here = [], []
    for g in range(4):
        l = np.full(4, b)
        l[g] = a
        d = np.empty((10, 3))
        d[:4] = (4.0 * l - 1.0)[:, None] * dl
        for k, (s, t) in enumerate(mg.TET10_EDGES):
            d[4 + k] = 4.0 * (l[s] * dl[t] + l[t] * dl[s])
        x = p.coords[p.conn]
        here.append(np.linalg.det(np.einsum("ai,nar->nir", d, x)))
        straight.append(np.linalg.det(np.einsum("ai,nar->nir", dl, x[:, :4])))
    ratio = np.abs(np.array(here) / np.array(straight))[:, ::7]
    assert 0.17 < ratio.min() and ratio.max() < 0.73


@gpu_only
@pytest.mark.parametrize("every", [7, 1])
def test_an_elastic_solve_counts_every_block(gpu, oracle_lib, every):
    # 1e-10 of the oracle at 1e-13, the tolerance of the parity tests
    p = elastic(every)
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-13)
    assert ref["status"] == 0
    s, keep = problem_struct(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads, tol=1e-13)
    r, out = _result_struct(p.n_nodes, p.n_elems, 4)
    assert gpu.maille_gpu_elastic_solve(ctypes.byref(s), ctypes.byref(r)) == 0, _lib.last_error()
    assert np.linalg.norm(out["u"] - ref["u"]) < 1e-10 * np.linalg.norm(ref["u"])
    assert np.linalg.norm(out["reactions"] - ref["reactions"]) < 1e-10 * np.linalg.norm(ref["reactions"])


@gpu_only
def test_a_batch_counts_every_block(gpu, oracle_lib):
    p = elastic()
    ref = oracle_lib.model_solve(p, solver=2, tol=1e-13)
    with BatchSolver([p, elastic(3)], [p.loads[:, None], p.loads[:, None]], tol=1e-13) as b:
        f = b.solve()
    assert f.info["status_code"] == 0
    assert np.linalg.norm(f.displacements[0][:, 0] - ref["u"]) < 1e-10 * np.linalg.norm(ref["u"])


@gpu_only
@pytest.mark.parametrize("every", [7, 1])
def test_a_thermal_step_counts_every_entry(gpu, oracle_lib, every):
    # 1e-9 of the largest temperature, as the thermal parity tests
    p = mg.thermal_cube(4, True, increments=2, time_period=0.1)
    p.conn, unused = collapse(p.conn, every)
    p.fixed[unused] = 1
    p.c_elem, p.c_face, p.c_film, p.c_sink = (a[:0] for a in (p.c_elem, p.c_face, p.c_film, p.c_sink))
    ref = oracle_lib.thermal_transient(p, solver=2)
    s, out = solve_problem(p, f=ref["f"])
    assert s == 0
    assert np.abs(out["temps"] - ref["temps"]).max() < 1e-9 * np.abs(ref["temps"]).max()
