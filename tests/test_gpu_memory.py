"""The library's device memory pool (memory.cu): handles reuse the memory their predecessors
freed, and maille_gpu_trim_memory hands the unused part back without disturbing later solves."""
import ctypes

import numpy as np
import pytest
import torch

import maille_b200 as mb
from maille_b200 import _lib
from maille_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def solve_once(p):
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                             (p.p_elem, p.p_face, p.p_value))
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(1e-12)
    return m.solve()


def test_repeated_handles_reuse_the_pool_and_trim_returns_it(gpu):
    L = _lib.load()
    p = mg.mixed_tet10(6)
    first = solve_once(p).displacements
    free_after_first = torch.cuda.mem_get_info(0)[0]
    for _ in range(3):  # create / solve / destroy again: same result, no growth of reserved memory
        again = solve_once(p).displacements
        assert np.array_equal(again, first)
        assert torch.cuda.mem_get_info(0)[0] >= free_after_first - (64 << 20)
    assert L.maille_gpu_trim_memory(0) == _lib.MAILLE_OK, _lib.last_error()
    assert torch.cuda.mem_get_info(0)[0] >= free_after_first  # the pool's reserve went back
    assert np.array_equal(solve_once(p).displacements, first)  # and the pool refills on demand


@pytest.mark.parametrize("cells", [20, 24, 25])
def test_large_copies_give_the_bytes_of_small_ones(gpu, cells):
    # results below, around and above the size from which copies are shared by threads (4 MB; the last piece
    # of 2 MB is a partial one), to page-locked and to pageable buffers: the same bytes
    p = mg.mixed_tet10(cells)
    m = mb.Model.from_arrays(p.coords, p.conn, p.young, p.poisson, p.fixed, p.imposed, p.loads,
                             (p.p_elem, p.p_face, p.p_value))
    m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(1e-6)
    with mb.SolverHandle(m) as h:
        a = h.solve()
        pinned = [torch.zeros(x.shape, dtype=torch.float64).pin_memory().numpy()
                  for x in (a.displacements, a.reactions, a.stresses, a.von_mises)]
        r = _lib.ElasticResult(u=_lib.ptr(pinned[0], _lib._d), reactions=_lib.ptr(pinned[1], _lib._d),
                               gauss_stress=_lib.ptr(pinned[2], _lib._d), von_mises=_lib.ptr(pinned[3], _lib._d))
        f = np.ascontiguousarray(h._f)
        assert h._L.maille_gpu_solve(h._h, _lib.ptr(f, _lib._d), ctypes.byref(r)) == 0, _lib.last_error()
    for x, y in zip((a.displacements, a.reactions, a.stresses, a.von_mises), pinned):
        assert np.array_equal(x, y)
