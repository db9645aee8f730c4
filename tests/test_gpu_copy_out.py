"""Arrays handed back to pageable and page-locked host memory: sizes around
the smallest that goes through the context's page-locked pieces (2 MB) and
around whole pieces (256 KB)."""
import threading

import numpy as np
import pytest

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P

pytestmark = pytest.mark.gpu


def _one_element(npoin):
    coord, lnods = P.structured_box(1, 1, 1, 1.0, 1.0, 1.0)
    coord = np.concatenate([coord, np.zeros((npoin - 8, 3))])   # the other nodes belong to no element
    props = P.nitinol_props(**P.NITI)[None, :]
    return P.Problem(coord=coord, lnods=lnods, props=props, e_mart=np.zeros(1), densi=np.array([P.NITI_DENSITY]),
                     fixno=np.zeros((npoin, 3), np.int32), bcfun=np.full(npoin, -1, np.int32),
                     fun_npts=np.array([2], np.int32), fun_smooth=np.array([0], np.int32),
                     fun_tab=np.array([[0.0, 0, 0, 0], [1.0, 0, 0, 0]]), dtime=1e-8)


@pytest.mark.parametrize("npoin", [8, 87_381, 87_382, 98_304, 98_305, 700_001])
def test_nodal_arrays_come_back_whole(npoin):
    import torch
    s = sma.ExplicitSolid(_one_element(npoin))
    u = np.random.default_rng(npoin).normal(size=(npoin, 3))
    s.set("displ", u)
    for _ in range(2):
        assert np.array_equal(s.get("displ"), u)
    pinned = torch.empty((npoin, 3), dtype=torch.float64, pin_memory=True).numpy()
    sma._check(sma.lib().sma_get_nodal(s._ctx, sma.FIELD["displ"], pinned.ctypes.data))
    assert np.array_equal(pinned, u)
    s.close()


def test_two_contexts_in_two_threads():
    sizes, got = (200_003, 150_001), {}

    def work(n):
        s = sma.ExplicitSolid(_one_element(n))
        u = np.random.default_rng(n).normal(size=(n, 3))
        s.set("veloc", u)
        got[n] = all(np.array_equal(s.get("veloc"), u) for _ in range(5))
        s.close()

    th = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert all(got.get(n) for n in sizes)
