"""The step's time data is made by one warp beside the elements: more time
functions than lanes hold in one turn (3 directions each), and ranges of
elements around the wide instance's limit of 64 elements per SM."""
import dataclasses

import numpy as np
import pytest

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfun", [1, 10, 11, 16])
def test_many_time_functions(oracle, nfun):
    p = P.bar_40x4x4(nsteps=60)
    tip = P.face_nodes(p.coord, 0, 40.0)
    fixno, bcfun = p.fixno.copy(), np.full(p.npoin, -1, np.int32)
    fixno[tip] = 1
    bcfun[tip] = np.arange(tip.size) % nfun
    t = 60 * p.dtime
    tabs = [np.array([[0, 0, 0, 0], [0.3 * t, 0.02 * (f + 1), 0.001 * f, -0.001 * f], [t, 0.01, 0, 0]])
            for f in range(nfun)]
    q = dataclasses.replace(p, fixno=fixno, bcfun=bcfun, fun_npts=np.full(nfun, 3, np.int32),
                            fun_smooth=(np.arange(nfun) % 2).astype(np.int32), fun_tab=np.concatenate(tabs))
    o = oracle.Problem(q)
    o.run(q.dtime, 40)
    g = sma.ExplicitSolid(q, precision="fp64")
    for n in (1, 9, 30):                                     # eager steps, one graph, several
        g.step(n)
    d = g.get("displ")
    assert np.abs(d - o.displ).max() <= 1e-9 * np.abs(o.displ).max()
    assert abs(g.time - 40 * q.dtime) <= 1e-12 * t


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ny", [12, 13])
def test_either_side_of_the_wide_instance(oracle, ny, precision):
    """60 x 12 x 13 = 9,360 and 60 x 13 x 13 = 10,140 elements (148 SMs: 9,472)."""
    coord, lnods = P.structured_box(60, ny, 13, 60.0, float(ny), 13.0, 0.05, 3)
    b = P.bar_40x4x4()
    npo = len(coord)
    fixno = np.zeros((npo, 3), np.int32)
    fixno[P.face_nodes(coord, 0, 0.0)] = 1
    p = dataclasses.replace(b, coord=coord, lnods=lnods, fixno=fixno, bcfun=np.full(npo, -1, np.int32))
    u = P.prestrain(p, 0.012)
    g = sma.ExplicitSolid(p, precision=precision)
    r, ref = g.assemble(u)["rhsid"], oracle.Problem(p).assemble(u)["rhsid"]
    scale = np.abs(ref).max()
    assert np.abs(r - ref).max() <= (1e-8 if precision == "fp64" else 1e-3) * scale
