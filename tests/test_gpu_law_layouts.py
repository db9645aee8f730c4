"""The material plugin on row-major, column-major and strided deformation
gradients, at point counts around a block's 128 points (16 with the tangent)."""
import numpy as np
import pytest

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P

pytestmark = pytest.mark.gpu

NITI = P.nitinol_props(**P.NITI, C_AS=5.0, C_SA=5.0, T_ref=300.0)


def _points(n, seed=1):
    import torch
    rng = np.random.default_rng(seed)
    F = np.eye(3) + 0.02 * rng.normal(size=(n, 3, 3))
    s = np.stack([rng.choice([0.0, 0.4, 1.0], n), rng.uniform(100, 400, n), rng.uniform(100, 400, n)], 1)
    dev = dict(dtype=torch.float64, device="cuda")
    return torch.tensor(F, **dev), torch.tensor(s, **dev), torch.tensor(rng.uniform(300, 310, n), **dev)


@pytest.mark.parametrize("flagt,precision,sizes", [(0, "fp64", (1, 127, 128, 129, 1000)),
                                                   (0, "fp32", (1, 127, 128, 129, 1000)),
                                                   (1, "fp64", (1, 15, 16, 17, 129))])
def test_layouts_give_the_same_points(flagt, precision, sizes):
    import torch
    for n in sizes:
        F, s, t = _points(n)
        kw = dict(gptmp=t, flagt=flagt, e_mart=40000.0, precision=precision)
        ref = sma.eval_sld_stress_model_160(NITI, F, s, **kw)
        col = F.transpose(1, 2).contiguous().transpose(1, 2)          # column-major in memory
        wide = torch.full((n, 5, 4), 7.0, dtype=torch.float64, device="cuda")
        wide[:, 1:4, :3] = F
        for G in (col, wide[:, 1:4, :3], F.cpu().numpy()):
            out = sma.eval_sld_stress_model_160(NITI, G, s, **kw)
            for x, y in zip(out, ref):
                assert torch.equal(x, y), n
        # a point's result does not depend on its place or neighbours
        last = sma.eval_sld_stress_model_160(NITI, F[-1:], s[-1:], **dict(kw, gptmp=t[-1:]))
        for x, y in zip(last, ref):
            assert torch.equal(x[0], y[-1]), n
