"""The matrix logarithm of the law on both sides of the strain where the
polynomial form hands over to the eigenvalue form (|F F^T - I| = 1/4)."""
import numpy as np
import pytest

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P

pytestmark = pytest.mark.gpu

# thresholds out of reach: the stress is K theta I + 2 G dev(ln V)
ELASTIC = P.nitinol_props(E=60000.0, nu=0.33, eps_L=0.05, Ss_AS=1e9, Sf_AS=2e9, Ss_SA=-1e9, Sf_SA=-2e9)


def _points(norm, n, seed):
    """Symmetric A = F F^T - I with |A|_F = norm, and F = sqrt(I + A) Q."""
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(2 * n, 3, 3)))
    q *= np.sign(np.linalg.det(q))[:, None, None]
    w = rng.normal(size=(n, 3))
    w[: n // 4] = w[: n // 4, :1]                          # volumetric: a triple eigenvalue
    w[n // 4: n // 2, 1] = w[n // 4: n // 2, 0]             # a double eigenvalue
    w *= norm / np.linalg.norm(w, axis=1, keepdims=True)
    w = np.maximum(w, -0.9)
    v = q[:n]
    F = (v * np.sqrt(1.0 + w)[:, None, :]) @ v.transpose(0, 2, 1) @ q[n:]
    lnv = (v * (0.5 * np.log1p(w))[:, None, :]) @ v.transpose(0, 2, 1)
    return F, lnv


@pytest.mark.parametrize("norm", [1e-6, 1e-3, 0.1, 0.2499, 0.2501, 0.6, 1.2])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_stress_of_a_known_strain(precision, norm):
    F, lnv = _points(norm, 512, 3)
    S, _, fl = sma.eval_sld_stress_model_160(ELASTIC, F, np.tile([0.0, 1e12, -1e12], (len(F), 1)), precision=precision)
    assert int(fl.max()) == 0
    E, nu = ELASTIC[0], ELASTIC[1]
    th = np.trace(lnv, axis1=1, axis2=2)[:, None, None] * np.eye(3)
    tau = E / (3 - 6 * nu) * th + E / (1 + nu) * (lnv - th / 3)
    Fi = np.linalg.inv(F)
    ref = Fi @ tau @ Fi.transpose(0, 2, 1)
    err = np.abs(S.cpu().numpy() - ref).max(axis=(1, 2)) / np.abs(ref).max(axis=(1, 2))
    # FP32 rounds F - I = H to 2^-24 |H|, |H| of order one with the rotation,
    # so ln V is known to 2^-24 / norm; some 40 more roundings in the stress
    # and the pull-back.  In FP64 the expected value itself is off by up to
    # 83 / norm units (the orthogonal factors, used five times; measured
    # against the eigenvalues of F F^T - I): three times that.
    tol = 2.0 ** -53 * (256 + 256 / norm) if precision == "fp64" else 2.0 ** -24 * (64 + 32 / norm)
    assert err.max() < tol, err.max()



@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_nan_and_singular_gradients_stay_visible(precision):
    """A NaN or a zero deformation gradient gives no finite stress."""
    F = np.tile(np.eye(3), (3, 1, 1))
    F[0, 0, 0] = np.nan
    F[1] = 0.0
    S = sma.eval_sld_stress_model_160(ELASTIC, F, np.zeros((3, 3)), precision=precision)[0].cpu().numpy()
    assert not np.isfinite(S[0]).all() and not np.isfinite(S[1]).all() and np.abs(S[2]).max() == 0.0
