"""Autotuner bookkeeping that needs no GPU: size buckets and the cache."""
import dataclasses

import numpy as np

from alya_sma_b200 import problem as P
from alya_sma_b200 import tune


def test_buckets_are_powers_of_two():
    assert tune.bucket(1) == 1
    assert tune.bucket(640000) == 1 << 19
    assert tune.bucket(1998848) == 1 << 21
    assert tune.bucket(800) == tune.bucket(1200)


def test_cache_round_trip(tmp_path, monkeypatch):
    monkeypatch.setenv("ALYA_SMA_CACHE", str(tmp_path))
    assert tune.load_cache() == {}
    tune.save_cache({"fp32/cd/1024": {"block": 128, "scatter": "atomic"}})
    assert tune.load_cache()["fp32/cd/1024"]["block"] == 128
    assert tune.cache_path().startswith(str(tmp_path))


def test_key_tells_apart_what_decides_the_kernel():
    """Precision, scheme, size, damping and the material layout; entries of
    other candidates or kernels (keys of another form) are never read."""
    p = P.bar_40x4x4(nsteps=4)
    ne = p.nelem
    many = dataclasses.replace(p, props=np.tile(p.props, (ne, 1)), lmate=np.arange(ne, dtype=np.int32))
    few = dataclasses.replace(p, props=np.tile(p.props, (3, 1)), lmate=np.arange(ne, dtype=np.int32) % 3)
    damped = dataclasses.replace(p, dampi=np.array([[1e4, 0.0]]))
    keys = [tune._key("fp32", "cd", q) for q in (p, many, few, damped)]
    keys += [tune._key("fp64", "cd", p), tune._key("fp32", "tw", p)]
    assert len(set(keys)) == len(keys)
    assert tune._key("fp32", "cd", dataclasses.replace(p, dampi=np.zeros((1, 2)))) == keys[0]
    assert all(k.startswith(f"{tune.GENERATION}/") for k in keys)


def test_candidates_hold_the_librarys_own_choice():
    assert (0, "atomic", "auto") in tune.CANDIDATES
    assert any(v == "auto" and 0 < b <= 64 for b, _, v in tune.CANDIDATES)
