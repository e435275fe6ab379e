"""The f64 Barnes-Hut walk where the number of lanes per body changes (4, 2, 1 by the number of
targets), in a last warp that is not full, and with softened distances outside FP32's range."""
import numpy as np
import pytest

from particular_gb300 import AccelerationSoftened, Between, cuda

pytestmark = pytest.mark.gpu


def cloud(n, seed, scale=1.0):
    r = np.random.default_rng(seed)
    return np.concatenate([r.normal(scale=scale, size=(n, 3)), r.uniform(0.5, 1.5, (n, 1))], 1)


@pytest.mark.parametrize("n_aff,scale", [(1, 1.0), (9, 1.0), (24320, 1.0), (24321, 1.0), (48640, 1.0), (48641, 1.0),
                                         (333, 1e22), (333, 1e-22)])
def test_walk_matches_reference(res, oracle, n_aff, scale):
    src = cloud(1500, 3, scale)
    aff = cloud(n_aff, 4, scale)
    aff[: min(n_aff, 40)] = src[: min(n_aff, 40)]
    m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.0), dvec3=True)
    got = m.compute(Between(aff, src))
    want, acc = oracle.bh_dvec3(aff, src, 0.7, 0.0, True, accepted=True)
    assert m.stats()["interactions"] == int(acc.sum())
    # the terms and their sum each within some 2^-52 of the terms' magnitudes; bodies whose
    # terms cancel lose digits in both, so against the typical acceleration
    mag = np.linalg.norm(want, axis=1)
    assert (np.linalg.norm(got - want, axis=1) <= 1e-13 * np.maximum(mag, np.median(mag))).all()
