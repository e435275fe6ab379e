"""Ensembles of sizes around the j-tile and the quads it is read by, from fewer items than SMs
to more than the chip holds at once: each system as its own brute-force leapfrog."""
import numpy as np
import pytest

from test_ensemble_gpu import run_each, run_ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 0.05])
@pytest.mark.parametrize("sizes", [[1], [2, 3], [4, 5, 6, 7, 127, 128, 129, 255, 256, 257, 513],
                                   [64 + k % 70 for k in range(900)]])
def test_systems_match_their_own_leapfrog(res, sizes, eps):
    r = np.random.RandomState(len(sizes))
    n = sum(sizes)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    b = np.concatenate([r.uniform(-1, 1, (n, 3)), r.uniform(0.5, 1.5, (n, 1)) / 100], 1).astype(np.float32)
    v = np.concatenate([r.normal(size=(n, 3)) * 0.1, np.zeros((n, 1))], 1).astype(np.float32)
    if len(sizes) > 100:  # the whole ensemble against itself, system by system, on a few of them
        eb, ev = run_ensemble(res, offsets, b, v, 2, eps=eps, dt=1e-4)
        for k in (0, 1, 69, 450, 899):
            s, e = int(offsets[k]), int(offsets[k + 1])
            rb, rv = run_each(res, np.array([0, e - s], np.uint32), b[s:e], v[s:e], 2, eps=eps, dt=1e-4)
            assert np.abs(eb[s:e] - rb).max() < 1e-5 and np.abs(ev[s:e] - rv).max() < 1e-4 * (1 + np.abs(rv).max())
        assert np.isfinite(eb).all() and np.isfinite(ev).all()
        return
    eb, ev = run_ensemble(res, offsets, b, v, 2, eps=eps, dt=1e-4)
    rb, rv = run_each(res, offsets, b, v, 2, eps=eps, dt=1e-4)
    assert np.abs(eb - rb).max() < 1e-5 and np.abs(ev - rv).max() < 1e-4 * (1 + np.abs(rv).max())
