"""The reference-rule walk where the bodies per warp change with the number of targets (2 to
64, the last groups of the larger two in halves), in last warps that are not full."""
import numpy as np
import pytest

from particular_gb300 import Acceleration, Between, cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quad", [False, True])
def test_sizes_agree_with_the_oracle(res, oracle, quad):
    r = np.random.RandomState(8)
    src = np.concatenate([r.normal(size=(3000, 3)), r.uniform(0.5, 1.5, (3000, 1))], 1).astype(np.float32)
    src[7] = src[8]  # two bodies at one place: a leaf of several bodies
    m = cuda.BarnesHut(0.8, res, Acceleration.checked(), quadrupole=quad)
    tree = m.build(src)
    sms = res.sm_count
    sizes = [1, 3, 9, 40 * sms, 40 * sms + 1, 80 * sms, 80 * sms + 1, 160 * sms, 160 * sms + 1, 432 * sms + 17, 3520 * sms, 3520 * sms + 33]
    probe = np.concatenate([src[:200], np.concatenate([r.normal(size=(56, 3)), np.zeros((56, 1))], 1)]).astype(np.float32)
    want = cuda.BarnesHut(0.8, res, Acceleration.checked(), quadrupole=quad).compute(Between(probe, src))
    tree = m.build(src)
    ref, acc = oracle.bh_f32(probe, src, 0.8, 0.0, True, accepted=True)
    per = None
    for n in sizes:
        # the probe over and over: copies of a body are neighbours in key order
        tgt = probe[np.arange(n) % len(probe)]
        got = m.compute(Between(tgt, tree))
        st = m.stats()
        assert np.isfinite(got).all()
        if n >= len(probe):
            per = st["interactions"] / n
            assert abs(per - acc.mean()) <= 5e-3 * acc.mean()
        # the same accepted nodes, summed in another order and in other partial sums
        scale = np.linalg.norm(want, axis=1)[np.arange(n) % len(probe)]
        d = np.linalg.norm(got.astype(np.float64) - want[np.arange(n) % len(probe)], axis=1)
        assert np.median(d / scale) <= 2e-7 and (d <= 1e-5 * np.maximum(scale, np.median(scale))).all()
    if not quad:
        d = np.linalg.norm(want - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert np.median(d) < 1e-5
