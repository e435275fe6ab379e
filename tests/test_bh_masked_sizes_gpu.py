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


# leaves of several bodies, at one place or closer than their keys tell apart, softened enough
# that a body may meet itself in its leaf, and not; theta = 0 adds up every body by itself
@pytest.mark.parametrize("soft", [0.0, 1e-20, 9e-7, 1.1e-6, 0.01])
@pytest.mark.parametrize("n", [600, 40000, 130000])
def test_bodies_of_a_shared_leaf(res, oracle, soft, n):
    from particular_gb300 import AccelerationSoftened
    r = np.random.RandomState(9)
    x = r.normal(size=(n // 10, 3))
    b = np.concatenate([np.repeat(x, 10, axis=0), r.uniform(0.5, 1.5, (n, 1))], 1).astype(np.float32)
    near = r.uniform(-1, 1, (n, 3)) * (r.uniform(0, 1, (n, 1)) < 0.5)  # half of them at one place
    b[:, :3] += (near * 2e-7).astype(np.float32)
    m = cuda.BarnesHut(0.0, res, AccelerationSoftened(soft) if soft else Acceleration.checked())
    got = m.compute(b)
    g = m.export_tree()
    shared = (g["links"][:, 2] < 0) | (g["links"][:, 3] > 1)
    assert ((g["links"][:, 2] >= 0) & shared).sum() > n // 20
    # a node whose centre of mass is a body's place is skipped whole for it, as the reference does
    centres = {tuple(c) for c in g["com_mass"][shared, :3]}
    pick = np.array([i for i in np.linspace(0, n - 1, 200).astype(int) if tuple(b[i, :3]) not in centres])
    assert len(pick) > 100
    want = oracle.bf_f64(b[pick], b, soft, True)
    d = b[None, :, :3].astype(np.float64) - b[pick, None, :3].astype(np.float64)
    r2 = (d * d).sum(-1)
    scale = (b[None, :, 3] * np.sqrt(r2) / np.where(r2 > 0, r2 + float(np.float32(soft)) ** 2, 1.0) ** 1.5).sum(1)
    # per pair 3 rsqrt factors (2^-22 each); a list's 128 entries in two packed halves
    assert np.isfinite(got).all()
    assert (np.abs(got[pick] - want).max(1) <= 1e-5 * scale).all()
