"""The f64 Barnes-Hut walk where the number of lanes per body changes (16 to 1 by the number of
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


# 16, 8, 4, 2 and 1 lanes per body: the same accepted sets on either side of each turn
@pytest.mark.parametrize("lanes", [16, 8, 4, 2])
def test_lanes_per_body_agree(res, oracle, lanes):
    slots = 20 * 32 * res.sm_count
    turn = {16: slots // 16, 8: slots // 8, 4: 5 * slots // 8, 2: 4 * slots}[lanes]
    src = cloud(300, 6)
    aff = cloud(turn + 1, 7)
    m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.0), dvec3=True)
    want, acc = oracle.bh_dvec3(aff, src, 0.7, 0.0, True, accepted=True)
    for n in (turn, turn + 1):
        got = m.compute(Between(aff[:n], src))
        assert m.stats()["interactions"] == int(acc[:n].sum())
        mag = np.linalg.norm(want[:n], axis=1)
        assert (np.linalg.norm(got - want[:n], axis=1) <= 1e-13 * np.maximum(mag, np.median(mag))).all()


def accepted_pairs(g, b, theta):
    """Pairs that the reference's rule accepts on the exported tree: a node at distance zero is
    skipped, a cell opened where theta^2 d^2 < w^2, all in f64."""
    total, stack = 0, [(0, len(g["links"]), np.arange(len(b)))]
    while stack:
        node, end, who = stack.pop()
        while node < end and len(who):
            d = g["com_mass"][node, :3] - b[who, :3]
            d2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
            after, w = int(g["links"][node, 1]), g["width"][node]
            opens = (d2 > 0) & (theta * theta * d2 < w * w) & bool(g["links"][node, 2] < 0)
            total += int(((d2 > 0) & ~opens).sum())
            stack.append((node + 1, after, who[opens]))
            node = after
    return total


# Decisions at the line: a lattice whose cells' centres of mass lie at distances where
# theta^2 d^2 equals w^2, the same off by a last bit, and far from the origin; products that
# leave FP32's range
@pytest.mark.parametrize("theta", [0.0, 0.5, 1.0, 1e-18])
@pytest.mark.parametrize("kind", ["lattice", "nudged", "far", "huge", "tiny"])
def test_decisions_at_the_line(res, theta, kind):
    g = np.stack(np.meshgrid(*[np.arange(10.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    if kind == "nudged":
        r = np.random.default_rng(5)
        g = np.where(r.random(g.shape) < 0.5, np.nextafter(g, 100.0), g)
    elif kind == "far":
        g = g + 3.0 * 2.0 ** 30
    elif kind != "lattice":
        g = g * (1e18 if kind == "huge" else 1e-19)
    b = np.concatenate([g, np.ones((len(g), 1))], 1)
    m = cuda.BarnesHut(theta, res, AccelerationSoftened(0.0), dvec3=True)
    assert np.isfinite(m.compute(b)).all()
    assert m.stats()["interactions"] == accepted_pairs(m.export_tree_dvec3(), b, theta)
