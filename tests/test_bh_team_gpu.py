"""The group walk with 8, 4 or 1 warps per group, which the number of groups decides: the
same groups are walked among few, some and many others and keep their accelerations."""
import numpy as np
import pytest

from particular_gb300 import Acceleration, AccelerationSoftened, Between, cuda

pytestmark = pytest.mark.gpu


def scattered(r, n, lo, hi, mass):
    return np.concatenate([r.uniform(lo, hi, (n, 3)), np.full((n, 1), mass)], 1).astype(np.float32)


@pytest.mark.parametrize("soft", [0.0, 0.01])
@pytest.mark.parametrize("kw", [{}, {"quadrupole": True}, {"quadrupole": True, "local": True},
                                {"relative": 2.5e-3}, {"quadrupole": True, "local": True, "relative": 2.5e-3}])
def test_team_sizes_agree(res, kw, soft):
    r = np.random.RandomState(4)
    src = scattered(r, 30000, -1, 1, 1 / 30000)
    src[0, :3], src[1, :3] = -1, 1  # a root box about the origin
    # 50 full groups of targets in the half x < 0, sources among them; the others' keys are
    # the highest (x, y, z >= 0), so they fill groups of their own
    tgt = src[src[:, 0] < -0.05][:3200]
    assert len(tgt) == 3200
    it = AccelerationSoftened(soft) if soft else Acceleration.checked()
    m = cuda.BarnesHut(0.7, res, it, group=True, **kw)
    tree = m.build(src)
    sms = res.sm_count
    got = {}
    for groups in (50, 5 * sms // 2 + 1, 11 * sms + 1):  # 8, 4 and 1 warps per group
        more = scattered(r, 64 * (groups - 50), 0.1, 1, 0)
        out = m.compute(Between(np.concatenate([tgt, more]), tree))
        assert np.isfinite(out).all()
        st = m.stats()
        assert st["overflow"] == 0 and st["warps"] == groups
        got[groups] = out[:3200]
    want = got[11 * sms + 1].astype(np.float64)
    # the same nodes, added in another order: compensated sums, local expansions to a few
    # roundings of their 19 coefficients
    scale = np.linalg.norm(want, axis=1) + np.median(np.linalg.norm(want, axis=1))
    for out in got.values():
        assert (np.linalg.norm(out - want, axis=1) <= 2e-6 * scale).all()


@pytest.mark.parametrize("kw", [{"relative": 2.5e-3}, {"quadrupole": True, "relative": 2.5e-3},
                                {"quadrupole": True, "local": True, "relative": 2.5e-3}, {},
                                {"quadrupole": True, "local": True}])
def test_order_of_the_groups_does_not_show(res, kw):
    """From 20 groups per SM on (24 without an error bound) the walk takes them by how much each
    is likely to open; every group keeps its accelerations, to the bit, and none is left out."""
    r = np.random.RandomState(5)
    src = scattered(r, 30000, -1, 1, 1 / 30000)
    src[0, :3], src[1, :3] = -1, 1
    tgt = src[src[:, 0] < -0.05][:3200]
    m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.01), group=True, **kw)
    tree = m.build(src)
    turn = (20 if "relative" in kw else 24) * res.sm_count
    want = None
    for groups, last in ((turn, 64), (turn + 1, 64), (turn + 257, 1)):
        more = scattered(r, 64 * (groups - 51) + last, 0.1, 1, 0)
        more[::3, :3] *= 1000.0 / more[::3, :3].max()  # far outside the box: keys of many octaves
        out = m.compute(Between(np.concatenate([tgt, more]), tree))
        assert m.stats()["warps"] == groups
        assert np.isfinite(out).all() and (out != 0).any(1).all()
        want = out[:3200] if want is None else want
        assert np.array_equal(out[:3200].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("quadrupole", [False, True])
def test_order_of_the_masked_walk_does_not_show(res, quadrupole):
    """The same for the reference's rule: 16 bodies a warp in tree order and by width, 32 and 64
    by width with the last ones in halves."""
    r = np.random.RandomState(6)
    src = scattered(r, 30000, -1, 1, 1 / 30000)
    src[0, :3], src[1, :3] = -1, 1
    tgt = src[src[:, 0] < -0.05][:3200]
    m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.01), quadrupole=quadrupole)
    tree = m.build(src)
    want = None
    for n in (24 * 16 * res.sm_count, 24 * 16 * res.sm_count + 1, 24 * 32 * res.sm_count + 31,
              110 * 32 * res.sm_count + 1):
        more = scattered(r, n - 3200, 0.1, 1, 0)
        more[::3, :3] *= 1000.0 / more[::3, :3].max()
        out = m.compute(Between(np.concatenate([tgt, more]), tree))
        assert np.isfinite(out).all() and (out != 0).any(1).all()
        got, want = out[:3200].astype(np.float64), out[:3200].astype(np.float64) if want is None else want
        # the same nodes, added in another order: compensated sums
        scale = np.linalg.norm(want, axis=1) + np.median(np.linalg.norm(want, axis=1))
        assert (np.linalg.norm(got - want, axis=1) <= 2e-6 * scale).all()


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("turn", [24 * 32, 110 * 32])
def test_ordered_walks_repeat_to_the_bit(res, quadrupole, turn):
    """The reference's rule with its groups (of 32 bodies, of 64) taken in order and the last
    ones halved: a call gives the same bits every time, and graph-replayed steps those of eager
    ones."""
    import torch
    from particular_gb300 import _native as N
    L, n = N.lib(), turn * res.sm_count + 31
    r = np.random.RandomState(7)
    x = r.normal(size=(n, 3)) * r.uniform(0.1, 1, (n, 1))
    b = torch.from_numpy(np.concatenate([x, np.full((n, 1), 1 / n)], 1).astype(np.float32)).cuda()
    fl = N.PT_BH_QUADRUPOLE if quadrupole else 0
    outs = [torch.empty((n, 3), device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    for o in outs:
        N.check(L.pt_bh_accel_f32_device(res.handle, b.data_ptr(), n, b.data_ptr(), n, 0.9, 0.01, fl, o.data_ptr()))
    res.synchronize()
    assert all(torch.equal(outs[0].view(torch.int32), o.view(torch.int32)) for o in outs[1:])
    end = []
    for use_graph in (0, 1):
        p, v, a = b.clone(), torch.zeros((n, 4), device="cuda"), outs[0].clone()
        torch.cuda.synchronize()
        for _ in range(2):
            N.check(L.pt_leapfrog_device(res.handle, p.data_ptr(), v.data_ptr(), a.data_ptr(), n, 1e-3, 2,
                                         N.PT_METHOD_BARNES_HUT, 0.9, 0.01, fl, use_graph))
        res.synchronize()
        end.append((p, v, a))
    for e, g in zip(*end):
        assert torch.equal(e.view(torch.int32), g.view(torch.int32))
