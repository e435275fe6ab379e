"""The tree build where its blocks end: chunks of 512 leaf units and blocks of 64 chunks
(32768 units), full, one short and one over; massless and coincident bodies across them."""
import numpy as np
import pytest

from particular_gb300 import AccelerationSoftened, cuda
from test_bh_gpu import oracle_preorder

pytestmark = pytest.mark.gpu


def tree_of(res, b):
    m = cuda.BarnesHut(0.5, res, AccelerationSoftened(0.01), quadrupole=True)
    m.compute(b)
    return m.export_tree()


def clumpy(n, seed):
    """Dense knots in a wide cloud: cells of many levels across every block boundary."""
    r = np.random.RandomState(seed)
    knot = r.uniform(-50, 50, (max(1, n // 700), 3))
    x = knot[r.randint(0, len(knot), n)] + r.normal(size=(n, 3)) * 10.0 ** r.uniform(-3, 1, (n, 1))
    return np.concatenate([x, r.uniform(0.5, 1.5, (n, 1))], 1).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 3, 511, 512, 513, 1025, 32767, 32768, 32769, 70001])
def test_tree_and_moments(res, oracle, n):
    b = clumpy(n, n)
    b[::7, 3] = 0.0  # massless bodies; below also whole massless cells
    b[: n // 10, 3] = 0.0
    g = tree_of(res, b)
    order, e = oracle_preorder(oracle.Tree(b))
    internal = e["internal"][order].astype(bool)
    cells = g["links"][:, 2] < 0
    assert np.array_equal(internal, cells)
    skip = np.asarray(g["links"][:, 1], np.int64)
    assert skip[0] == len(skip) and (skip > np.arange(len(skip))).all()
    w_ref = (e["box"][order, 3] - e["box"][order, 0])[internal]
    assert np.array_equal(g["width"][cells], w_ref.astype(np.float32))
    assert np.array_equal(g["com_mass"][~cells], e["data"][order][~internal])
    # mass and centre of mass of each cell's bodies (their plain mean where massless)
    rng, bp = e["range"][order][internal], b[e["perm"]].astype(np.float64)
    got, w = g["com_mass"][cells].astype(np.float64), g["width"][cells].astype(np.float64)
    for k in np.unique(np.linspace(0, len(rng) - 1, 4000).astype(int)) if len(rng) else []:
        x = bp[rng[k, 0]: rng[k, 0] + rng[k, 1]]
        M = x[:, 3].sum()
        com = (x[:, :3] * x[:, 3:]).sum(0) / M if M else x[:, :3].mean(0)
        assert abs(got[k, 3] - M) <= 1e-6 * M
        # f32 coordinates, and sums about the cell's centre
        assert np.abs(got[k, :3] - com).max() <= 2.0 ** -23 * np.abs(com).max() + 1e-6 * w[k]


@pytest.mark.parametrize("copies", [2, 600])
def test_coincident_bodies_across_blocks(res, copies):
    """Bodies that share a key make one leaf of several bodies, wherever its run lies."""
    b = np.repeat(clumpy(40000 // copies, 5), copies, axis=0)
    b[:, 3] = np.random.RandomState(6).uniform(0.5, 1.5, len(b))
    g = tree_of(res, b)
    cells = g["links"][:, 2] < 0
    assert g["links"][~cells, 3].sum() == len(b) and (~cells).sum() == len(b) // copies
    M = b[:, 3].astype(np.float64).sum()
    com = (b[:, :3].astype(np.float64) * b[:, 3:]).sum(0) / M
    assert abs(g["com_mass"][0, 3] - M) <= 1e-6 * M
    assert np.abs(g["com_mass"][0, :3] - com).max() <= 1e-5


def reference_order(b):
    """Bodies in ascending key order: the root box and 21 subdivisions in the build's f32 ops."""
    x = b[:, :3]
    mn, mx = x.min(0), x.max(0)
    c = (mn + mx) * np.float32(0.5)
    half = np.float32((mx - mn).max()) * np.float32(0.5)
    lo, hi = np.tile(c - half, (len(b), 1)), np.tile(c + half, (len(b), 1))
    key = np.zeros(len(b), np.uint64)
    for _ in range(21):
        c = (lo + hi) * np.float32(0.5)
        left = x < c
        hi, lo = np.where(left, c, hi), np.where(left, lo, c)
        o = left[:, 0] + 2 * left[:, 1].astype(int) + 4 * left[:, 2].astype(int)
        key = (key << np.uint64(3)) | (7 - o).astype(np.uint64)
    return np.argsort(key, kind="stable"), key


# tiles of 256 keys, from 16385 on of 1024, from 65537 on of 2048, three launches a pass from
# 262145 on; and clusters so much smaller than the box that their keys share the upper bits
# the passes sort, in runs short and long
@pytest.mark.parametrize("n", [1, 255, 257, 2047, 2048, 2049, 16384, 16385, 65536, 65537, 131072, 131073, 262144,
                               262145])
@pytest.mark.parametrize("kind", ["cube", "runs", "core"])
def test_bodies_are_in_key_order(res, n, kind):
    r = np.random.RandomState(n)
    x = r.uniform(-1, 1, (n, 3))
    if kind == "runs":  # knots of 1 to 30 bodies, 1e-5 of the box wide
        x = np.repeat(x, r.randint(1, 31, n), axis=0)[:n] + r.uniform(-1e-5, 1e-5, (n, 3))
        x = x[r.permutation(n)]
    elif kind == "core":  # all but a few within 1e-5 of the box
        x[20:] *= 1e-5
    b = np.concatenate([x, np.ones((n, 1))], 1).astype(np.float32)
    order, key = reference_order(b)
    g = tree_of(res, b)
    leaves = g["links"][:, 2] < 0
    first, count = g["links"][~leaves, 2], g["links"][~leaves, 3]
    assert count.sum() == n and np.array_equal(first, np.cumsum(count) - count)
    assert np.array_equal(count, np.unique(key, return_counts=True)[1])
    single = count == 1
    assert np.array_equal(g["com_mass"][~leaves][single], b[order[first[single]]])


# runs of bodies that share the bits the sort's passes sort, of lengths about those where
# another kernel takes the run: a thread per body, a block, a cluster of blocks, one and
# several tiles
@pytest.mark.parametrize("seed,long", [(0, 0), (1, 20000), (2, 70001), (3, 300000)])
def test_long_runs_of_close_bodies_are_in_key_order(res, seed, long):
    r = np.random.RandomState(seed)
    lengths = np.array([1, 2, 127, 128, 129, 130, 255, 256, 257, 2047, 2048, 2049, 4095, 4096, 4097, 4098, 16384, 16385,
                        1 + long])
    lengths = r.permutation(np.concatenate([lengths, r.randint(1, 400, 60)]))
    cell = 2.0 ** -13  # the box is [-1, 1]: cells of the 14th level
    knot = (r.randint(-8000, 8000, (len(lengths), 3)) + 0.5) * cell
    x = np.repeat(knot, lengths, axis=0) + r.uniform(-0.12, 0.12, (lengths.sum(), 3)) * cell
    x = np.concatenate([x, [[-1, -1, -1], [1, 1, 1]]])[r.permutation(lengths.sum() + 2)]
    b = np.concatenate([x, np.ones((len(x), 1))], 1).astype(np.float32)
    order, key = reference_order(b)
    runs = np.unique(key >> np.uint64(23), return_counts=True)[1]
    assert np.isin([128, 129, 130, 4096, 4097], runs).all() and runs.max() >= max(16385, long)
    g = tree_of(res, b)
    leaves = g["links"][:, 2] < 0
    first, count = g["links"][~leaves, 2], g["links"][~leaves, 3]
    assert count.sum() == len(b) and np.array_equal(first, np.cumsum(count) - count)
    assert np.array_equal(count, np.unique(key, return_counts=True)[1])
    single = count == 1
    assert np.array_equal(g["com_mass"][~leaves][single], b[order[first[single]]])


# three launches a pass from 262145 bodies on: where many share the upper bits the lower ones are
# sorted first; where few do, the few long runs are sorted by themselves
@pytest.mark.parametrize("spread,crowded", [(300000, False), (0, True), (150000, True)])
def test_large_trees_with_long_runs_are_in_key_order(res, spread, crowded):
    r = np.random.RandomState(spread + 1)
    lengths = np.concatenate([[127, 128, 129, 130, 2048, 2049, 4096, 4097, 6000], r.randint(1, 400, 20)])
    if crowded:
        lengths = np.concatenate([lengths, r.randint(50, 3000, 200)])
    cell = 2.0 ** -13
    knot = (r.randint(-8000, 8000, (len(lengths), 3)) + 0.5) * cell
    x = np.repeat(knot, lengths, axis=0) + r.uniform(-0.12, 0.12, (lengths.sum(), 3)) * cell
    x = np.concatenate([x, r.uniform(-1, 1, (spread, 3)), [[-1, -1, -1], [1, 1, 1]]])
    x = x[r.permutation(len(x))]
    assert len(x) > 262144
    b = np.concatenate([x, np.ones((len(x), 1))], 1).astype(np.float32)
    order, key = reference_order(b)
    # of 1024 bodies, how many share their cell with an earlier one: far from the turn
    some = key[np.arange(1024) * len(b) // 1024] >> np.uint64(23)
    shared = 1024 - len(np.unique(some))
    assert shared * len(b) > 2 * 52428800 if crowded else shared * len(b) < 52428800 / 2
    g = tree_of(res, b)
    leaves = g["links"][:, 2] < 0
    first, count = g["links"][~leaves, 2], g["links"][~leaves, 3]
    assert count.sum() == len(b) and np.array_equal(first, np.cumsum(count) - count)
    assert np.array_equal(count, np.unique(key, return_counts=True)[1])
    single = count == 1
    assert np.array_equal(g["com_mass"][~leaves][single], b[order[first[single]]])


# bytes that an earlier build of the tree found enough, for bodies that are their own targets and
# for separate targets
@pytest.mark.parametrize("f64,separate,n,limit", [
    (False, False, 1, 36700), (False, True, 1, 37100), (False, False, 513, 350600), (False, False, 16384, 9000000),
    (True, False, 1, 64200), (True, True, 100, 138200), (True, False, 513, 403300), (True, True, 1000, 802100),
    (True, False, 5000, 3225300), (True, True, 5000, 3754300), (True, False, 16384, 10821000),
    (True, False, 65536, 43107700), (True, True, 65536, 48457900)])
def test_a_call_fits_the_capacity_it_did(native_lib, f64, separate, n, limit):
    from particular_gb300 import Between, CudaResources
    r = np.random.RandomState(n)
    b = np.concatenate([r.uniform(-1, 1, (n, 3)), np.ones((n, 1))], 1).astype(np.float64 if f64 else np.float32)
    with CudaResources(0) as res:
        m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.01), dvec3=f64)
        want = m.compute(Between(b.copy(), b) if separate else b)
    with CudaResources(0) as res:
        res.set_capacity_limit(limit)
        m = cuda.BarnesHut(0.7, res, AccelerationSoftened(0.01), dvec3=f64)
        got = m.compute(Between(b.copy(), b) if separate else b)
        assert native_lib.pt_ctx_device_bytes(res.handle) <= limit
        # and again: nothing is left to grow
        assert np.array_equal(got, m.compute(Between(b.copy(), b) if separate else b))
    assert np.array_equal(got, want)


# past 2^23 bodies, where the sort makes another pass, and past 2048 scan tiles of 4096: evenly
# spread, and in knots that share the sorted bits
@pytest.mark.parametrize("kind", ["cube", "knots"])
def test_largest_trees_are_in_key_order(native_lib, kind):
    import ctypes
    import torch
    from particular_gb300 import CudaResources, _native as N
    n = (1 << 23) + 4097
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda") * 2 - 1
    b = torch.cat([rand(n, 3), (rand(n, 1) * 0.25 + 1) / n], 1)
    if kind == "knots":  # of some 300 bodies, a quarter of a cell of the 16th level wide
        k = torch.floor(rand(n // 300, 3) * 32000)[torch.randint(0, n // 300, (n,), generator=g, device="cuda")]
        b[:, :3] = (k + 0.5) * 2.0 ** -15 + rand(n, 3) * 2.0 ** -18
    b[0, :3], b[1, :3] = -1, 1  # the root box
    lo, hi = torch.full((n, 3), -1.0, device="cuda"), torch.full((n, 3), 1.0, device="cuda")
    key = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _ in range(21):  # the build's subdivision in its f32 ops
        c = (lo + hi) * 0.5
        left = b[:, :3] < c
        hi, lo = torch.where(left, c, hi), torch.where(left, lo, c)
        key = key * 8 + 7 - (left.long() * torch.tensor([1, 2, 4], device="cuda")).sum(1)
    del lo, hi, c, left
    order = torch.sort(key, stable=True)[1]
    unique, counts = torch.unique_consecutive(key[order], return_counts=True)
    torch.cuda.synchronize()
    with CudaResources(0) as res:
        N.check(native_lib.pt_bh_build_device(res.handle, b.data_ptr(), n, None))
        res.synchronize()
        st = N.BhStats()
        N.check(native_lib.pt_bh_last_stats(res.handle, ctypes.byref(st)))
        assert st.leaves == len(unique)
        cm, ln = np.zeros((st.nodes, 4), np.float32), np.zeros((st.nodes, 4), np.int32)
        N.check(native_lib.pt_bh_export_tree(res.handle, cm.ctypes.data, ln.ctypes.data, None, st.nodes))
    leaves = ln[:, 2] >= 0
    first, count = ln[leaves, 2].astype(np.int64), ln[leaves, 3].astype(np.int64)
    assert np.array_equal(count, counts.cpu().numpy()) and np.array_equal(first, np.cumsum(count) - count)
    single = count == 1
    rows = b[order].cpu().numpy()[first[single]]
    assert np.array_equal(cm[leaves][single], rows)
    x = b.double()
    M = x[:, 3].sum().item()
    com = ((x[:, :3] * x[:, 3:]).sum(0) / M).cpu().numpy()
    assert ln[0, 1] == st.nodes and abs(cm[0, 3] - M) <= 1e-6 * M and np.abs(cm[0, :3] - com).max() <= 1e-6
