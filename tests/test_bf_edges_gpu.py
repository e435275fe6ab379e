"""Brute force at the sizes where its kernels change shape: rounds and tiles of sources that
end early, blocks of targets that are not full, and the sizes where a dispatch turns."""
import numpy as np
import pytest

from particular_gb300 import Acceleration, AccelerationSoftened, Between, cuda

pytestmark = pytest.mark.gpu


def bodies(n, seed, dtype=np.float32):
    r = np.random.RandomState(seed)
    b = np.concatenate([r.uniform(-1, 1, (n, 3)), r.uniform(0.5, 1.5, (n, 1))], 1)
    return np.ascontiguousarray(b.astype(dtype))


# ordered sums: 8 targets a block, 64 sources a round; a thread per target from 65536 on
@pytest.mark.parametrize("n_aff,n_src", [(1, 1), (7, 63), (8, 64), (9, 65), (17, 127), (65535, 129), (65536, 66)])
@pytest.mark.parametrize("vec3a", [False, True])
def test_exact_sums_are_the_sequential_ones(res, oracle, n_aff, n_src, vec3a):
    src = bodies(n_src, n_src)
    aff = bodies(n_aff, 7)
    aff[: min(n_aff, n_src, 4)] = src[: min(n_aff, n_src, 4)]  # coincident pairs
    got = cuda.BruteForce(res, Acceleration.checked(), exact=True, vec3a=vec3a).compute(Between(aff, src))
    rows = np.unique(np.r_[0:min(n_aff, 64), max(0, n_aff - 64):n_aff])
    want = (oracle.bf_f32_vec3a if vec3a else oracle.bf_f32)(aff[rows], src, 0.0, True)
    assert np.array_equal(got[rows].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n_aff,n_src", [(1, 1), (7, 63), (8, 64), (9, 65), (130, 128)])
def test_f64_sums_are_the_sequential_ones(res, oracle, n_aff, n_src):
    src = bodies(n_src, n_src, np.float64)
    aff = bodies(n_aff, 7, np.float64)
    aff[: min(n_aff, n_src, 4)] = src[: min(n_aff, n_src, 4)]
    got = cuda.BruteForce(res, AccelerationSoftened(0.01), dvec3=True).compute(Between(aff, src))
    want = oracle.bf_dvec3(aff, src, 0.01, True)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


# tiles of 256 sources, the last one in runs of 8, or each source compensated
# where it is the only one; sources laid out beforehand from 16640 on
# when no pair has to be tested for coincidence
@pytest.mark.parametrize("n_src", [1, 2, 7, 15, 16, 17, 255, 256, 257, 271, 272, 273, 513, 16639, 16640])
@pytest.mark.parametrize("soft", [0.0, 0.05])
def test_fast_sums_at_tile_edges(res, oracle, n_src, soft):
    src = bodies(n_src, n_src)
    src[n_src // 2, 3] = 0.0  # a massless source
    aff = bodies(333, 9)
    k = min(n_src, 200)
    aff[:k] = src[n_src - k:]  # targets that are sources, the last ones among them
    it = AccelerationSoftened(soft) if soft else Acceleration.checked()
    got = cuda.BruteForce(res, it).compute(Between(aff, src))
    want = oracle.bf_f64(aff, src, soft, True)
    # per pair 3 rsqrt factors (2^-22 each) and the differences; a run adds at most 128
    # terms into each packed half: 1e-5 of the sum of the terms' magnitudes
    d = src[None, :, :3].astype(np.float64) - aff[:, None, :3].astype(np.float64)
    r2 = (d * d).sum(-1)
    eps = float(np.float32(soft))
    scale = (src[None, :, 3] * np.sqrt(r2) / np.where(r2 > 0, r2 + eps * eps, 1.0) ** 1.5).sum(1)
    assert np.isfinite(got).all()
    assert (np.abs(got - want).max(1) <= 1e-5 * scale + 1e-30).all()


# Slices added by the last block of a small call or by a kernel of its own (up to 4096 x 4096
# pairs and beyond), host calls through page-locked memory or without (14043 bodies and beyond):
# the same sums in the same order, also when a call follows one of another shape.
@pytest.mark.parametrize("n", [1, 127, 129, 257, 1024, 4096, 4097, 14042, 14044])
def test_small_calls_add_their_slices_in_the_same_order(res, native_lib, n):
    import torch
    from particular_gb300 import _native as N

    b = bodies(n, n)
    d = torch.from_numpy(b).cuda()
    own = torch.empty((n, 3), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    N.check(native_lib.pt_bf_accel_f32_noalloc(d.data_ptr(), n, d.data_ptr(), n, 0.01, 1, own.data_ptr(), stream))
    want = own.cpu().numpy()
    method = cuda.BruteForce(res, AccelerationSoftened(0.01))
    for m in (n, 300, n, n):
        got = method.compute(b[:m])
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


# The sources of a last, shorter tile behind whole ones: each one's rounding error is kept. Two
# that cancel with a small one between them, in every place of the tile.
@pytest.mark.parametrize("targets_per_thread", [1, 2, 4])
@pytest.mark.parametrize("soft", [0.0, 0.05])
@pytest.mark.parametrize("tail", [3, 16, 21, 255])
def test_each_source_of_a_short_tile_is_compensated(res, native_lib, targets_per_thread, soft, tail):
    from particular_gb300 import _native as N

    src = bodies(256 + tail, 3)
    src[:, 3] = 0.0
    big, small = 256 + np.array([0, tail - 1]), 256 + tail // 2
    src[big] = [[1, 0, 0, 1e6], [-1, 0, 0, 1e6]]
    src[small] = [1, 0, 0, 1e-2]
    aff = bodies(300, 4)
    aff[::7, :3] = 0.0
    it = AccelerationSoftened(soft) if soft else Acceleration.checked()
    try:
        N.check(native_lib.pt_bf_set_plan(res.handle, targets_per_thread, 1))
        got = cuda.BruteForce(res, it).compute(Between(aff, src))[::7]
    finally:
        N.check(native_lib.pt_bf_set_plan(res.handle, 0, 0))
    want = 1e-2 / (1.0 + float(np.float32(soft)) ** 2) ** 1.5
    # the two cancel exactly; the small one's three rsqrt factors (2^-22 each) remain
    assert (np.abs(got[:, 0] - want) <= 2e-6 * want).all() and (got[:, 1:] == 0).all()


# The places of a short tile behind its last source hold no source: a target anywhere, at the
# origin and far outside the others too, meets the sources alone (unchecked and unsoftened, where a
# pair at one place would be NaN).
@pytest.mark.parametrize("n_src", [1, 2, 3, 255, 257, 300, 1022])
@pytest.mark.parametrize("at", [0.0, 1e30, -1e30, 3.4e38])
def test_no_source_behind_the_last_one(res, oracle, n_src, at):
    src = bodies(n_src, n_src)
    aff = bodies(40, 8)
    aff[::3, :3] = at
    got = cuda.BruteForce(res, Acceleration.unchecked()).compute(Between(aff, src))
    want = oracle.bf_f64(aff, src, 0.0, False)
    assert np.isfinite(got).all()
    if at:  # r^2 overflows in f32: exactly 0
        assert (got[::3] == 0).all()
    rest = np.ones(len(aff), bool)
    rest[::3] = at == 0
    scale = np.linalg.norm(want[rest], axis=1)
    # one sum of at most 256 terms' rounding, rsqrt factors of 2^-22
    assert (np.linalg.norm(got[rest] - want[rest], axis=1) <= 1e-4 * scale + 1e-5 * n_src).all()


# A target that is a source, anywhere in a warp and in any tile: few to a tile, so that a warp does
# them one after the other, half a warp and more, and a warp's targets one by one in all tiles. Calls of
# up to 4096 x 4096 pairs (more = 37) test every pair.
@pytest.mark.parametrize("more", [37, 14037])
@pytest.mark.parametrize("targets_per_thread", [1, 2, 4])
@pytest.mark.parametrize("per_warp", [1, 15, 16, 17, 31, 32])
def test_targets_meet_themselves_in_any_order(res, native_lib, oracle, targets_per_thread, per_warp, more):
    from particular_gb300 import _native as N

    src = bodies(1280, 5)
    r = np.random.RandomState(per_warp)
    spread = src[r.permutation(len(src))]  # a warp's targets in all five tiles
    close = bodies(640, 6)
    for w in range(0, 640, 32):  # some of a warp's targets in one tile
        close[w + r.permutation(32)[:per_warp]] = src[256 * (w // 32 % 5) + r.permutation(256)[:per_warp]]
    aff = np.concatenate([close, spread, bodies(more, 7)])
    aff[3], src[1279, 3] = src[1279], 0.0  # and a massless one
    try:
        N.check(native_lib.pt_bf_set_plan(res.handle, targets_per_thread, 1))
        got = cuda.BruteForce(res, Acceleration.checked()).compute(Between(aff, src))
    finally:
        N.check(native_lib.pt_bf_set_plan(res.handle, 0, 0))
    assert np.isfinite(got).all()
    aff, got = aff[:1957], got[:1957]
    want = oracle.bf_f64(aff, src, 0.0, True)
    d = src[None, :, :3].astype(np.float64) - aff[:, None, :3].astype(np.float64)
    r2 = (d * d).sum(-1)
    scale = (src[None, :, 3] * np.sqrt(r2) / np.where(r2 > 0, r2, 1.0) ** 1.5).sum(1)
    # as above: 3 rsqrt factors a pair, at most 128 terms into each packed half
    assert (np.abs(got - want).max(1) <= 1e-5 * scale).all()
