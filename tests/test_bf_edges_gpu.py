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
