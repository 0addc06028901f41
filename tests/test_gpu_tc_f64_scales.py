"""FP64 form, tensor-core projection: directions of any scale a double can
hold, one scale or several, give the FP64 projection's extrema bit for bit."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


def decompose(y, d, **kw):
    C, L = y.shape
    plan = mg.Plan(C, L, d.shape[0], 2, 2, **kw)
    plan.set_trace(True)
    out = torch.empty((2, C, L), dtype=torch.float64, device="cuda")
    plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    tr = plan.trace().copy()
    plan.close()
    return out.cpu().numpy(), tr


def record(C, L):
    rng = np.random.default_rng([C, L])
    y = rng.standard_normal((C, L)).cumsum(axis=1) + 3.0 * rng.standard_normal((C, L))
    y[:, 300:400] *= 1e-28  # differences that scaled floats flush to zero, or keep in part
    y[:, 400:500] *= 1e-38
    y[:, 500:600] = np.round(y[:, 500:600])
    return y


# past 2^19 (flushed differences times the direction), near the largest float (sums of products overflow), past it, and
# far below the smallest
@pytest.mark.parametrize("C", [5, 32, 40])
@pytest.mark.parametrize("scale", [1e-300, 1e-45, 1e-38, 1e7, 1e20, 1e37, 3e38, 1e39, 1e200])
def test_directions_of_any_scale(C, scale):
    y, d = record(C, 900), oracle.directions(C, 24) * scale
    a, ta = decompose(y, d, tuning={"proj_tile_n": 32})
    b, tb = decompose(y, d, projection=mg.PROJ_CUDA_CORES)
    assert np.array_equal(ta["count"], tb["count"]) and np.array_equal(ta["hash"], tb["hash"])
    assert np.array_equal(a, b, equal_nan=True)


def test_directions_of_several_scales():
    C, K = 8, 40
    y, rng = record(C, 900), np.random.default_rng(4)
    d = oracle.directions(C, K) * 10.0 ** rng.integers(-300, 250, (K, 1)) * 10.0 ** rng.integers(-45, 45, (K, C))
    d[3] = 0.0
    a, ta = decompose(y, d, tuning={"proj_tile_n": 32})
    b, tb = decompose(y, d, projection=mg.PROJ_CUDA_CORES)
    assert np.array_equal(ta["count"], tb["count"]) and np.array_equal(ta["hash"], tb["hash"])
    assert np.array_equal(a, b, equal_nan=True)


def same(y, d):
    a, ta = decompose(y, d, tuning={"proj_tile_n": 32})
    b, tb = decompose(y, d, projection=mg.PROJ_CUDA_CORES)
    assert np.array_equal(ta["count"], tb["count"]) and np.array_equal(ta["hash"], tb["hash"])
    assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("scale", [1.0, 3e38, 1e60])
def test_partial_sums_past_the_largest_float(scale):
    # the first half of the channels adds up to far more than the whole, of the other sign
    C, K = 32, 20
    rng = np.random.default_rng(6)
    y = rng.standard_normal((1, 900)) * np.where(np.arange(C) < 16, 1.0, 1.05)[:, None] + 1e-3 * rng.standard_normal((C, 900))
    d = np.where(np.arange(C) < 16, 1.0, -1.0) * rng.uniform(0.9, 1.0, (K, 1)) * rng.uniform(0.999, 1.0, (K, C))
    same(y, d * scale)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 60, 2.0 ** 100])
def test_flushed_differences_times_large_entries(scale):
    # 2^-128 and 2^-119 of the record's largest sample over whole tiles: the first channel's scaled differences are
    # flushed, and its entry is 2^11 times the second's
    K = 24
    rng = np.random.default_rng(7)
    y = rng.standard_normal((2, 1200))
    y[0, 200:900] *= 2.0 ** -128
    y[1, 200:900] *= 2.0 ** -119
    d = np.stack([np.ones(K), rng.choice([-1.0, 1.0], K) * 2.0 ** -11 * rng.uniform(0.5, 2.0, K)], axis=1)
    same(y, d * scale)


# a loud sample in every tile of 128: every quiet sample's sign is doubtful in every direction, at the warps' first and
# last samples too; channel counts around the batches of eight loads, more and fewer directions than sixteen
@pytest.mark.parametrize("C,K", [(1, 5), (7, 16), (8, 17), (33, 40), (20, 70)])
def test_doubtful_signs_everywhere(C, K):
    rng = np.random.default_rng([C, K])
    y = rng.standard_normal((C, 1111))
    y[:, 60::128] *= 1e9
    same(y, oracle.directions(C, K))
