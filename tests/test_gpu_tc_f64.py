"""FP64 form: the tensor-core projection (certified, near ties decided again in
FP64) gives the FP64 projection's extrema bit for bit: every count, set hash
and IMF equals the CUDA-core projection's."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu
TC = {"proj_tile_n": 64}  # a given tile width: on the tensor cores at any size


def decompose(y, d, nimf, it, **kw):
    C, L = y.shape
    plan = mg.Plan(C, L, d.shape[0], nimf, it, **kw)
    plan.set_trace(True)
    out = torch.empty((nimf, C, L), dtype=torch.float64, device="cuda")
    st = plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    tr = plan.trace().copy()
    plan.close()
    return out.cpu().numpy(), tr, st


def both(y, d, nimf, it, **kw):
    a, ta, sa = decompose(y, d, nimf, it, tuning=TC, **kw)
    b, tb, sb = decompose(y, d, nimf, it, projection=mg.PROJ_CUDA_CORES, **kw)
    assert np.array_equal(ta["count"], tb["count"]) and np.array_equal(ta["hash"], tb["hash"])
    assert np.array_equal(a, b, equal_nan=True)
    assert sa.flags == sb.flags
    return sa


def walk(C, L, seed):
    rng = np.random.default_rng([seed, C, L])
    return rng.standard_normal((C, L)).cumsum(axis=1) + 3.0 * rng.standard_normal((C, L))


# tiles of 128 samples (and the halo row after them), 32-channel blocks, 64-direction tiles
@pytest.mark.parametrize("C,L,K,kw", [(1, 100, 3, {}), (3, 128, 16, {}), (5, 129, 17, {}), (31, 257, 64, {}),
                                      (32, 1000, 65, {}), (33, 1025, 20, {"dir_chunk": 7}), (128, 700, 24, {}),
                                      (8, 3000, 40, {"stop_mode": 1}), (6, 2000, 30, {"boundary": 1})])
def test_tensor_core_projection_equals_fp64_projection(C, L, K, kw):
    both(walk(C, L, 1), oracle.directions(C, K), 4, 4, **kw)


def test_ties_flat_stretches_and_scales():
    d = oracle.directions(4, 24)
    y = walk(4, 1500, 2)
    y[:, 200:700] = y[:, 200:201]           # every neighbour equal
    y[1:, 800:1100] = y[1:, 800:801]         # all channels but one flat
    y[:, 1200:1300] = np.round(y[:, 1200:1300])  # repeated values
    y[:, 1300:1400] = 1e5 + 1e-10 * y[:, 1300:1400]  # changes below the projections' rounding
    assert both(y, d, 3, 3).refined > 0
    for scale in (1e-200, 1e-30, 1e25, 1e200):
        both(y * scale, d, 2, 2)
    both(y, d * 1e60, 2, 1)
    mixed_scales = y * np.array([[1e-40], [1.0], [1e30], [1e-3]])
    both(mixed_scales, d, 2, 2)
    z = y.copy()
    z[2, 60], z[0, 900] = np.nan, np.inf
    both(z, d, 2, 1)


def test_batched_runs():
    lengths = [700, 1500, 64, 129]
    rng = np.random.default_rng(5)
    recs = [walk(5, n, i) * 10.0 ** rng.integers(-20, 20) for i, n in enumerate(lengths)]
    offs = np.cumsum([0] + [5 * n for n in lengths[:-1]])
    y = torch.as_tensor(np.concatenate([r.ravel() for r in recs])).cuda()
    dd = torch.as_tensor(oracle.directions(5, 21)).cuda()
    outs = []
    for kw in (dict(tuning=TC), dict(projection=mg.PROJ_CUDA_CORES)):
        plan = mg.Plan(5, max(lengths), 21, 3, 4, max_epochs=4, **kw)
        o = torch.empty(3 * y.numel(), dtype=torch.float64, device="cuda")
        plan.run_batched(y, lengths, offs, dd, o)
        plan.close()
        outs.append(o.cpu().numpy())
    assert np.array_equal(outs[0], outs[1], equal_nan=True)
