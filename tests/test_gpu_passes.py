"""FP64 fixed mode in several direction passes: every direction is projected
once a sift, and its doubtful signs are counted once."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning", [None, {"proj_tile_n": 32}])  # CUDA cores; tensor cores (and their split)
@pytest.mark.parametrize("C,L,K,chunk", [(4, 1500, 24, 7), (3, 3001, 20, 10)])
def test_every_direction_is_projected_once_a_sift(C, L, K, chunk, tuning):
    rng = np.random.default_rng([C, L])
    y = np.round(4.0 * rng.standard_normal((C, L)).cumsum(axis=1)) / 4.0
    y, d = torch.as_tensor(y).cuda(), torch.as_tensor(oracle.directions(C, K)).cuda()
    sifts = 2 * 3
    outs, refined = [], []
    for ch in (0, chunk):
        plan = mg.Plan(C, L, K, 3, 3, dir_chunk=ch, tuning=tuning)
        out = torch.empty((3, C, L), dtype=torch.float64, device="cuda")
        refined.append(plan.run(y, d, out).refined)
        prof = plan.profile(y, d, out)
        passes = -(-K // ch) if ch else 1
        assert prof.launches[mg.STAGES.index("project")] == sifts * (passes + (1 if tuning else 0))
        plan.close()
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], outs[1]) and refined[0] == refined[1]
    assert refined[0] > 0 if tuning else refined[0] == 0
