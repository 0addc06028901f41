"""Direct evaluation on either side of the rules for its CTAs per tile (four,
two, one: as many as stay resident, three per SM, and have a direction for each
of their eight warps), odd channel counts and lengths, against the oracle."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [15, 16, 31, 33])
@pytest.mark.parametrize("share", [4, 2])  # CTAs per tile up to this many tiles
@pytest.mark.parametrize("more", [0, 1])  # tiles past it
def test_direct_evaluation_matches_oracle_at_the_limits(share, more, K):
    C = 3  # tiles of 32 samples, four channel lanes
    tiles = 3 * torch.cuda.get_device_properties(0).multi_processor_count // share + more
    L = 32 * tiles - 13
    rng = np.random.default_rng([K, L])
    y = rng.standard_normal((C, L)) + np.sin(np.arange(L) * rng.uniform(0.05, 0.4, (C, 1)))
    d = oracle.directions(C, K)
    plan = mg.Plan(C, L, K, 2, 2, mean_eval=1)
    out = torch.empty((2, C, L), dtype=torch.float64, device="cuda")
    plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    plan.close()
    want, _ = oracle.memd(y, d, 2, 2)
    # two sifts, each with a few roundings (2^-53) of values a few times the signal's
    assert np.abs(out.cpu().numpy() - want).max() <= 2 * 64 * 2.0 ** -53 * np.abs(y).max()
