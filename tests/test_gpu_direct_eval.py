"""Direct evaluation of the envelopes (stop mode, mirrored ends) against the
oracle at the sizes where its tiles, lane groups and the CTAs a tile's
directions are dealt to change."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


# fewer than 152 tiles: four CTAs a tile; 152 .. 303: two; from 304 on: one; 600 large tiles: 8 warps of long runs
@pytest.mark.parametrize("C,L,K,stop", [(1, 70, 3, True), (3, 31, 9, False), (5, 2081, 40, True), (8, 4831, 17, False),
                                        (9, 4897, 33, True), (16, 9761, 7, False), (33, 3300, 12, True),
                                        (4, 77000, 5, False)])
def test_direct_evaluation_matches_oracle(C, L, K, stop):
    rng = np.random.default_rng([C, L])
    y = rng.standard_normal((C, L)) + np.sin(np.arange(L) * rng.uniform(0.05, 0.4, (C, 1)))
    d = oracle.directions(C, K)
    kw = dict(stop_mode=mg.STOP_CRITERION) if stop else dict(boundary=mg.BOUNDARY_MIRROR)
    plan = mg.Plan(C, L, K, 2, 6 if stop else 2, **kw)
    out = torch.empty((2, C, L), dtype=torch.float64, device="cuda")
    st = plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    plan.close()
    want, info = oracle.memd(y, d, 2, 6 if stop else 2, stop_mode=stop, boundary=0 if stop else 1)
    got = out.cpu().numpy()
    if stop:
        assert st.n_imfs == info["n_imfs"] and list(st.sifts[:1]) == list(info["sifts"][:1])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    # six sifts at most, each with a few roundings (2^-53) of values a few times the signal's
    assert np.nanmax(np.abs(got - want), initial=0.0) <= 6 * 64 * 2.0 ** -53 * np.abs(y).max()
