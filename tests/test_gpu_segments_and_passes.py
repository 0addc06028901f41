"""The substitution's segments do not depend on the direction passes: with a
halo of four knots, where a segment starts shows in the result."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


# 2 K systems, more than the 256 below which their number does not count, of about 1,800 knots: segments of 128 by all
# directions (4096 x 128 / 360 = 1456 knots), of 64 by a pass's (2048)
@pytest.mark.parametrize("precision", [mg.PREC_F64, mg.PREC_MIXED])
@pytest.mark.parametrize("chunk", [16, 50])
def test_segments_do_not_depend_on_the_passes(chunk, precision):
    C, L, K = 4, 5400, 180
    tdt = torch.float64 if precision == mg.PREC_F64 else torch.float32
    y = torch.as_tensor(np.random.default_rng(3).standard_normal((C, L)), dtype=tdt).cuda()
    d = torch.as_tensor(oracle.directions(C, K), dtype=tdt).cuda()
    outs = []
    for kw in ({}, {"dir_chunk": chunk}):
        plan = mg.Plan(C, L, K, 2, 1, precision, solve_window=4, mean_eval=1, **kw)
        plan.set_trace(True)
        out = torch.empty((2, C, L), dtype=tdt, device="cuda")
        plan.run(y, d, out)
        knots = plan.trace()["count"][0, 0]
        plan.close()
        assert 1456 < knots.min() and knots.max() < 2048
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
