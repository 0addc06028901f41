"""Mixed form, impulse-accumulation mean: the anchors of many directions are
summed in double-float with its rounding (2^-49 of the sum an addition)."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


def test_anchor_sums_of_many_directions():
    # 2^23 plus zeros and ones: the mean is all but the record, so the float32 IMF shows the mean's last bits
    C, L, K = 32, 8192, 1024
    y = 2.0 ** 23 + np.random.default_rng(1).integers(0, 2, (C, L)).astype(np.float64)
    d = oracle.directions(C, K)
    got = []
    for precision, tdt in ((mg.PREC_F64, torch.float64), (mg.PREC_MIXED, torch.float32)):
        plan = mg.Plan(C, L, K, 2, 1, precision)
        out = torch.empty((2, C, L), dtype=tdt, device="cuda")
        plan.run(torch.as_tensor(y, dtype=tdt).cuda(), torch.as_tensor(d, dtype=tdt).cuda(), out)
        plan.close()
        got.append(out[0].cpu().numpy().astype(np.float64))
    # at the anchors (every 32 samples at these knots; between them the walk's rounding comes on top). rms, of 2^23: a warp's sum of 256 terms in double-float 2^-47.5, eight of them 2^-49.0; the sum to 48 bits and the
    # IMF to float32 2^-49.8 each: 2^-48.6 (a low word never brought back to half an ulp of the high word: 2^-47.5)
    rms = np.sqrt(np.mean((got[1] - got[0])[:, 16::32] ** 2)) / 2.0 ** 23
    assert np.log2(rms) <= -48.05
