"""The checked build compares every FP64 quotient that the kernels form without
the division instruction with that instruction's (a flag in the run's state):
the pivots' reciprocals and the division of the mean by its count."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"spline_end": mg.SPLINE_NOT_A_KNOT}, {"boundary": mg.BOUNDARY_MIRROR},
                                {"dir_chunk": 19}, {"stop_mode": mg.STOP_CRITERION}])
@pytest.mark.parametrize("C,L,K", [(3, 30000, 37), (5, 4000, 64)])
def test_quotients_are_correctly_rounded(C, L, K, kw):
    y, d = mg.synth_eeg(C, L, 256.0, seed=L), oracle.directions(C, K)
    plan = mg.Plan(C, L, K, 4, 5, library=mg.checked_lib(), **kw)
    out = torch.empty((4, C, L), dtype=torch.float64, device="cuda")
    st = plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    plan.close()
    assert st.flags == 0
