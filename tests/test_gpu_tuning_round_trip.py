"""A plan made from another plan's tuning() runs the same launches: none of the
reported values pins down what the plan chooses by the data."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [mg.PREC_F64, mg.PREC_F32, mg.PREC_MIXED])
@pytest.mark.parametrize("tuning", [None, {"factor_segment": 16}, {"factor_segment": 8, "solve_segment": 128}])
def test_a_plan_made_from_a_plans_tuning_is_the_same_plan(precision, tuning):
    first = mg.Plan(3, 900, 8, 2, 2, precision, tuning=tuning)
    t = first.tuning()
    second = mg.Plan(3, 900, 8, 2, 2, precision, tuning=t)
    assert second.tuning() == t
    # a chosen value is reported; the default for the forms that shorten it where the knots are few is 0, "by the knots"
    fixed = (tuning or {}).get("factor_segment", 16 if precision == mg.PREC_F32 else 0)
    assert t["factor_segment"] == fixed
    first.close()
    second.close()


@pytest.mark.parametrize("precision", [mg.PREC_F64, mg.PREC_F32, mg.PREC_MIXED])
def test_a_plan_without_segments_reports_none(precision):
    first = mg.Plan(3, 9000, 8, 2, 2, precision, solve_window=-1)
    t = first.tuning()
    second = mg.Plan(3, 9000, 8, 2, 2, precision, solve_window=-1, tuning=t)
    assert second.tuning() == t and t["solve_segment"] == t["solve_min_segment"] == t["factor_segment"] == 0
    first.close()
    second.close()
