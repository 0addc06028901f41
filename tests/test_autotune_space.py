"""The autotuner's search space: no form tries its own default twice, and every
form with a tensor-core projection tries its tile width."""
import pytest

import memd_autotune as at
import memd_gb300 as mg

DEFAULTS = {mg.PREC_F64: {"solve_segment": 512}, mg.PREC_MIXED: {"solve_segment": 512},
            mg.PREC_F32: {"solve_segment": 256, "factor_segment": 16}}


@pytest.mark.parametrize("precision", [mg.PREC_F64, mg.PREC_F32, mg.PREC_MIXED])
def test_space_goes_by_the_form(precision):
    space = at.search_space(precision, precision == mg.PREC_MIXED)
    for knob, values in space.items():
        assert values[0] == 0 and len(set(values)) == len(values)
        assert {"solve_segment": 512, "solve_min_segment": 64, "mean_ctas": 2048, "proj_tile_n": 64,
                **DEFAULTS[precision]}.get(knob) not in values
    assert {128, 256, 512} <= set(space["solve_segment"]) | {DEFAULTS[precision]["solve_segment"]}
    assert ("proj_tile_n" in space) == (precision != mg.PREC_F32)
