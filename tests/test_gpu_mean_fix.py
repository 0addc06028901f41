"""FP64 form, fixed mode: the mean by impulse accumulation in fixed point
against the direct evaluation of every envelope (mean_eval = 1), one sift, at
the edges of its spans, anchors and lane groups."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


def one_sift(y, d, **kw):
    C, L = y.shape
    plan = mg.Plan(C, L, d.shape[0], 2, 1, **kw)
    out = torch.empty((2, C, L), dtype=torch.float64, device="cuda")
    st = plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    plan.close()
    return out.cpu().numpy(), st


def signal(C, L, period, seed):
    """Noise of extrema about `period` samples apart, uneven over the record."""
    rng = np.random.default_rng([seed, C, L])
    n = np.arange(L)
    y = np.zeros((C, L))
    for _ in range(4):
        p = period * rng.uniform(0.7, 1.6, (C, 1))
        y += rng.normal(size=(C, 1)) * np.sin(2 * np.pi * n / p + rng.uniform(0, 6.28, (C, 1)))
    return y * (1.0 + 0.5 * np.sin(2 * np.pi * n / L)) + 3.0 * n / L


# spans of 32 and 64 samples; anchors every 8, 16, 32, 64 (extrema 2.x .. 40 apart); 8, 16 and 32 channel lanes
@pytest.mark.parametrize("C,L,K,period", [(1, 31, 4, 4), (2, 33, 6, 5), (8, 64, 16, 3), (9, 65, 5, 9), (17, 257, 20, 14),
                                          (33, 1000, 12, 24), (32, 4099, 33, 45), (5, 3001, 64, 130), (3, 8193, 140, 8)])
def test_fixed_point_mean_matches_direct_evaluation(C, L, K, period):
    y, d = signal(C, L, period, 3), oracle.directions(C, K)
    a, sa = one_sift(y, d)
    b, sb = one_sift(y, d, mean_eval=1)
    assert sa.flags == sb.flags
    # each of the two carries a few rounding errors of the envelopes' values (2^-53 each, of values
    # up to a few times the record's largest) and the update's: 64 of them bound the difference
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.nanmax(np.abs(a - b), initial=0.0) <= 64 * 2.0 ** -53 * np.abs(y).max()


@pytest.mark.parametrize("chunk", [1, 7, 16])
def test_fixed_point_mean_does_not_depend_on_the_passes(chunk):
    y, d = signal(6, 3000, 12, 5), oracle.directions(6, 40)
    a, _ = one_sift(y, d)
    b, _ = one_sift(y, d, dir_chunk=chunk)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("chunk", [0, 9])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e300, 1e-310])
def test_values_outside_the_fixed_point_range_are_evaluated_directly(value, chunk):
    """A non-finite end value (a knot of every envelope) spoils what the direct
    evaluation says it spoils, and no other channel; tiny and huge scales work."""
    y, d = signal(4, 2500, 10, 7), oracle.directions(4, 24)
    if np.isfinite(value):
        y = y * value / np.abs(y).max()
    else:
        y[2, -1] = value
    a, _ = one_sift(y, d, dir_chunk=chunk)
    b, _ = one_sift(y, d, dir_chunk=chunk, mean_eval=1)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    # 1e-310: the values are subnormal, multiples of 2^-1074
    tol = 64 * max(2.0 ** -53 * np.abs(np.where(np.isfinite(y), y, 0.0)).max(), 2.0 ** -1074)
    assert (np.abs(np.where(np.isfinite(b), a - b, 0.0)) <= tol).all()


# records whose mirrored knots reach the ends from one or two extrema, spans of 32 to 128 samples
@pytest.mark.parametrize("chunk", [0, 5])
@pytest.mark.parametrize("C,L,K,period", [(1, 40, 4, 6), (3, 65, 8, 9), (8, 500, 12, 30), (17, 1000, 9, 60),
                                          (32, 4099, 20, 14), (5, 3001, 16, 300)])
def test_impulse_means_with_mirrored_ends_match_direct_evaluation(C, L, K, period, chunk):
    y, d = signal(C, L, period, 11), oracle.directions(C, K)
    kw = dict(boundary=mg.BOUNDARY_MIRROR, dir_chunk=chunk)
    a, sa = one_sift(y, d, **kw)
    b, sb = one_sift(y, d, mean_eval=1, **kw)
    assert sa.flags == sb.flags and np.array_equal(np.isnan(a), np.isnan(b))
    assert np.nanmax(np.abs(a - b), initial=0.0) <= 64 * 2.0 ** -53 * np.abs(y).max()
    outs = []
    for mean_eval in (0, 1):  # mixed form: double-float means, float32 outputs of the same input
        plan = mg.Plan(C, L, K, 2, 1, mg.PREC_MIXED, mean_eval=mean_eval, **kw)
        o = torch.empty((2, C, L), dtype=torch.float32, device="cuda")
        plan.run(torch.as_tensor(y, dtype=torch.float32).cuda(), torch.as_tensor(d, dtype=torch.float32).cuda(), o)
        plan.close()
        outs.append(o.cpu().numpy().astype(np.float64))
    assert np.array_equal(np.isnan(outs[0]), np.isnan(outs[1]))
    # both round a mean good to ~1e-13 to float32: one ulp of the largest value apart at most
    assert np.nanmax(np.abs(outs[0] - outs[1]), initial=0.0) <= 2.0 ** -22 * np.abs(y).max()


# spans of 128 samples (few knots on average) of which some hold more knots than a pair has lanes; 8, 16, 32 lanes
@pytest.mark.parametrize("C,L,K", [(3, 16384, 9), (12, 16385, 17), (33, 16415, 6)])
def test_mixed_mean_of_spans_with_more_knots_than_lanes(C, L, K):
    y, d = signal(C, L, 400, 13), oracle.directions(C, K)
    y[:, 6000:6500] += 0.3 * np.random.default_rng(5).normal(size=(C, 500))
    outs = []
    for mean_eval in (0, 1):
        plan = mg.Plan(C, L, K, 2, 1, mg.PREC_MIXED, mean_eval=mean_eval)
        o = torch.empty((2, C, L), dtype=torch.float32, device="cuda")
        plan.run(torch.as_tensor(y, dtype=torch.float32).cuda(), torch.as_tensor(d, dtype=torch.float32).cuda(), o)
        plan.close()
        outs.append(o.cpu().numpy().astype(np.float64))
    # both round a mean good to ~1e-13 to float32: one ulp of the largest value apart at most
    assert np.abs(outs[0] - outs[1]).max() <= 2.0 ** -22 * np.abs(y).max()


# factorisation segments of 4, 8 and 16 rows (the knots of 2 x 64 systems: about L / 3.6 each), odd remainders
@pytest.mark.parametrize("spline", [mg.SPLINE_NATURAL, mg.SPLINE_NOT_A_KNOT])
@pytest.mark.parametrize("C,L,K", [(2, 37, 3), (2, 2003, 64), (3, 6001, 64), (2, 12007, 64), (5, 1000, 9)])
def test_factorisation_segments_leave_the_pivots_alone(C, L, K, spline):
    y, d = signal(C, L, 3.6, 17), oracle.directions(C, K)
    a, sa = one_sift(y, d, spline_end=spline)
    b, sb = one_sift(y, d, spline_end=spline, tuning=dict(factor_segment=16))
    # 24 warm-up rows bring the start error (at most 1/2, 12 times less a row) to 4e-27, which rounding removes
    assert sa.flags == sb.flags and np.array_equal(a, b, equal_nan=True)
