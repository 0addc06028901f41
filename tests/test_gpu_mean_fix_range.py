"""FP64 form, fixed mode: the fixed-point mean of a channel whose loudness
varies by many orders of magnitude keeps every stretch's own accuracy, as the
direct evaluation of every envelope (mean_eval = 1) does."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


def first_imf(y, d, **kw):
    C, L = y.shape
    plan = mg.Plan(C, L, d.shape[0], 2, 1, **kw)
    out = torch.empty((2, C, L), dtype=torch.float64, device="cuda")
    plan.run(torch.as_tensor(y).cuda(), torch.as_tensor(d).cuda(), out)
    plan.close()
    return out[0].cpu().numpy()


def tones(C, L, period, seed):
    rng = np.random.default_rng([seed, C, L])
    n = np.arange(L)
    return sum(rng.normal(size=(C, 1)) * np.sin(2 * np.pi * n / (period * rng.uniform(0.7, 1.6, (C, 1))) +
                                                rng.uniform(0, 6.28, (C, 1))) for _ in range(4))


def widest(a, r):
    """max of a over r samples on either side, per channel"""
    p = np.pad(a, ((0, 0), (r, r)))
    return np.lib.stride_tricks.sliding_window_view(p, 2 * r + 1, axis=1).max(axis=2)


# anchors every 8, 16, 32 and 64 samples; lane groups of 8, 16 and 32 channels; one pass and several
@pytest.mark.parametrize("chunk", [0, 7])
@pytest.mark.parametrize("C,L,K,period", [(3, 3000, 16, 3), (12, 4000, 16, 12), (33, 6000, 12, 30), (4, 16000, 20, 130)])
def test_quiet_stretches_keep_their_accuracy(C, L, K, period, chunk):
    y, d = tones(C, L, period, 1), oracle.directions(C, K)
    y[:, 5 * period] = 2.0 ** 40  # one artefact near the left end
    a, b = first_imf(y, d, dir_chunk=chunk), first_imf(y, d, mean_eval=1, dir_chunk=chunk)
    # past 80 knots its ripple (a factor 1/2 or less a knot, 1/3.7 in the mean) is far below the tones' rounding.
    # Both carry a few roundings (2^-53 each) of values up to a few times the largest near by: 64 of them
    far = 90 * period
    near = widest(np.abs(y[:, far:]), 2 * period)
    assert (np.abs(a - b)[:, far:] <= 64 * 2.0 ** -53 * near).all()


# zeros, a step of twelve orders of magnitude and the quiet side of it, which the ripple outweighs by far (the
# substitution's window of 48 knots cuts the ripple off 27 orders below the loud side, for either evaluation)
@pytest.mark.parametrize("chunk", [0, 5])
@pytest.mark.parametrize("C,L,K,period", [(2, 2000, 9, 4), (9, 4100, 12, 25), (32, 8200, 8, 110)])
def test_values_from_outside_a_span_larger_than_its_samples(C, L, K, period, chunk):
    y, d = tones(C, L, period, 2), oracle.directions(C, K)
    y[:, L // 2:] *= 1e-12
    y[:, L // 4:L // 4 + 3 * period + 70] = 0.0
    a, b = first_imf(y, d, dir_chunk=chunk), first_imf(y, d, mean_eval=1, dir_chunk=chunk)
    # the envelopes' knots reach twice the longest spacing and the stretch of zeros; values there, or the mean itself
    near = np.maximum(widest(np.maximum(np.abs(y), np.abs(y - b)), 8 * period), 1e-300)
    assert np.isfinite(a).all() and (np.abs(a - b) <= 64 * 2.0 ** -53 * near).all()
