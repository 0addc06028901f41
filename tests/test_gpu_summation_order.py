"""Direct evaluation: results that do not depend on how the directions are
dealt to passes (FP64) and CTAs, or on the batch a record is in."""
import numpy as np
import pytest
import torch

import memd_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


def near_constant(C, L, seed):
    """2^23 plus zeros and ones: the mean is all but the record, so that the float32 IMF of the mixed form shows the
    mean's last bits (2^-49 of its size)."""
    return 2.0 ** 23 + np.random.default_rng([seed, C, L]).integers(0, 2, (C, L)).astype(np.float64)


def single(y, d, nimf, it, precision, **kw):
    C, L = y.shape
    tdt = torch.float64 if precision == mg.PREC_F64 else torch.float32
    plan = mg.Plan(C, L, d.shape[0], nimf, it, precision, **kw)
    out = torch.empty((nimf, C, L), dtype=tdt, device="cuda")
    plan.run(torch.as_tensor(y, dtype=tdt).cuda(), torch.as_tensor(d, dtype=tdt).cuda(), out)
    plan.close()
    return out.cpu().numpy()


# fewer directions than two groups of eight, more and a remainder; tiles of one, two and four CTAs; passes that end
# within a group and between two
@pytest.mark.parametrize("C,L,K,stop", [(1, 70, 13, False), (3, 701, 40, True), (5, 2081, 70, False), (8, 4831, 67, True),
                                        (9, 9001, 35, False), (33, 2600, 50, True)])
def test_direct_evaluation_does_not_depend_on_the_passes(C, L, K, stop):
    y, d = near_constant(C, L, 1), oracle.directions(C, K)
    kw = dict(stop_mode=mg.STOP_CRITERION) if stop else dict(mean_eval=1)
    a = single(y, d, 2, 3, mg.PREC_F64, **kw)
    for chunk in (5, 16, 33):
        assert np.array_equal(a, single(y, d, 2, 3, mg.PREC_F64, dir_chunk=chunk, **kw), equal_nan=True), chunk


@pytest.mark.parametrize("precision", [mg.PREC_F64, mg.PREC_MIXED])
def test_direct_evaluation_of_a_batch_equals_its_records(precision):
    C, K = 6, 40  # alone a record's tiles have four CTAs, the last two records' two and one; in the batch one
    lengths = [300 + 37 * e for e in range(40)] + [4700, 9000]
    recs = [near_constant(C, n, 10 + e) for e, n in enumerate(lengths)]
    d = oracle.directions(C, K)
    tdt = torch.float64 if precision == mg.PREC_F64 else torch.float32
    y = torch.as_tensor(np.concatenate([r.ravel() for r in recs]), dtype=tdt, device="cuda")
    off = [C * sum(lengths[:e]) for e in range(len(lengths))]
    out = torch.empty(2 * y.numel(), dtype=tdt, device="cuda")
    plan = mg.Plan(C, max(lengths), K, 2, 2, precision, max_epochs=len(lengths), mean_eval=1)
    plan.run_batched(y, lengths, off, torch.as_tensor(d, dtype=tdt).cuda(), out)
    plan.close()
    out = out.cpu().numpy()
    for e in (0, 7, 23, 39, 40, 41):
        n = lengths[e]
        got = out[2 * off[e]:2 * off[e] + 2 * C * n].reshape(2, C, n)
        assert np.array_equal(got, single(recs[e], d, 2, 2, precision, mean_eval=1)), e
