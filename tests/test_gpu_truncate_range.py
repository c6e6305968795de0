"""The truncation's threshold where the ranges of its passes end: the first pass bins the weights
from 2^-63 to 2 and takes what lies below or above into its end bins, so cuts just above 2^-63,
below it, above 2 and on the end bins' edges narrow a range that is no whole number of bins.
Compared with the reference's rule on the host (the last maxstates of a stable ascending
argsort, in index order): exact."""

import numpy as np
import pytest

from tests.test_gpu_truncate_select import _basis

pytestmark = pytest.mark.gpu

LOW = 2.0 ** -63                    # where the first pass's regular bins start
EDGE = LOW * (1.0 + 2.0 ** -6)      # where its lowest bin ends


def _weights(kind, n, rng):
    """Weights and the interval that the cuts are taken from."""
    few, half = 300, n // 2
    w = 2.0 ** rng.uniform(-80.0, -70.0, n)              # far below: all in the lowest bin
    at = rng.permutation(n)
    if kind == "few_in_the_lowest_bins_end":             # settled from a list
        w[at[:half]] = 2.0 ** rng.uniform(-64.0, -62.0, half)
        w[at[:few]] = LOW * (1.0 + rng.random(few) / 64.0)
        return w, LOW, EDGE
    if kind == "many_in_the_lowest_bins_end":            # more passes
        w[at[:half]] = LOW * (1.0 + rng.random(half) / 64.0)
        w[at[:2 * few]] = LOW * rng.uniform(1.02, 1.24, 2 * few)
        return w, LOW, EDGE
    if kind == "ties_in_the_lowest_bins_end":            # every pass, thousands of ties at the cut
        w[at[:half]] = LOW * (1.0 + rng.integers(0, 3, half) * 2.0 ** -9)
        w[at[:few]] = LOW * rng.uniform(1.02, 1.24, few)
        return w, LOW, EDGE
    if kind == "below":                                  # the cut itself far below
        w[at[:half]] = 2.0 ** rng.uniform(-63.5, -62.0, half)
        return w, 2.0 ** -80, 2.0 ** -63.2
    if kind == "edges":                                  # neighbours of the bins' edges, many times
        near = [x for e in (LOW, EDGE, 2.0) for x in (np.nextafter(e, 0, dtype=np.float32), e,
                                                      np.nextafter(e, 4, dtype=np.float32))]
        return rng.choice(np.array(near, dtype=np.float64), n), 0.0, 4.0
    if kind == "above":                                  # the highest bin, open upwards
        w[at[:half]] = np.exp(rng.uniform(0.69, 80.0, half))
        return w, 2.0, 1e36
    raise ValueError(kind)


KINDS = ["few_in_the_lowest_bins_end", "many_in_the_lowest_bins_end", "ties_in_the_lowest_bins_end", "below", "edges",
         "above"]


@pytest.mark.parametrize("precision", ["c128", "c64", "weights"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [6000, 70000])
def test_cuts_in_the_end_bins(precision, kind, n):
    import torch
    from tests import gpu_helpers
    rng = np.random.default_rng(n + 17)
    eng, b, rows = _basis("c64" if precision == "c64" else "c128", n)
    w, lo, hi = _weights(kind, n, rng)
    if precision == "c64":
        w = w.astype(np.float32)
    cuts = np.nonzero((np.sort(w)[::-1] >= lo) & (np.sort(w)[::-1] < hi))[0] + 1  # states kept when the cut is there
    assert len(cuts) > 100
    for m in sorted({int(cuts[i]) for i in (0, 1, len(cuts) // 3, len(cuts) // 2, -2, -1)} - {n}):
        if precision == "weights":
            out = eng.truncate_weighted(b, torch.as_tensor(w, device=eng.device), m)
        else:  # a real amplitude's magnitude is the weight itself
            out = eng.truncate(b, torch.as_tensor(w, device=eng.device).to(eng.cdtype), m)
        keep = np.sort(np.argsort(w, kind="stable")[-m:])
        assert np.array_equal(gpu_helpers.ref_rows(eng, out), rows[keep]), (m, kind)
    assert eng.read_status() == 0
    eng.close()
