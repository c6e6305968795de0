"""The truncation's selection at its edges: the threshold settled from a short list of weights or
by all radix rounds (many equal weights), tiles of the compaction that are full, ragged or one
state long, cuts that keep one state or drop one.  Compared with the reference's rule on the
host (the last maxstates of a stable ascending argsort, in index order): exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _basis(precision, states, nchain=16):
    from tests import gpu_helpers
    eng = gpu_helpers.engine_for(nchain, 16, 1.0, cap=1 << 17, precision=precision, periodic=True)
    b = eng.basis_from_ref(gpu_helpers.initial_rows(nchain))
    while b.count() < states:
        b = eng.expand(b)
    rows = gpu_helpers.ref_rows(eng, b)[:states]
    return eng, eng.basis_from_ref(rows, cap=states), rows


def _weights(kind, n, rng):
    if kind == "spread":
        return np.exp(rng.normal(0.0, 6.0, n))
    if kind == "ties":            # three values: every radix round, thousands of ties at the cut
        return rng.choice([0.25, 0.5, 0.75], n)
    if kind == "equal":
        return np.full(n, 0.125)
    if kind == "zeros":           # fewer non-zero weights than most cuts keep
        w = np.zeros(n)
        w[rng.integers(0, n, max(n // 50, 1))] = 1.0 + rng.random(max(n // 50, 1))
        return w
    if kind == "close":           # the same top 24 bits: the listed weights' low bits decide
        return 1.0 + rng.integers(0, 1 << 20, n) * 2.0 ** -52
    raise ValueError(kind)


@pytest.mark.parametrize("precision", ["c128", "c64", "weights"])
@pytest.mark.parametrize("kind", ["spread", "ties", "equal", "zeros", "close"])
@pytest.mark.parametrize("n", [1, 33, 1023, 1024, 1025, 20481, 70000])
def test_kept_states(precision, kind, n):
    import torch
    from tests import gpu_helpers
    rng = np.random.default_rng(n)
    eng, b, rows = _basis("c64" if precision == "c64" else "c128", n)
    w = _weights(kind, n, rng)
    if precision == "c64":
        w = w.astype(np.float32)
    for m in sorted({1, 2, n // 3 + 1, n - 1, n, n + 5} - {0}):
        if precision == "weights":
            out = eng.truncate_weighted(b, torch.as_tensor(w, device=eng.device), m)
        else:  # a real amplitude's magnitude is the weight itself
            out = eng.truncate(b, torch.as_tensor(w, device=eng.device).to(eng.cdtype), m)
        keep = np.sort(np.argsort(w, kind="stable")[-m:]) if m < n else np.arange(n)
        assert np.array_equal(gpu_helpers.ref_rows(eng, out), rows[keep]), (m, kind)
    eng.close()
