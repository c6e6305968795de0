"""H x with infinite amplitudes: a row's missing neighbours add nothing, so a row is infinite or NaN
exactly where the sum over its stored elements is (the reference's CSR product)."""

import numpy as np
import pytest

from tests import gpu_helpers

pytestmark = pytest.mark.gpu

MODELS = {"open chain": dict(nchain=7), "ring": dict(nchain=7, periodic=True), "chain with J2": dict(nchain=7, J2=0.5),
          "square": dict(nchain=9, geo_dim=2), "square with J2": dict(nchain=9, geo_dim=2, J2=-0.5),
          "cube": dict(nchain=27, geo_dim=3, J2=0.25)}


def _expected(p, h, S, x):
    """Real and imaginary parts of the sum of the stored elements, and the rows with both couplings."""
    nbr = h.nbr[:S].cpu().numpy()
    meta = h.meta[:S].cpu().numpy().view(np.uint32)
    n = ((meta >> 8) & 0xFF).astype(np.float64)
    channels = [(nbr[:, k], p.J) for k in (0, 1)]
    if h.xnbr is not None:
        per_term = p.geo_dim
        x_nbr = h.xnbr.view(-1, h.cap, 2)[:, :S].cpu().numpy()
        for c in range(len(x_nbr)):
            channels += [(x_nbr[c, :, k], p.J if c + 1 < per_term else p.J2) for k in (0, 1)]
    channels += [(nbr[:, 2], p.g * np.sqrt(n)), (nbr[:, 3], p.g * np.sqrt(n + 1.0))]
    d = p.eps_sys + p.hbar_omega * (meta >> 16)
    out = []
    for part in (x.real.astype(np.float64), x.imag.astype(np.float64)):
        with np.errstate(invalid="ignore"):
            y = d * part
            for idx, amp in channels:
                y = y + np.where(idx >= 0, np.broadcast_to(amp, S) * part[np.maximum(idx, 0)], 0.0)
        out.append(y)
    return out, (nbr[:, 2] >= 0) & (nbr[:, 3] >= 0)


# (a complex64 row multiplies its missing couplings by zero, a chain's row its missing hops as well)
CASES = [(m, "c128") for m in MODELS] + [(m, "c64") for m, kw in MODELS.items() if "geo_dim" in kw or "J2" in kw]


@pytest.mark.parametrize("model,precision", CASES)
def test_missing_neighbours_add_nothing_to_infinite_rows(model, precision):
    import torch
    from paces_b200.engine import Engine, ModelParams
    kw = MODELS[model]
    nchain, dim = kw["nchain"], 4
    eng = Engine(ModelParams(max_ho_dims=[dim] * nchain, g=1.3, eps_sys=0.5, precision=precision, **kw), cap=1 << 15)
    b = eng.basis_from_ref(gpu_helpers.initial_rows(nchain, dim))
    for _ in range(4):
        b = eng.expand(b)
    s, h, _ = eng.assemble(b)
    S = s.count()
    rng = np.random.default_rng(5)
    x = rng.normal(size=S) + 1j * rng.normal(size=S)
    at = rng.choice(S, S // 7, replace=False)
    x.real[at[0::3]] = np.inf
    x.imag[at[1::3]] = -np.inf
    x[at[2::3]] = complex(np.inf, np.inf)
    xt = torch.zeros(s.cap, dtype=eng.cdtype, device=eng.device)
    xt[:S] = torch.view_as_complex(torch.as_tensor(np.stack([x.real, x.imag], axis=1), device=eng.device)).to(eng.cdtype)
    y = eng.apply_h(s, h, xt)[:S].cpu().numpy()
    (re, im), both = _expected(eng.params, h, S, x)
    rows = both if precision == "c64" else np.ones(S, dtype=bool)
    # a cut-off sum of at most sixteen terms of order ten, in the vector's precision
    tol = 16 * 10 * 16 * np.finfo(np.float32 if precision == "c64" else np.float64).eps
    hit = 0
    for got, want in ((y.real, re), (y.imag, im)):
        got, want = got[rows], want[rows]
        finite = np.isfinite(want)
        hit += int((~finite).sum())
        assert np.array_equal(np.isfinite(got), finite)
        assert np.array_equal(got[~finite].astype(np.float64), want[~finite], equal_nan=True)
        assert np.abs(got[finite] - want[finite]).max() < tol
    assert hit  # some rows are infinite or NaN
    eng.close()
