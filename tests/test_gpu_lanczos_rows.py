"""The Lanczos propagation on bases whose rows end inside, at and behind a warp's unit of 64 rows,
and with fewer rows than warps, against the oracle's restatement on the same input."""

import numpy as np
import pytest
import torch

from oracle import paces_oracle as po
from tests import gpu_helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maxstates", [1, 4, 6, 7, 30, 700, 9000])
@pytest.mark.parametrize("order", [1, 2, 12])
def test_ragged_rows_match_the_oracle(maxstates, order):
    nchain, g = 6, 1.2
    eng = gpu_helpers.engine_for(nchain, 16, g, cap=1 << 17)
    tr, _ = gpu_helpers.grown_trajectory(eng, nchain, maxstates, initpos=2)
    for _ in range(6):
        tr.step(evolve=True, dt=0.05)
    b, h = tr.basis, tr.h
    n = b.count()
    psi = torch.zeros(b.cap, dtype=torch.complex128, device=eng.device)
    rng = np.random.default_rng(maxstates + order)
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    psi[:n] = torch.as_tensor(x / np.linalg.norm(x)).to(eng.device)
    out, dbg = eng.lanczos(b, h, psi, 0.05, order)
    assert dbg == [False, 0, 0.0, 0.0]
    m = po.Model(nchain, [16] * nchain, g=g)
    diag, mats, _ = gpu_helpers.csr_from_table(eng, b, h, 1.0, g)
    asm = po.Assembly(gpu_helpers.ref_rows(eng, b), diag, mats, None, None, 0)
    ref, _ = po.lanczos(asm, psi[:n].cpu().numpy(), 0.05, order)
    np.testing.assert_allclose(out[:n].cpu().numpy(), ref, rtol=0, atol=1e-13)
    eng.close()
