"""The values that the propagators fold over the grid -- the series' maxima, the Lanczos sums --
are read behind a grid barrier by the lanes of one warp.  A lane that read too early would take a
stale value into the stop decision or a coefficient: every call repeated many times, at sizes
from one block to every block of the grid, gives the same bits."""

import pytest

from tests.test_gpu_taylor_schedules import _state

pytestmark = pytest.mark.gpu

REPEATS = 60


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("lattice,maxstates", [(False, 40), (False, 700), (False, 60000), (True, 3000)])
def test_repeated_propagations_give_the_same_bits(precision, lattice, maxstates):
    import torch
    eng, s, h, psi, S = _state(precision, lattice, maxstates)
    krylov = eng.new_krylov(s.cap, 9)
    out = torch.zeros_like(psi)
    calls = {
        "taylor": lambda: eng.taylor(s, h, psi, 0.05, psi_out=out),
        "lanczos": lambda: eng.lanczos(s, h, psi, 0.05, 9, psi_out=out, krylov=krylov),
        "scaled": lambda: (out, eng.expm_scaled(s, h, psi, out, 0.05, 0.5, 30, 2, 1.0)),
    }
    for name, call in calls.items():
        first, info = call()
        first = first[:S].clone()
        assert bool(torch.isfinite(torch.view_as_real(first)).all())
        for _ in range(REPEATS):
            got, again = call()
            assert again == info, name
            assert torch.equal(got[:S], first), name
    eng.close()
