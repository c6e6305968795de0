"""The Taylor kernel's schedules against each other: chunks kept in shared memory, chunks streamed
with the sum one term behind, and direct rows that update the sum in every sweep.  The terms,
sums, norms and stop decisions are the same, so everything is compared bit for bit; the direct
schedule itself is pinned to the reference's series by the stage and trajectory tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(precision, lattice, maxstates, seed=3):
    import torch
    from paces_b200.engine import Engine, ModelParams
    from tests import gpu_helpers
    n, dim = 16, (4 if lattice else 16)
    eng = Engine(ModelParams(nchain=n, max_ho_dims=[dim] * n, g=1.3, periodic=not lattice, precision=precision,
                             geo_dim=2 if lattice else 1, J2=0.5 if lattice else None), cap=12 * maxstates + 4096)
    b = eng.basis_from_ref(gpu_helpers.initial_rows(n, dim))
    while b.count() < maxstates:
        b = eng.expand(b)
    gen = torch.Generator(device=eng.device)
    gen.manual_seed(seed)
    w = torch.rand(b.cap, generator=gen, device=eng.device, dtype=torch.float64)
    b = eng.truncate(b, w.to(eng.cdtype), maxstates)
    s, h, _ = eng.assemble(b)
    S = s.count()
    psi = torch.zeros(s.cap, dtype=torch.complex128, device=eng.device)
    psi[:S] = torch.complex(*(torch.randn(S, generator=gen, device=eng.device, dtype=torch.float64) for _ in range(2)))
    psi /= torch.linalg.vector_norm(psi)
    return eng, s, h, psi.to(eng.cdtype), S


# rows per block of the wave that stay on chip: 1024; one block per SM below
@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("lattice,maxstates", [(False, 40), (False, 700), (False, 37000), (False, 90000), (True, 80000)])
def test_schedules_agree_bit_for_bit(precision, lattice, maxstates):
    import torch
    from paces_b200 import autotune
    eng, s, h, psi, S = _state(precision, lattice, maxstates)
    sms = torch.cuda.get_device_properties(eng.device).multi_processor_count
    if maxstates >= 80000:
        assert S > sms * 1024  # streams
    for m_star, tol, dt in ((1, None, 0.05), (2, None, 0.05), (3, None, 0.05), (100, None, 0.05), (100, 1e-3, 0.02),
                            (100, 3e-2, 0.01), (100, None, 0.13)):
        got = []
        for variant in (0, 1):
            autotune.set_tuning(eng, 160, 1, variant)
            out, info = eng.taylor(s, h, psi, dt, m_star=m_star, tol=tol)
            got.append((out[:S].cpu().numpy(), info))
        assert got[0][1] == got[1][1]
        assert np.array_equal(got[0][0], got[1][0])
    eng.close()


def test_a_zero_state_runs_to_the_term_limit():
    import torch
    from paces_b200 import autotune
    eng, s, h, psi, S = _state("c128", False, 90000)
    for variant in (0, 1):
        autotune.set_tuning(eng, 160, 1, variant)
        out, info = eng.taylor(s, h, torch.zeros_like(psi), 0.05, m_star=4)
        assert info[:2] == [False, 3] and not bool(out[:S].any())
    eng.close()
