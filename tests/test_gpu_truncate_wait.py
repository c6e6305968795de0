"""The truncation's selection when a grid-barrier wait runs out: with a 10 ms limit one block of the
cooperative launch gives up without arriving (the arrival nothing else provides), every other
block's wait expires, the kernel returns and PACES_ERR_TIMEOUT reaches the host.  Nothing is
written -- the new basis is empty, its buffer as it was -- and the next call succeeds."""

import numpy as np
import pytest
import torch

from tests.test_gpu_failures import WAIT_NS, _nat, _pair, _same_record
from tests.test_gpu_truncate_select import _basis

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("block", [0, 3])
@pytest.mark.parametrize("precision", ["c128", "c64", "weights"])
def test_selection_timeout_writes_nothing(precision, block, shuffle):
    nat = _nat()
    n, m = 70000, 20000
    eng, b, _ = _basis("c64" if precision == "c64" else "c128", n)
    w = np.random.default_rng(3).choice([0.25, 0.5, 0.75], n)  # ties at the cut
    if precision == "weights":
        x, call = torch.as_tensor(w, device=eng.device), eng.truncate_weighted
    else:
        x, call = torch.as_tensor(w, device=eng.device).to(eng.cdtype), eng.truncate
    args = dict(shuffle=shuffle, seed=5, step=2)
    good = call(b, x, m, **args)
    assert good.count() == m
    out = eng.new_basis(b.cap)
    out.keys.fill_(7)
    out.blk.fill_(11)
    eng.set_test_hooks(WAIT_NS, block)
    try:
        with pytest.raises(nat.PacesError) as err:
            call(b, x, m, out=out, **args)
        assert err.value.code == nat.ERR_TIMEOUT
    finally:
        eng.set_test_hooks(0, -1)
    assert bool((out.keys == 7).all()) and not bool(out.blk.any())
    call(b, x, m, out=out, **args)
    assert torch.equal(out.blk, good.blk) and torch.equal(out.keys[:m], good.keys[:m])
    eng.close()


@pytest.mark.parametrize("precision", ["c128", "c64"])
def test_step_without_propagation_leaves_the_state_intact(precision):
    nat = _nat()
    bad, witness = _pair(precision)
    bad.eng.set_test_hooks(WAIT_NS, 1)
    try:
        with pytest.raises(nat.PacesError) as err:
            bad.step(evolve=False)
        assert err.value.code == nat.ERR_TIMEOUT
    finally:
        bad.eng.set_test_hooks(0, -1)
    _same_record(bad.step(evolve=False), witness.step(evolve=False))
    for _ in range(2):
        _same_record(bad.step(evolve=True, dt=0.05), witness.step(evolve=True, dt=0.05))
