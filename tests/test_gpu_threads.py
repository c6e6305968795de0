"""Host threads that step their own trajectories at the same time -- chains of different lengths with
different merge tiles, so that one kernel is launched with different amounts of shared memory --
get what each gets alone."""

import threading

import pytest

from tests import gpu_helpers

pytestmark = pytest.mark.gpu

STEPS = 150
# nchain, maxstates, merge stride: one key word each
SPECS = [(6, 700, 64), (8, 1500, 240), (12, 3000, 160), (16, 3000, 96)]


def _trajectory(nchain, maxstates, stride):
    from paces_b200 import autotune
    eng = gpu_helpers.engine_for(nchain, 16, 1.3, cap=1 << 15, precision="c64", periodic=True)
    autotune.set_tuning(eng, stride)
    return gpu_helpers.grown_trajectory(eng, nchain, maxstates, initpos=1)[0]


def _run(tr, out):
    import torch
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(STEPS):
                rec = tr.step(evolve=True, dt=0.05)
            out += [rec.n_states, rec.norm, rec.energy_re, tr.psis[tr.cur][:rec.n_states].cpu()]
    except Exception as e:  # seen by the main thread
        out.append(e)


def test_concurrent_trajectories_equal_themselves_alone():
    import torch
    alone = []
    for spec in SPECS:
        alone.append([])
        _run(_trajectory(*spec), alone[-1])
    trajs, together = [_trajectory(*s) for s in SPECS], [[] for _ in SPECS]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=_run, args=(t, o)) for t, o in zip(trajs, together)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got, want in zip(together, alone):
        assert len(got) == len(want) == 4, (got, want)
        assert got[:3] == want[:3] and torch.equal(got[3], want[3])
