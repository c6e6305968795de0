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


FIRST_USE = """
import threading, torch
from tests import gpu_helpers
for nchain in (16, 32, 48, 64, 80, 96, 112, 128):  # one to eight key words: kernels of their own
    for precision in ("c64", "c128"):
        items = []
        for _ in range(4):
            eng = gpu_helpers.engine_for(nchain, 16, 1.0, cap=1 << 12, precision=precision)
            b, h, _ = eng.assemble(eng.basis_from_ref(gpu_helpers.initial_rows(nchain)))
            psi = eng.new_vector(b.cap)
            psi[:b.count()] = 0.5
            items.append((eng, b, h, psi))
        torch.cuda.synchronize()
        gate, out = threading.Barrier(len(items)), [None] * len(items)

        def run(i):
            eng, b, h, psi = items[i]
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                try:
                    out[i] = eng.observables(b, h, psi)["norm"]
                except Exception as e:
                    out[i] = repr(e)
        threads = [threading.Thread(target=run, args=(i,)) for i in range(len(items))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert out[0] == out[1] == out[2] == out[3], (nchain, precision, out)
"""


def test_first_observables_of_a_process_on_several_threads():
    import os
    import subprocess
    import sys
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", FIRST_USE], cwd=repo, capture_output=True, text=True, timeout=240)
    assert run.returncode == 0, run.stderr[-2000:]
