"""A batch with fewer trajectories than streams, or with trajectories of very different sizes: the
front stages get the GPU that is there -- a single trajectory on eight streams is as fast as on one
-- and every trajectory's results are those of stepping it alone."""

import pytest

from tests import gpu_helpers
from tests.test_gpu_batch import _same

pytestmark = pytest.mark.gpu


def _trajectory(nchain, maxstates, cap, precision="c64"):
    eng = gpu_helpers.engine_for(nchain, 16, 1.3, cap=cap, precision=precision, periodic=True)
    return gpu_helpers.grown_trajectory(eng, nchain, maxstates, initpos=1)[0]


def _front_ms(tr, n_streams):
    """The shortest front of the same step, taken again and again."""
    from paces_b200.engine import TrajectoryBatch
    batch = TrajectoryBatch([tr], n_streams=n_streams)
    batch.set_profiling(True)
    cur, times = tr.cur, []
    for _ in range(20):
        tr.cur = cur
        batch.step(True, 0.05)
        times.append(batch.stage_times()["front"])
    tr.cur = cur
    batch.close()
    return min(times)


def test_unused_streams_take_nothing_from_the_front():
    tr = _trajectory(16, 1 << 19, 1 << 22)
    for _ in range(3):
        tr.step(evolve=True, dt=0.05)
    one, eight = _front_ms(tr, 1), _front_ms(tr, 8)
    assert eight < 1.1 * one, (one, eight)
    tr.eng.close()


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("n_streams", [1, 2, 8, 64])
def test_uneven_trajectories_equal_themselves_alone(precision, n_streams):
    from paces_b200.engine import TrajectoryBatch
    specs = [(16, 60000, 1 << 19), (8, 900, 1 << 13), (12, 4000, 1 << 15)]
    alone, together = ([_trajectory(n, m, cap, precision) for n, m, cap in specs] for _ in range(2))
    batch = TrajectoryBatch(together, n_streams=n_streams)
    for _ in range(4):
        for r, t in zip(batch.step(evolve=True, dt=0.05), alone):
            _same(t.step(evolve=True, dt=0.05), r)
    batch.close()
    for t in alone + together:
        t.eng.close()
