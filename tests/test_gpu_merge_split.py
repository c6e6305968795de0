"""The merges' partition: inputs of a few states (cut finer than the tuned stride), inputs whose
splitters are searched by eight lanes each, and inputs with a thread per splitter give the
oracle's enlarged basis, rows and order exactly, for keys of 1 to 8 words."""

import numpy as np
import pytest

from oracle import paces_oracle as po
from tests import gpu_helpers

pytestmark = pytest.mark.gpu

# (sites, occupations per site) -> key words
WIDTHS = {1: (16, 16), 2: (32, 16), 3: (48, 16), 4: (64, 16), 5: (40, 256), 6: (48, 256), 8: (64, 256)}


def _basis(model, n, dim, seed):
    """n distinct states, half of them on one site: that block's runs are longer than the rest's."""
    rng = np.random.default_rng(seed)
    raw = np.zeros((2 * n + 64, model.nchain + 1), dtype=np.uint32)
    raw[:, 0] = np.where(rng.random(len(raw)) < 0.5, model.nchain // 2, rng.integers(0, model.nchain, len(raw)))
    for s in rng.permutation(model.nchain)[:12]:
        raw[:, 1 + s] = rng.choice([0, 0, 0, 1, 2, dim - 2], len(raw))
    rows = po.unique_rows(po.compress(model, raw))
    return rows[np.sort(rng.choice(len(rows), min(n, len(rows)), replace=False))]


@pytest.mark.parametrize("words", sorted(WIDTHS))
@pytest.mark.parametrize("n,stride", [(1, None), (2, None), (33, None), (4097, None), (120000, None), (120000, 64)])
def test_expansion_matches_the_oracle(words, n, stride):
    from paces_b200 import autotune
    nchain, dim = WIDTHS[words]
    model = po.Model(nchain=nchain, max_ho_dims=[dim] * nchain)
    rows = _basis(model, n, dim, 31 * words + n)
    eng = gpu_helpers.engine_for(nchain, dim, 1.0, cap=1 << 20)
    try:
        if stride is not None:
            autotune.set_tuning(eng, merge_stride=stride)
        out = eng.expand(eng.basis_from_ref(rows))
        assert np.array_equal(gpu_helpers.ref_rows(eng, out), po.enlarge(model, rows))
    finally:
        eng.close()


@pytest.mark.parametrize("words", [1, 4])
def test_thread_per_splitter_matches_the_oracle(words):
    """More than 16384 splitters at the smallest stride."""
    from paces_b200 import autotune
    nchain, dim = WIDTHS[words]
    model = po.Model(nchain=nchain, max_ho_dims=[dim] * nchain)
    rows = _basis(model, 260000, dim, words)
    assert 5 * len(rows) > 17000 * 64
    eng = gpu_helpers.engine_for(nchain, dim, 1.0, cap=1 << 21)
    try:
        autotune.set_tuning(eng, merge_stride=64)
        out = eng.expand(eng.basis_from_ref(rows))
        assert np.array_equal(gpu_helpers.ref_rows(eng, out), po.enlarge(model, rows))
    finally:
        eng.close()
