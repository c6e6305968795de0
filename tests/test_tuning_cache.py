"""The tuner's cache file (CPU): choices timed on kernels that are gone are not taken up."""

import json
import types

import torch


def test_choices_of_earlier_kernels_are_not_reused(tmp_path, monkeypatch):
    from paces_b200 import autotune
    monkeypatch.setattr(autotune, "CACHE_PATH", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(autotune, "_memory", {})
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "GPU")
    eng = types.SimpleNamespace(device="cuda:0", nw=2, c64=True)
    choice = {"merge_stride": 96, "taylor_blocks_per_sm": 1, "taylor_variant": 0, "assemble_stride": 96}
    # layouts 1 and 2: merge tiles in four launches, Taylor chunks by bulk copies
    stale = {f"{kind}{v}GPU|nw2|c64|s20{end}": choice for v in ("", "v1|", "v2|") for kind, end in (("", ""), ("batch|", "|n4"))}
    (tmp_path / "tuning.json").write_text(json.dumps(stale))
    key = autotune._key(eng, 1 << 20)
    for k in (key, "batch|" + key + "|n4"):
        assert autotune._lookup(k, True) is None
        autotune._save_file(k, choice)
        assert autotune._lookup(k, True) == choice
    assert set(stale) < set(autotune._load_file())
