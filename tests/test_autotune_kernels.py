"""A tuned schedule belongs to the kernels it was timed on: the cache key changes with their sources."""
import importlib
import json


def test_key_changes_with_the_sources(dense, monkeypatch, tmp_path):
    autotune, build = (importlib.import_module("2dense_gb300." + m) for m in ("autotune", "build"))
    cfgs = [dense.config_default(ni=64, nj=64, benchmark=11, splitting=101, recon=255)]
    base = autotune.batch_key(cfgs)
    assert autotune.batch_key(cfgs) == base
    cache = tmp_path / "autotune.json"
    cache.write_text(json.dumps({base: {"schedule": [1, 2, 0, 0]}}))
    monkeypatch.setattr(autotune, "CACHE", str(cache))
    assert autotune.tune(cfgs)[1]["cached"]
    src = tmp_path / "csrc"
    src.mkdir()
    monkeypatch.setattr(build, "CSRC", str(src))
    monkeypatch.setattr(build, "INCLUDE", str(src))
    keys = set()
    for text in ("one", "two"):
        (src / "kernels.cu").write_text(text)
        autotune._kernels_key.cache_clear()
        keys.add(autotune.batch_key(cfgs))
    monkeypatch.undo()
    autotune._kernels_key.cache_clear()
    assert len(keys) == 2 and base not in keys
    assert autotune.batch_key(cfgs) == base
