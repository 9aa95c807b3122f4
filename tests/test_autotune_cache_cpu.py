"""The tuning cache: entries of another version are not taken, its own are."""

import json


def test_entries_of_older_builds_are_not_taken(tmp_path, monkeypatch):
    from crocodile_gb300 import autotune
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "sub" / "tuning.json"))
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda: "GPU")
    sig = "H4096_W4096_S16_Q8_4d_n2097152"
    new = {"config": {"tile": 16, "chunk": 0, "rows": 0, "groups": 0, "layout": 3, "dvis": 3}}
    autotune._store(sig, new)
    path = tmp_path / "sub" / "tuning.json"
    data = json.loads(path.read_text())
    assert autotune.load_cached(sig) == new
    old = {"config": {"tile": 16, "chunk": 512, "rows": 0, "groups": 0, "layout": 3, "dvis": 0}}
    path.write_text(json.dumps({"GPU|" + sig: old}))  # the key before versions
    assert autotune.load_cached(sig) is None
    path.write_text(json.dumps({"GPU|" + sig: old, **data}))
    assert autotune.load_cached(sig) == new
