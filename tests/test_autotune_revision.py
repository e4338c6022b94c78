"""A configuration tuned for other kernels than these is not applied."""

import json

from heu_gb300 import autotune


def test_entries_of_other_kernels_are_ignored(tmp_path):
    path = str(tmp_path / "tuning.json")
    cfg = {"variant": 1, "dec_variant": 1, "mul_window": 5, "dec_window": 5}
    name = autotune.device_name()
    with open(path, "w") as f:  # as it was written before entries had a revision
        json.dump({name: {"2048": {"config": cfg, "rates": {"mul": 2.2e6}}}}, f)
    assert autotune.load(2048, path=path) is None
    autotune.save(cfg, 3072, path=path)
    assert autotune.load(3072, path=path) == cfg and autotune.load(2048, path=path) is None
    data = json.load(open(path))
    assert "2048" in data[name]  # a save keeps what it does not replace
    data[name]["3072"]["revision"] += 1
    json.dump(data, open(path, "w"))
    assert autotune.load(3072, path=path) is None
    autotune.save(dict(cfg, mul_window=4), 2048, path=path)
    assert autotune.load(2048, path=path)["mul_window"] == 4
