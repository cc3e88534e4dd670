"""The cache key of the batched refinement's tuned schedules on the host: a choice
that was timed with other kernels, or with another meaning of a knob, is not taken."""

import json
from types import SimpleNamespace

from test_autotune_cpu import _cost, _Tunee, batch  # noqa: F401


def test_choices_of_earlier_kernels_are_not_read(batch, tmp_path, monkeypatch):  # noqa: F811
    monkeypatch.setattr(batch.torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(batch.torch.cuda, "get_device_properties",
                        lambda d: SimpleNamespace(name="B200", multi_processor_count=148))
    b = batch.BatchRefiner.__new__(batch.BatchRefiner)
    b.sizes, b.p = [(1024, 1024)] * 4, SimpleNamespace(R=10, paths=8)
    key = b._key()
    # an entry as the first kernels' library wrote it: no version in its key
    plain = key[key.index("B200"):]
    assert plain.startswith("B200|sm148|R10|paths8|n4|px") and key != plain
    entry = {"config": {"px_per_block": 512, "sgm_threads": 256, "sgm_ctas_per_sm": 16,
                        "sgm_fetch": 32}, "ms": 1.0, "default_ms": 2.0, "candidates": 9}
    (tmp_path / "batch_tune.json").write_text(json.dumps({plain: entry}))
    t = _Tunee(batch, _cost, key=key)
    assert not batch.BatchRefiner.autotune(t, reps=1)["cached"]
    assert t.config.as_dict()["sgm_ctas_per_sm"] == 8
