"""The autotuner's cache holds choices for the kernels they were timed on."""
import json
from types import SimpleNamespace

import pytest

from atrip_gb300 import autotune


@pytest.mark.parametrize("form", ["fp64", "split_bf16"])
def test_choices_for_other_kernels_are_not_used(tmp_path, monkeypatch, form):
    path = tmp_path / "tuning.json"
    monkeypatch.setattr(autotune, "CACHE", str(path))
    monkeypatch.setattr(autotune, "_device_name", lambda device: "a device")
    new = {"tuning": {}, "ms": 1.0, "trials": []}
    monkeypatch.setattr(autotune, "tune_fp64", lambda ctx: new)
    monkeypatch.setattr(autotune, "tune_split", lambda ctx, slices, form: new)
    monkeypatch.setattr(autotune, "choose_slices",
                        lambda ctx, tol, form: {"form": form, "slices": 3, "estimates": {}})
    # as written when fp64_tile_rows was a parameter of the only FP64 kernel
    old = {"tuning": {"fp64_tile_rows": 64}, "form": form, "slices": 0, "seconds": 1.0}
    path.write_text(json.dumps({f"a device|No=8|Nv=40|{form}": old}))
    set_to = []
    ctx = SimpleNamespace(device=0, No=8, Nv=40, set_tuning=lambda **kw: set_to.append(kw))
    got = autotune.tune(ctx, form)
    assert not got["cached"] and got["tuning"] == {}
    assert {"fp64_tile_rows": 64} not in set_to
    again = autotune.tune(ctx, form)
    assert again["cached"] and again["tuning"] == {} and set_to[-1] == {}
