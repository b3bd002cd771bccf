"""The autotuner's decisions, on the CPU: a kind that wins only beyond 64
columns keeps those shapes on the tensor cores (64, not 65), and bounds cached
by other kernels are not read."""
import json

import pytest

from qutree_gb300 import autotune


def timings(wins):
    return {a: {"tensor_cores_ms": 0.5 if a in wins else 1.0, "fp32_pipe_ms": 1.0} for a in autotune.SIZES}


@pytest.mark.parametrize("wins,bound", [((), 65), ((72, 96), 64), ((64, 72, 96), 64), ((40, 48, 56, 64, 72, 96), 40),
                                        ((32, 40, 48, 56, 64), 65), ((16, 32, 96), 64), (autotune.SIZES, 16)])
def test_bound_from_timings(wins, bound):
    assert max(autotune.SIZES) > 64
    assert autotune.choose(timings(wins)) == bound


def test_bounds_of_other_kernels_are_ignored(tmp_path, monkeypatch):
    monkeypatch.setenv("QT_AUTOTUNE_DIR", str(tmp_path))
    monkeypatch.setattr(autotune, "_device_key", lambda device: "some_device-sm1")
    builtin = tuple(autotune.DEFAULT[k] for k in autotune.KINDS)
    rec = {"bounds": {"mp": 65, "hp": 65, "acc": 65}}
    for kernels in (None, "0123456789abcdef"):
        if kernels:
            rec["kernels"] = kernels
        with open(autotune.cache_path(0), "w") as f:
            json.dump(rec, f)
        assert autotune.cached(0) == builtin
    rec["kernels"] = autotune._kernels()
    with open(autotune.cache_path(0), "w") as f:
        json.dump(rec, f)
    assert autotune.cached(0) == (65, 65, 65)
