"""The tuner's cache: a choice is applied to plans of its bucket only while the
kernels are those that it was timed with."""
import json
from types import SimpleNamespace

import pytest

from thousandthchicken_b200 import autotune

torch = pytest.importorskip("torch")
DEVICE = "A GPU"


@pytest.fixture
def plan(monkeypatch, tmp_path):
    """A plan whose context records what is set on it."""
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "tune.json")
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: DEVICE)
    info = dict(ncblk=1024, reversible=0, width=2048, height=2048, ncomp=3)
    plan = SimpleNamespace(infos=[info], ctx=SimpleNamespace(device=0, handle=None))
    monkeypatch.setattr(autotune, "_set", lambda ctx, lanes=None, dwt=None: setattr(ctx, "set", (lanes, dwt)))
    return plan


@pytest.mark.parametrize("key", ["{device}|{bucket}", "{device}|0123456789abcdef|{bucket}", "other|{revision}|{bucket}"])
def test_choices_of_other_kernels_are_ignored(plan, key):
    key = key.format(device=DEVICE, bucket=autotune.bucket(plan), revision=autotune.revision())
    autotune.CACHE.write_text(json.dumps({key: {"lanes": 8, "dwt": "cp.async"}}))
    assert autotune.apply(plan) is None
    assert plan.ctx.set == (32, autotune.L.TC_DWT_TMA)


def test_choices_of_these_kernels_are_applied(plan):
    key = f"{DEVICE}|{autotune.revision()}|{autotune.bucket(plan)}"
    autotune.CACHE.write_text(json.dumps({key: {"lanes": 8, "dwt": "cp.async"}}))
    assert autotune.apply(plan)["lanes"] == 8
    assert plan.ctx.set == (8, autotune.L.TC_DWT_CPASYNC)
    assert autotune.tune_plan(plan, None)["cached"]
