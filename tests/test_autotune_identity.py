"""The tuner's on-disk choices belong to the build, the GPU and the source terms
they were measured with; anything else is measured again (no GPU)."""
import json
from dataclasses import replace

import pytest

from walicxe3d_b200 import autotune, problems
from walicxe3d_b200 import config as C
from test_autotune_cache import FakeContext


def test_entry_of_the_old_key_is_measured_again(tmp_path):
    prob = problems.sedov(2)
    cache = tmp_path / "tuning.json"
    cfg = prob.cfg
    old = f"neq{cfg.neqtot}-s{cfg.solver_type}-l{cfg.limiter_type}-mhd{int(cfg.mhd)}-nb{prob.nblocks}-lev1:{prob.nblocks}"
    cache.write_text(json.dumps({old: {"zsplit": 8, "fused": False}}))
    ctx = FakeContext(best=1, fused=True)
    rec = autotune.tune(ctx, prob, cache=cache, reps=1)
    assert ctx.calls == 1 and rec["cached"] is False and (rec["zsplit"], rec["fused"]) == (1, True)


@pytest.mark.parametrize("what", ["build_identity", "device_identity"])
def test_another_build_or_gpu_is_measured_again(tmp_path, monkeypatch, what):
    prob = problems.sedov(2)
    cache = tmp_path / "tuning.json"
    autotune.tune(FakeContext(best=2), prob, cache=cache, reps=1)
    monkeypatch.setattr(autotune, what, lambda: "other")
    ctx = FakeContext(best=4)
    assert autotune.tune(ctx, prob, cache=cache, reps=1)["zsplit"] == 4 and ctx.calls == 1


def test_source_terms_are_part_of_the_key():
    cfg = problems.snr_h(nroot=2, maxlev=1).cfg
    key = autotune.signature(cfg, 8, [1] * 8)
    assert key != autotune.signature(replace(cfg, cooling_type=C.COOL_NONE), 8, [1] * 8)
    assert key != autotune.signature(replace(cfg, eos_type=C.EOS_ADIABATIC), 8, [1] * 8)
