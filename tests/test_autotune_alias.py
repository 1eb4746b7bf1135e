"""The tuner measures each kernel once: variants that name another one's kernel again
are not searched, so the choice between them is not left to the noise of the
timing; they are still accepted, and an earlier cache entry that holds one is
applied as it is.  On fake targets, without a GPU."""
import json

import pytest

from test_autotune import FakeBatch, FakeModel
from xbeach_gpu_b200 import autotune as at
from xbeach_gpu_b200.abi import XBG_PHASE_WAVE
from xbeach_gpu_b200.model import Batch, Model


@pytest.fixture(autouse=True)
def _gpu(monkeypatch):
    monkeypatch.setattr(at, "_gpu", lambda: ("fake", 148))


class AliasModel(FakeModel):
    variant_alias = Model.variant_alias


class AliasBatch(FakeBatch):
    variant_alias = Batch.variant_alias


def test_the_same_kernel_is_not_measured_twice(tmp_path):
    assert (XBG_PHASE_WAVE, 2) in Model.variant_alias and (XBG_PHASE_WAVE, 2) in Batch.variant_alias
    m = AliasModel()
    assert at.tune(m, cache=str(tmp_path / "m.json"), reps=1)["wave_variant"] in (0, 1)
    assert m.steps == 6 + 2   # six tile-phase settings and two wave variants
    a, b = AliasBatch(), FakeBatch()
    assert at.tune(a, cache=str(tmp_path / "a.json"), reps=1)["wave_variant"] in (0, 1)
    at.tune(b, cache=str(tmp_path / "b.json"), reps=1)
    assert b.steps - a.steps == len(at.FACTORS)


def test_a_cached_alias_is_applied(tmp_path):
    cache = tmp_path / "m.json"
    m = AliasModel()
    at.tune(m, cache=str(cache), reps=1)
    db = json.loads(cache.read_text())
    key = next(k for k in db if k.startswith("wave_rows|"))
    db[key] = [[XBG_PHASE_WAVE, 2]]
    cache.write_text(json.dumps(db))
    m2 = AliasModel()
    assert at.tune(m2, cache=str(cache), reps=1)["wave_variant"] == 2 and m2.steps == 0
