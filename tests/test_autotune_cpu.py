"""The tuner of a single grid's plan (fvleg_2d_gb300/autotune.py) on a stand-in handle."""
import json

import pytest

from fvleg_2d_gb300 import _lib, autotune, fluid
from fvleg_2d_gb300.config import SchemeConfig


class _Handle:
    """Times of its own per plan; the default is a plan that no list of candidates has."""
    default, ms, made = (64, 1), {}, 0

    def __init__(self, cfg):
        _Handle.made += 1
        self.plan = _Handle.default

    def initialize(self, *prims):
        return self

    def get_plan(self):
        return self.plan

    def set_plan(self, threads, rows):
        self.plan = (threads, rows)

    def run_timed(self, steps):
        return _Handle.ms.get(self.plan, 9.0) * steps, None

    def close(self):
        pass


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"one build")
    monkeypatch.setattr(_lib, "lib_path", lambda: str(lib))
    monkeypatch.setattr(fluid, "Fluid", _Handle)
    monkeypatch.setenv("CATO_TUNE_CACHE", str(tmp_path / "tune.json"))
    _Handle.made = 0
    cfg = SchemeConfig(ni=200, nj=160, dx=1.0, dy=1.0)
    return cfg, lib, tmp_path / "tune.json"


def test_the_default_plan_wins_when_it_is_fastest(tuner):
    cfg, _, _ = tuner
    _Handle.ms = {(64, 1): 1.0, (64, 8): 2.0}
    plan, table = autotune.tune(cfg, (), use_cache=False)
    assert plan == (64, 1) and table["64x1"] == 1.0 and "64x8" in table


def test_explicit_candidates_are_the_only_ones(tuner):
    cfg, _, _ = tuner
    _Handle.ms = {(64, 1): 1.0, (64, 8): 2.0}
    plan, table = autotune.tune(cfg, (), candidates=[(64, 8), (128, 8)], use_cache=False)
    assert plan == (64, 8) and set(table) == {"64x8", "128x8"}


def test_a_cached_winner_is_of_this_build(tuner):
    cfg, lib, path = tuner
    _Handle.ms = {(64, 16): 1.0}
    assert autotune.tune(cfg, ())[0] == (64, 16)
    _Handle.ms = {(64, 8): 0.5}
    assert autotune.tune(cfg, ())[0] == (64, 16) and _Handle.made == 1  # the same build: cached
    lib.write_bytes(b"another")
    assert autotune.tune(cfg, ())[0] == (64, 8)
    assert len(json.loads(path.read_text())) == 2
