"""The launch shape rules (fvleg_2d_gb300/csrc/cato_shape.h), compiled for the host."""
import ctypes
import os
import random
import shutil
import subprocess
from collections import namedtuple

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
FP64, MIXED, MIXED_DF = 0, 1, 2
SMS = 152
Shape = namedtuple("Shape", "width threads rows block warps variant")
GRIDS = [(64, 48), (128, 100), (200, 200), (256, 256), (400, 40), (448, 40), (512, 512), (1024, 1024),
         (4096, 4096), (3, 3), (5000, 3), (3, 5000), (100, 2000)]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    so = str(tmp_path_factory.mktemp("shape") / "libshape.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-shared", "-fPIC",
                    os.path.join(HERE, "shape_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _call(fn, *args):
    out = (ctypes.c_int * 6)()
    fn(*args, out)
    return Shape(*out)


def _grids():
    rng = random.Random(3)
    return GRIDS + [(int(2 ** rng.uniform(1.6, 13)), int(2 ** rng.uniform(1.6, 13)))
                    for _ in range(300)]


@pytest.mark.parametrize("precision", [FP64, MIXED, MIXED_DF])
@pytest.mark.parametrize("ng", [2, 3])
def test_a_plan_survives_get_and_set(rules, precision, ng):
    for ni, nj in _grids():
        d = _call(rules.default_shape, SMS, ni, nj, ng, precision)
        p = _call(rules.plan_shape, SMS, ni, nj, ng, precision, d.width, d.rows)
        assert p == d, (ni, nj)


def test_the_register_budget_is_ignored_outside_fp64(rules):
    for ni, nj in GRIDS:
        for precision in (FP64, MIXED, MIXED_DF):
            d = _call(rules.default_shape, SMS, ni, nj, 2, precision)
            forms = [_call2(rules.launched_form, SMS, ni, nj, 2, precision, d.width, d.rows, v)
                     for v in (0, 1, 2)]
            if precision == FP64:
                assert [v for v, _ in forms] == [0, 1, 2]
            else:
                assert forms[0] == forms[1] == forms[2] and forms[0][0] == 0, (ni, nj)


def _call2(fn, *args):
    out = (ctypes.c_int * 2)()
    fn(*args, out)
    return tuple(out)


@pytest.mark.parametrize("precision", [FP64, MIXED, MIXED_DF])
@pytest.mark.parametrize("ni,nj", [(2, 2_097_121), (3, 4_194_240), (64, 2_100_000), (3, 1 << 30)])
def test_tall_grids_fit_the_launch_limit(rules, precision, ni, nj):
    d = _call(rules.default_shape, SMS, ni, nj, 2, precision)
    assert -(-nj // d.rows) <= 65535, d


def _tune(rules, ni, nj, ng, precision, width, rows):
    out = (ctypes.c_int * 512)()
    n = rules.tune_shapes(SMS, ni, nj, ng, precision, width, rows, out)
    return [Shape(*out[6 * k:6 * k + 6]) for k in range(n)]


@pytest.mark.parametrize("precision", [FP64, MIXED, MIXED_DF])
@pytest.mark.parametrize("ni,nj", [(60, 5000), (100, 2000), (119, 900), (96, 104), (700, 500)])
def test_the_default_plan_is_a_tuning_candidate(rules, precision, ni, nj):
    d = _call(rules.default_shape, SMS, ni, nj, 2, precision)
    shapes = _tune(rules, ni, nj, 2, precision, d.width, d.rows)
    assert d in shapes
    assert {s.variant for s in shapes} == ({0, 1, 2} if precision == FP64 else {0})
    assert len(set(shapes)) == len(shapes)


@pytest.mark.parametrize("precision", [FP64, MIXED, MIXED_DF])
def test_shapes_follow_the_number_of_sms(rules, precision):
    # a grid of half the columns of tiles on half the SMs takes the same shape
    for tiles in (2, 4, 10, 40, 300):
        a, b = (_call(rules.default_shape, n * SMS, 60 * tiles * n, 120, 2, precision) for n in (1, 2))
        assert a == b, tiles
    shapes = {_call(rules.default_shape, n, 400, 200, 2, precision) for n in (20, 152, 1000)}
    assert len(shapes) > 1


@pytest.mark.parametrize("precision", [FP64, MIXED_DF])
def test_batch_rows_are_bounded_by_the_tallest_grid(rules, precision):
    rng = random.Random(5)
    grids = [(rng.randint(8, 512), rng.randint(8, 512)) for _ in range(2000)]
    ni = (ctypes.c_int * len(grids))(*(g[0] for g in grids))
    nj = (ctypes.c_int * len(grids))(*(g[1] for g in grids))
    for n in (1, 3, 40, 2000):
        tall = -(-max(nj[:n]) // 4) * 4
        # a search over every multiple of four up to 2^31 would not end
        rows = [rules.batch_rows(SMS, precision, plan, n, 60, ni, nj)
                for plan in (tall, tall + 1, 100_000, 2**31 - 1)]
        assert len(set(rows)) == 1 and 4 <= rows[0] <= tall, (n, rows)
    assert rules.batch_rows(SMS, precision, 3, 40, 60, ni, nj) == 3
