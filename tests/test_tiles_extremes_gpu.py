"""Tiles whose fluxes read pressures around the edge, in the precisions without an oracle, and
reconstruction data of widely different magnitudes against the oracle."""
import numpy as np
import pytest

from conftest import random_prims
from fvleg_2d_gb300.fluid import Fluid, FluxSolver
from test_tiles_gpu import FIELDS, SIZES, _cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "mixed_df"])
@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("limiter,flux", [("superbee", "Roe"), ("minmod", "SD-SLAU"),
                                          ("van_leer", "M-AUSMPW+")])
def test_result_is_independent_of_the_shape(precision, ni, nj, limiter, flux):
    cfg = _cfg(ni, nj, limiter, flux, precision)
    prims = random_prims(cfg, np.random.default_rng(ni * 100 + nj))
    states = []
    for plan in (None, (64, 1), (64, 2), (96, 3), (128, 7), (192, 5), (224, 9), (256, 30)):
        f = Fluid(cfg).initialize(*prims)
        if plan:
            f.set_plan(*plan)
        f.run_timed(2)
        states.append(f.state(FIELDS))
        f.close()
    for s in states[1:]:
        for k in FIELDS:
            np.testing.assert_array_equal(s[k], states[0][k])


@pytest.mark.parametrize("limiter", ["van_leer", "MLP3", "MLP5"])
@pytest.mark.parametrize("lo,hi", [(-52, 58), (-20, 20), (-100, 100)])
def test_wide_magnitudes_equal_the_oracle(oracle, limiter, lo, hi):
    cfg = _cfg(300, 200, limiter, "HLLC")
    g = cfg.ghost_layers()
    rng = np.random.default_rng(23)
    prims = []
    for k in range(4):
        d = np.exp2(rng.uniform(lo, hi, (cfg.ni, cfg.nj)))
        if k in (1, 2):  # velocities of either sign, and zeros
            d *= rng.choice([-1.0, 1.0, 0.0], d.shape, p=[0.4, 0.4, 0.2])
        a = np.zeros(cfg.halo_shape, order="F")
        a[g:g + cfg.ni, g:g + cfg.nj] = d
        prims.append(a)
    want = oracle.solve(cfg, *[p.copy(order="F") for p in prims])
    got = FluxSolver(cfg).solve(*[p.copy(order="F") for p in prims])
    for k in range(4):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("limiter", ["superbee", "van_leer", "MLP3", "MLP5"])
@pytest.mark.parametrize("flux", ["AUSMPW+", "SLAU2", "SD-SLAU", "Roe", "AUSM+-up", "M-AUSMPW+"])
@pytest.mark.parametrize("width", [2, 10, 60])
def test_wild_states_equal_the_oracle(oracle, limiter, flux, width):
    # magnitudes 2^-width .. 2^width next to each other: negative edge pressures, NaN, overflow
    cfg = _cfg(97, 61, limiter, flux)
    g = cfg.ghost_layers()
    rng = np.random.default_rng(width)
    prims = []
    for k in range(4):
        d = np.exp2(rng.uniform(-width, width, (cfg.ni, cfg.nj)))
        if k in (1, 2):
            d *= rng.choice([-1.0, 1.0, 0.0], d.shape, p=[0.4, 0.4, 0.2])
        d[20:50, 10:40] = d[20, 10]  # a flat stretch
        a = np.zeros(cfg.halo_shape, order="F")
        a[g:g + cfg.ni, g:g + cfg.nj] = d
        prims.append(a)
    ref = oracle.OracleFluid(cfg)
    ref.set_primitive(*prims)
    f = Fluid(cfg).initialize(*prims)
    want_code = ref.integrate(1e-6)
    _, code = f.integrate(1e-6)
    want, got = ref.state(), f.state(FIELDS)
    f.close()
    assert code == want_code
    for k in FIELDS:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    for a in prims:  # and a residual with a NaN and an infinity among the values
        a[g + 5, g + 7], a[g + 60, g + 30] = np.nan, np.inf
    want = oracle.solve(cfg, *[p.copy(order="F") for p in prims])
    got = FluxSolver(cfg).solve(*[p.copy(order="F") for p in prims])
    for k in range(4):
        np.testing.assert_array_equal(got[k], want[k])
