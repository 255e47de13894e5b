"""Tile edges of the stage kernels: grids around the tile widths and block heights, every launch
shape and register budget, and reconstruction data at the limiters' decision points.  FP64 runs
equal the oracle bit for bit; every precision's result is independent of the launch shape."""
import numpy as np
import pytest

from conftest import random_prims
from fvleg_2d_gb300.batch import Batch
from fvleg_2d_gb300.config import SchemeConfig
from fvleg_2d_gb300.fluid import Fluid, FluxSolver

pytestmark = pytest.mark.gpu
FIELDS = ("rho", "rho_u", "rho_v", "rho_E")
# 28 / 60 / 124 cells fill a tile of 32 / 64 / 128 columns with 2 ghost layers (26 / 58 with 3)
SIZES = [(3, 3), (28, 4), (29, 5), (58, 9), (61, 33), (124, 7), (125, 66)]


def _cfg(ni, nj, limiter, flux, precision="fp64", **kw):
    return SchemeConfig(ni=ni, nj=nj, dx=1.0 / ni, dy=1.0 / nj, flux_solver=flux, limiter=limiter,
                        gamma=1.4, cfl=0.3, precision=precision, integration_strategy="ssp_rk3",
                        bc={"+x": "zero_gradient", "-x": "symmetry", "+y": "periodic",
                            "-y": "periodic"}, **kw)


@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("limiter,flux", [("van_leer", "HLLC"), ("superbee", "Roe"),
                                          ("minmod", "SD-SLAU"), ("MLP5", "SLAU"),
                                          ("MLP3", "AUSMPW+")])
def test_fp64_tiles_equal_the_oracle(oracle, ni, nj, limiter, flux):
    cfg = _cfg(ni, nj, limiter, flux)
    prims = random_prims(cfg, np.random.default_rng(ni * 100 + nj))
    ref = oracle.OracleFluid(cfg)
    ref.set_primitive(*prims)
    for _ in range(2):
        ref.integrate(ref.get_timestep())
    want = ref.state()
    for plan, variant in ((None, 0), ((64, 1), 0), ((64, 3), 1), ((128, 6), 2), ((256, 5), 0),
                          ((256, 40), 2)):
        f = Fluid(cfg).initialize(*prims)
        if plan:
            f.set_plan(*plan)
            f.set_kernel_variant(variant)
            assert f.get_plan() == plan
        f.run_timed(2)
        got = f.state(FIELDS)
        f.close()
        for k in FIELDS:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {plan} {variant}")


@pytest.mark.parametrize("precision", ["mixed", "mixed_df"])
@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("limiter,flux", [("van_leer", "HLLC"), ("minmod", "AUSMPW+"),
                                          ("MLP5", "SLAU")])
def test_result_is_independent_of_the_shape(precision, ni, nj, limiter, flux):
    cfg = _cfg(ni, nj, limiter, flux, precision)
    prims = random_prims(cfg, np.random.default_rng(ni * 100 + nj))
    states = []
    for plan in (None, (64, 1), (64, 4), (128, 7), (256, 30)):
        f = Fluid(cfg).initialize(*prims)
        if plan:
            f.set_plan(*plan)
        f.run_timed(2)
        states.append(f.state(FIELDS))
        f.close()
    for s in states[1:]:
        for k in FIELDS:
            np.testing.assert_array_equal(s[k], states[0][k])


def _decision_field(cfg, rng):
    """Values whose neighbouring differences have the ratios the limiters decide on: 0, 1/2, 1 and
    2, each also one unit in the last place off, differences at the epsilon flush and of either
    sign, flat stretches and exact zeros."""
    ratios = [0.0, 0.5, 1.0, 2.0, np.nextafter(0.5, 1), np.nextafter(1.0, 0), np.nextafter(2.0, 3),
              -1.0, 1e-15, 3.0]
    steps = np.where(rng.random((cfg.ni, cfg.nj)) < 0.5, 2.0 ** -6, 1e-3)
    steps = steps * rng.choice(ratios, size=steps.shape)
    a = np.cumsum(steps, axis=0) * (rng.random((cfg.ni, cfg.nj)) < 0.9)
    a[rng.random(a.shape) < 0.05] = 2.0 ** -52
    return a - a.mean(axis=0)


@pytest.mark.parametrize("limiter", ["minmod", "superbee", "van_leer", "MLP3", "MLP5"])
@pytest.mark.parametrize("flux", ["HLLC", "Roe", "AUSMPW+"])
def test_limiter_decisions_equal_the_oracle(oracle, limiter, flux):
    cfg = _cfg(66, 35, limiter, flux)
    g = cfg.ghost_layers()
    rng = np.random.default_rng(17)
    prims = [np.zeros(cfg.halo_shape, order="F") for _ in range(4)]
    for k, a in enumerate(prims):
        d = _decision_field(cfg, rng)
        if k in (0, 3):  # density and pressure: positive, a few jumps above a factor of two
            d = 1.0 + 0.4 * d / max(np.abs(d).max(), 1e-30)
            d[rng.random(d.shape) < 0.02] = 3.0
        a[g:g + cfg.ni, g:g + cfg.nj] = d
    want = oracle.solve(cfg, *[p.copy(order="F") for p in prims])
    got = FluxSolver(cfg).solve(*[p.copy(order="F") for p in prims])
    for k in range(4):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
@pytest.mark.parametrize("rows", [5, 12, 24, 28, 32])
def test_batch_rows_that_are_no_power_of_two(precision, rows):
    cfgs = [_cfg(ni, nj, "MLP5", "HLLC", precision) for ni, nj in [(59, 25), (200, 127), (16, 57)]]
    prims = [random_prims(c, np.random.default_rng(c.ni)) for c in cfgs]
    batch = Batch(len(cfgs), precision=precision, integration_strategy="ssp_rk3")
    batch.set_plan(128, rows)
    slots = [batch.add(c, p) for c, p in zip(cfgs, prims)]
    batch.step(3)
    for cfg, p, slot in zip(cfgs, prims, slots):
        f = Fluid(cfg).initialize(*p)
        f.run_timed(3)
        want = f.state(FIELDS)
        f.close()
        got = batch.state(slot)
        for k in FIELDS:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {cfg.ni}")
    batch.close()
