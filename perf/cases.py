"""What the performance of this framework is measured on: whole calls through its public entry
points, from the initial state in host arrays to the result in host arrays.

Four kinds of call, as user programs make them:

* ``solve``    -- one grid: ``Fluid.initialize``, ``Fluid.run`` for a number of steps, ``Fluid.state``;
* ``loop``     -- one grid stepped from the host, one ``Fluid.integrate`` per step (the reference's
  own time loop, which looks at dt and the error code of every step);
* ``batch``    -- many grids of uneven sizes in one ``Batch``: added, advanced in chunks until none
  is running, their states fetched and removed (parameter sweeps, and the served request stream);
* ``residual`` -- ``FluxSolver.solve``: the semi-discrete residual of a host state.

``exact`` integrates the same inputs with plain torch operations in 64 bits.
"""
import math

import numpy as np
import torch

from fvleg_2d_gb300.batch import Batch
from fvleg_2d_gb300.config import SchemeConfig
from fvleg_2d_gb300.fluid import FluxSolver, Fluid

FIELDS = ("rho", "rho_u", "rho_v", "rho_E")
ZERO_GRADIENT = "zero_gradient"
SHEAR = "shear"          # Kelvin-Helmholtz: periodic in x, reflecting walls in y
TUBE = "tube"            # shock tube: open in x, reflecting walls in y
QUADRANTS = "quadrants"  # four-state 2-D Riemann problem, open on every side
CIRCLES = "circles"      # random circles over a background, open on every side
RK_STAGES = {"ssp_rk2": 2, "ssp_rk3": 3, "rk(1,3)": 3, "rk(2,4)": 4}
SERVED_FLUXES = ("AUSM+-up", "AUSMPW+", "SLAU", "HLLC", "Roe")


def _case(kind, problem, ni, nj, precision, flux, limiter, rk, steps, **more):
    c = dict(kind=kind, problem=problem, ni=ni, nj=nj, precision=precision, flux=flux,
             limiter=limiter, rk=rk, steps=steps, harten=False, layered=False)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a coarse grid stepped from the host, where latency is everything
        _case("loop", QUADRANTS, 64, 48, "fp64", "HLLC", "van_leer", "ssp_rk3", 4,
              name="loop_64x48_fp64"),
        # the shock-tube configuration at its own size: hundreds of short steps on the device
        _case("solve", TUBE, 400, 40, "fp64", "AUSMPW+", "minmod", "ssp_rk2", 200,
              name="tube_400x40_fp64"),
        # the headline configuration in the drop-in precision, at its own size (the largest call)
        _case("solve", QUADRANTS, 4096, 4096, "fp64", "HLLC", "van_leer", "ssp_rk3", 5,
              name="quadrants_4096_fp64"),
        # the same in the fast precision
        _case("solve", QUADRANTS, 4096, 4096, "mixed", "HLLC", "van_leer", "ssp_rk3", 24,
              name="quadrants_4096_mixed"),
        # a medium grid of odd shape in the accurate mixed precision
        _case("solve", QUADRANTS, 1501, 1099, "mixed_df", "HLLC", "van_leer", "ssp_rk3", 30,
              name="quadrants_1501x1099_df"),
        # the shear-layer configuration (Roe, superbee, periodic and reflecting sides), ragged
        _case("solve", SHEAR, 1000, 700, "fp64", "Roe", "superbee", "ssp_rk3", 15,
              name="shear_1000x700_fp64"),
        # the same, large, with the entropy fix, in the fast precision
        _case("solve", SHEAR, 3000, 2010, "mixed", "Roe", "superbee", "ssp_rk3", 40, harten=True,
              name="shear_3000x2010_mixed"),
        # the batched sweep (SLAU, fifth-order limiter) in each precision
        _case("batch", CIRCLES, 512, 64, "fp64", "SLAU", "MLP5", "ssp_rk2", 48, count=16,
              name="sweep_fp64"),
        _case("batch", CIRCLES, 512, 64, "mixed_df", "SLAU", "MLP5", "ssp_rk2", 96, count=16,
              name="sweep_df"),
        _case("batch", CIRCLES, 1024, 64, "mixed", "SLAU", "MLP5", "ssp_rk2", 192, count=16,
              name="sweep_mixed"),
        # served requests: five schemes side by side, retiring one after the other
        _case("batch", CIRCLES, 768, 128, "mixed", "served", "minmod", "ssp_rk2", 160, count=12,
              name="served_mixed"),
        # one residual of a host state, third-order limiter
        _case("residual", QUADRANTS, 801, 603, "fp64", "AUSMPW+", "MLP3", "ssp_rk3", 1,
              name="residual_801x603_fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "batch", "loop", "residual"])
    precision = rng.choice(["fp64", "mixed", "mixed_df"])
    flux = rng.choice(["AUSMPW+", "SLAU", "SLAU2", "SD-SLAU", "Roe", "AUSM+-up", "HLLC"])
    limiter = rng.choice(["minmod", "superbee", "van_leer", "minmod", "van_leer", "MLP3", "MLP5"])
    rk = rng.choice(["ssp_rk2", "ssp_rk3", "ssp_rk2", "ssp_rk3", "rk(1,3)", "rk(2,4)"])
    problem = rng.choice([QUADRANTS, SHEAR, TUBE, CIRCLES])
    # cell updates in a pass: a fraction of the largest listed call's
    updates = {"fp64": 2.0e7, "mixed": 2.0e8, "mixed_df": 6.0e7}[precision]
    if kind == "batch":
        hi = _log(rng, 128, 768)
        count = rng.randrange(4, 17)
        steps = max(16, min(160, int(updates / 4 / (count * hi * hi / 4))))
        return _case(kind, CIRCLES, hi, 64, precision, rng.choice([flux, "served"]), limiter,
                     rk, steps, count=count)
    ni = _log(rng, 48, 2400)
    nj = max(24, min(2400, int(ni * math.exp(rng.uniform(-1.2, 0.6)))))
    if kind == "loop":
        ni, nj = min(ni, 700), min(nj, 700)
        return _case(kind, problem, ni, nj, precision, flux, limiter, rk, 4)
    if kind == "residual":
        # the residual entry point is the drop-in's: real64 in, real64 out
        return _case(kind, problem, ni, nj, "fp64", flux, limiter, "ssp_rk3", 1)
    steps = max(2, min(120, int(updates / 2 / (ni * nj))))
    return _case(kind, problem, ni, nj, precision, flux, limiter, rk, steps,
                 layered=rng.random() < 0.2, harten=rng.random() < 0.3)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _sizes(case):
    """The grids of a batch: long sides log-uniform down to `nj`, aspect ratios up to 4, in
    multiples of 16 (they go with the case, not with the seed)."""
    rng = np.random.default_rng(case["ni"] * 1000003 + case["count"] * 101 + case["steps"])
    out = []
    for _ in range(case["count"]):
        nx = math.exp(rng.uniform(math.log(case["nj"]), math.log(case["ni"])))
        ny = nx / rng.uniform(1.0, 4.0)
        out.append((max(16, int(nx) // 16 * 16), max(16, int(ny) // 16 * 16)))
    return out


def _steps_of(case, k):
    """The served requests end at different times: their step limits are spread out."""
    return case["steps"] if case["flux"] != "served" else \
        max(8, case["steps"] * (k + 2) // (case["count"] + 1))


def _bcs(problem):
    x = "periodic" if problem == SHEAR else ZERO_GRADIENT
    y = "symmetry" if problem in (SHEAR, TUBE) else ZERO_GRADIENT
    return {"+x": x, "-x": x, "+y": y, "-y": y}


def _config(case, ni, nj, flux):
    # unit length along x; the tube is a tenth as high, the batch's cells are square
    height = {TUBE: 0.1, CIRCLES: nj / ni}.get(case["problem"], 1.0)
    return SchemeConfig(
        ni=ni, nj=nj, dx=1.0 / ni, dy=height / nj, flux_solver=flux, limiter=case["limiter"],
        integration_strategy=case["rk"], precision=case["precision"], gamma=1.4,
        cfl=0.5 if case["rk"] == "ssp_rk2" else 0.4, bc=_bcs(case["problem"]),
        roe_entropy_fix="harten" if case["harten"] else "reference")


def _primitives(cfg, problem, rng):
    """(4, nj, ni) rho, u, v, p on the GPU: the problem's piecewise states, with smooth waves of
    a few percent over them (a developed flow is flat nowhere)."""
    dev = "cuda"
    ni, nj = cfg.ni, cfg.nj
    x = (torch.arange(ni, dtype=torch.float64, device=dev) + 0.5) / ni
    y = (torch.arange(nj, dtype=torch.float64, device=dev) + 0.5) / nj
    W = torch.empty((4, nj, ni), dtype=torch.float64, device=dev)
    X, Y = x[None, :], y[:, None]

    def put(mask, state):
        for k in range(4):
            W[k].masked_fill_(mask, float(state[k]))

    everywhere = (X >= 0) & (Y >= 0)
    if problem == QUADRANTS:
        east, north = X >= 0.5, Y >= 0.5
        put(east & north, (1.5, 0.0, 0.0, 1.5))
        put(~east & north, (0.5323, 1.206, 0.0, 0.3))
        put(~east & ~north, (0.138, 1.206, 1.206, 0.029))
        put(east & ~north, (0.5323, 0.0, 1.206, 0.3))
    elif problem == SHEAR:
        put(everywhere, (1.0, -0.5, 0.0, 2.5))
        put(everywhere & ((Y - 0.5).abs() < 0.25), (2.0, 0.5, 0.0, 2.5))
        W[2] += 0.01 * torch.sin(4.0 * math.pi * X)
    elif problem == TUBE:
        put(everywhere & (X < 0.5), (1.0, 0.0, 0.0, 1.0))
        put(everywhere & (X >= 0.5), (0.125, 0.0, 0.0, 0.1))
    else:
        def state():
            return (rng.uniform(0.5, 2.0), rng.normal(0.0, 0.25), rng.normal(0.0, 0.25),
                    math.exp(rng.uniform(math.log(0.4), math.log(2.5))))
        put(everywhere, state())
        h = nj / ni
        for _ in range(int(rng.integers(4, 17))):
            cx, cy, r = rng.uniform(0, 1), rng.uniform(0, h), rng.uniform(0.03, 0.25)
            put((X - cx) ** 2 + (Y * h - cy) ** 2 < r * r, state())

    def wave():
        kx, ky = int(rng.integers(1, 6)), int(rng.integers(1, 6))
        a, b = rng.uniform(0, 2 * math.pi, 2)
        return torch.cos(2 * math.pi * kx * X + a) * torch.cos(2 * math.pi * ky * Y + b)

    amplitude = 0.002 if problem == TUBE else 0.02
    for k in (0, 3):
        W[k] *= 1.0 + amplitude * wave()
    for k in (1, 2):
        W[k] += amplitude * wave()
    return W


def _host_fields(cfg, W):
    """Halo-padded Fortran-ordered float64 arrays, the layout of the reference's fields."""
    g = cfg.ghost_layers()
    out = []
    for k in range(4):
        a = torch.zeros((cfg.nj + 2 * g, cfg.ni + 2 * g), dtype=torch.float64)
        a[g:g + cfg.nj, g:g + cfg.ni] = W[k].cpu()
        out.append(a.numpy().T)
    return out


def _nodes(case, cfg):
    """A layered grid: three layers along x whose cells are 1 : 2 : 3 wide."""
    w = np.ones(cfg.ni)
    w[cfg.ni // 3:] = 2.0
    w[2 * cfg.ni // 3:] = 3.0
    x = np.concatenate([[0.0], np.cumsum(w / w.sum())])
    return x, np.linspace(0.0, cfg.dy * cfg.nj, cfg.nj + 1)


def _instances(case, seed):
    """[(configuration, device primitives, step limit)] of a case."""
    rng = np.random.default_rng(seed)
    if case["kind"] != "batch":
        cfg = _config(case, case["ni"], case["nj"], case["flux"])
        return [(cfg, _primitives(cfg, case["problem"], rng), case["steps"])]
    out = []
    for k, (ni, nj) in enumerate(_sizes(case)):
        flux = SERVED_FLUXES[k % len(SERVED_FLUXES)] if case["flux"] == "served" else case["flux"]
        cfg = _config(case, ni, nj, flux)
        out.append((cfg, _primitives(cfg, case["problem"], rng), _steps_of(case, k)))
    return out


def prepare(case, seed):
    inst = [(cfg, _host_fields(cfg, W), n) for cfg, W, n in _instances(case, seed)]
    cfg, prims, steps = inst[0]
    s = {"case": case, "instances": inst, "prims": prims, "steps": steps}
    if case["kind"] == "batch":
        s["batch"] = Batch(case["count"], precision=case["precision"],
                           integration_strategy=case["rk"])
    elif case["kind"] == "residual":
        s["solver"] = FluxSolver(cfg)
    else:
        s["fluid"] = Fluid(cfg)
        if case["layered"]:
            s["fluid"].set_rectilinear(*_nodes(case, cfg))
    return s


def run(state):
    kind = state["case"]["kind"]
    if kind == "solve":
        f = state["fluid"].initialize(*state["prims"])
        f.run(math.inf, state["steps"])
        return f.state(FIELDS)
    if kind == "loop":
        f = state["fluid"].initialize(*state["prims"])
        dts, codes = [], []
        for _ in range(state["steps"]):
            dt, code = f.integrate()
            dts.append(dt)
            codes.append(code)
        return {"dt": dts, "code": codes, **f.state(FIELDS)}
    if kind == "residual":
        return state["solver"].solve(*state["prims"])
    b = state["batch"]
    slots = [b.add(cfg, prims, max_steps=n) for cfg, prims, n in state["instances"]]
    b.run_until_done(chunk=16)
    out = []
    for slot in slots:
        out.append(b.state(slot))
        b.remove(slot)
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
# arithmetic operations per cell and stage: reconstruction of four variables in two directions,
# two edge fluxes, the primitive recovery, the divergence and the stage combine
_RECON_FLOPS = {"minmod": 100, "superbee": 110, "van_leer": 110, "MLP3": 240, "MLP5": 350}
_FLUX_FLOPS = {"HLLC": 120, "Roe": 220, "SLAU": 140, "SLAU2": 140, "SD-SLAU": 190,
               "AUSMPW+": 180, "AUSM+-up": 140}


def work(case):
    if case["kind"] == "batch":
        grids = [(ni * nj, SERVED_FLUXES[k % 5] if case["flux"] == "served" else case["flux"],
                  _steps_of(case, k)) for k, (ni, nj) in enumerate(_sizes(case))]
    else:
        grids = [(case["ni"] * case["nj"], case["flux"], case["steps"])]
    ns = RK_STAGES[case["rk"]]
    nbytes = flops = 0.0
    for cells, flux, steps in grids:
        per = _RECON_FLOPS[case["limiter"]] + _FLUX_FLOPS[flux] + 70
        if case["kind"] == "residual":
            nbytes += 64.0 * cells
            flops += per * cells
            continue
        # state: read in the first stage, read with the step's start in the others; written by all
        nbytes += cells * steps * (64.0 + 96.0 * (ns - 1)) + 64.0 * cells
        flops += per * cells * steps * ns
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------------------------
_G = 3  # ghost layers of the torch integration
_GAMMA = 1.4
_GM1 = _GAMMA - 1.0
_HQ = _GAMMA / _GM1


def _ghosts(n, kind, dev):
    i = torch.arange(-_G, n + _G, device=dev)
    flip = torch.zeros(n + 2 * _G, dtype=torch.bool, device=dev)
    if kind == "periodic":
        i = i % n
    elif kind == "symmetry":
        flip = (i < 0) | (i >= n)
        i = torch.where(i < 0, -i - 1, torch.where(i >= n, 2 * n - 1 - i, i))
    return i.clamp(0, n - 1), flip


def _padded(W, bc):
    jy, fy = _ghosts(W.shape[1], bc["+y"], W.device)
    ix, fx = _ghosts(W.shape[2], bc["+x"], W.device)
    P = W[:, jy][:, :, ix]
    P[1][:, fx] *= -1.0
    P[2][fy] *= -1.0
    return P


def _flushed(d):
    return torch.where(d.abs() < 2.0 ** -52, torch.zeros_like(d), d)


def _phi(limiter, r):
    if limiter == "minmod":
        return r.clamp(0.0, 1.0)
    if limiter == "superbee":
        return torch.maximum((2.0 * r).clamp(0.0, 1.0), r.clamp(max=2.0)).clamp(min=0.0)
    return torch.where(r > 0, 2.0 * r / (1.0 + r), torch.zeros_like(r))


def _edge_states(limiter, Q):
    """Left and right states of every edge; Q(n, t): the cells n along and t across from the
    edge's left cell."""
    a, b, c, d = Q(-1, 0), Q(0, 0), Q(1, 0), Q(2, 0)
    dm, d0, dp = _flushed(b - a), _flushed(c - b), _flushed(d - c)
    if limiter in ("minmod", "superbee", "van_leer"):
        return (b + 0.5 * _phi(limiter, d0 / (dm + 1e-16)) * dm,
                c - 0.5 * _phi(limiter, d0 / (dp + 1e-16)) * dp)
    S = 1e-30
    rL, rR = d0 / (dm + S), d0 / (dp + S)
    if limiter == "MLP5":
        dm3, dp5 = _flushed(a - Q(-2, 0)), _flushed(Q(3, 0) - d)
        bL = (-2.0 / (dm / (dm3 + S) + S) + 11.0 + 24.0 * rL - 3.0 * rL * (dp / (d0 + S))) / 30.0
        bR = (-2.0 / (dp / (dp5 + S) + S) + 11.0 + 24.0 * rR - 3.0 * rR * (dm / (d0 + S))) / 30.0
    else:
        bL, bR = (1.0 + 2.0 * rL) / 3.0, (1.0 + 2.0 * rR) / 3.0
    tL = (Q(0, 1) - Q(0, -1)).abs() / ((c - a).abs() + S)
    tR = (Q(1, 1) - Q(1, -1)).abs() / ((d - b).abs() + S)

    def side(r, r_other, beta, t_own, t_other):
        al = 2.0 * r.clamp(min=1.0) * (1.0 + (t_other / (r_other + S)).clamp(min=0.0)) / (1.0 + t_own)
        al = al.clamp(1.0, 2.0)
        phi = torch.minimum(torch.minimum(al * r, al), beta).clamp(min=0.0)
        return torch.where(r > 0, phi, torch.zeros_like(phi))

    return (b + 0.5 * side(rL, rR, bL, tL, tR) * dm, c - 0.5 * side(rR, rL, bR, tR, tL) * dp)


def _flux_hllc(L, R, **_):
    (rL, qL, tL, pL), (rR, qR, tR, pR) = L, R
    cL, cR = (_GAMMA * pL / rL).sqrt(), (_GAMMA * pR / rR).sqrt()
    ps = (0.5 * (pL + pR) - 0.5 * (qR - qL) * (0.5 * (rL + rR)) * (0.5 * (cL + cR))).clamp(min=0.0)
    gf = (_GAMMA + 1.0) / (2.0 * _GAMMA)
    one = torch.ones_like(ps)
    SL = qL - cL * torch.where(ps <= pL, one, (1.0 + gf * (ps / pL - 1.0)).clamp(min=0.0).sqrt())
    SR = qR + cR * torch.where(ps <= pR, one, (1.0 + gf * (ps / pR - 1.0)).clamp(min=0.0).sqrt())
    Ss = (pR - pL + rL * qL * (SL - qL) - rR * qR * (SR - qR)) / (rL * (SL - qL) - rR * (SR - qR))

    def side(r, q, t, p, S):
        E = p / _GM1 + 0.5 * r * (q * q + t * t)
        f = r * (S - q) / (S - Ss)
        U = (r, r * q, r * t, E)
        F = (r * q, r * q * q + p, r * q * t, q * (E + p))
        Us = (f, f * Ss, f * t, f * (E / r + (Ss - q) * (Ss + p / (r * (S - q)))))
        return F, tuple(F[k] + S * (Us[k] - U[k]) for k in range(4))

    FL, FsL = side(rL, qL, tL, pL, SL)
    FR, FsR = side(rR, qR, tR, pR, SR)
    return [torch.where(SL >= 0, FL[k], torch.where(Ss >= 0, FsL[k],
            torch.where(SR > 0, FsR[k], FR[k]))) for k in range(4)]


def _flux_slau(L, R, variant="SLAU", P=None, **_):
    (rL, qL, tL, pL), (rR, qR, tR, pR) = L, R
    cb = 0.5 * ((_GAMMA * pL / rL).sqrt() + (_GAMMA * pR / rR).sqrt())
    Vb = (rL * qL.abs() + rR * qR.abs()) / (rL + rR)
    v2 = 0.5 * (qL * qL + tL * tL + qR * qR + tR * tR)
    chi = (1.0 - (v2.sqrt() / cb).clamp(max=1.0)) ** 2
    Mp, Mm = qL / cb, qR / cb
    pb, rb = 0.5 * (pL + pR), 0.5 * (rL + rR)
    Bp = torch.where(Mp.abs() < 1, 0.25 * (2.0 - Mp) * (Mp + 1.0) ** 2,
                     0.5 * (1.0 + torch.copysign(torch.ones_like(Mp), Mp)))
    Bm = torch.where(Mm.abs() < 1, 0.25 * (2.0 + Mm) * (Mm - 1.0) ** 2,
                     0.5 * (1.0 + torch.copysign(torch.ones_like(Mm), -Mm)))

    def cut(d):
        return torch.where((d.abs() < 2.0 ** -52) | (d.abs() < 5e-3 * pb), torch.zeros_like(d), d)

    dp = cut(pR - pL)
    diss = chi
    if variant == "SD-SLAU":
        pairs = ((0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, -1, 1), (2, 0, 1), (1, 1, 1))
        m = dp.abs()
        for n, t, own in pairs:
            m = torch.maximum(m, cut(P(n, t) - P(own, 0)).abs())
        ratio = (0.01 * dp.abs() / pb + 0.01) / (m / pb + 0.01)
        diss = (ratio ** 2).clamp(max=1.0) * (1.0 - (Vb / cb).abs()).clamp(min=0.0)
    mid = pb + 0.5 * (Bp - Bm) * (pL - pR)
    pt = mid + (v2.sqrt() * rb * cb if variant == "SLAU2" else (1.0 - chi) * pb) * (Bp + Bm - 1.0)
    g = -(Mp.clamp(-1.0, 0.0) * Mm.clamp(0.0, 1.0))
    mf = 0.5 * (rL * qL + rR * qR - Vb * (rR - rL)) * (1.0 - g) - diss / (2.0 * cb) * dp
    mL, mR = mf.clamp(min=0.0), mf.clamp(max=0.0)
    HL = _HQ * pL / rL + 0.5 * (qL * qL + tL * tL)
    HR = _HQ * pR / rR + 0.5 * (qR * qR + tR * tR)
    return [mf, mL * qL + mR * qR + pt, mL * tL + mR * tR, mL * HL + mR * HR]


def _flux_roe(L, R, P=None, harten=False, **_):
    (rL, qL, tL, pL), (rR, qR, tR, pR) = L, R
    ra = (rL * rR).sqrt()
    HL = _HQ * pL / rL + 0.5 * (qL * qL + tL * tL)
    HR = _HQ * pR / rR + 0.5 * (qR * qR + tR * tR)
    w = ra / rL
    q, t, H = (qL + w * qR) / (1.0 + w), (tL + w * tR) / (1.0 + w), (HL + w * HR) / (1.0 + w)
    k = 0.5 * (q * q + t * t)
    c2 = _GM1 * (H - k)
    c = c2.sqrt()
    cL, cR = (_GAMMA * pL / rL).sqrt(), (_GAMMA * pR / rR).sqrt()
    dq, dt_, dr, dp = qR - qL, tR - tL, rR - rL, pR - pL
    e1, e2, e4 = torch.minimum(q - c, qL - cL).abs(), q.abs(), torch.maximum(q + c, qR + cR).abs()
    if harten:
        dl = 0.1 * c
        e1, e2, e4 = (torch.where(e > dl, e, 0.5 * (e * e + dl * dl) / dl) for e in (e1, e2, e4))
    a1, a5 = e1 * (dp - ra * c * dq) / (2.0 * c2), e4 * (dp + ra * c * dq) / (2.0 * c2)
    a3, a4 = e2 * (dr - dp / c2), e2 * ra
    F = [0.5 * (rR * q + rL * q - (a1 + a3 + a5)),
         0.5 * (rR * qR * q + pR + rL * qL * q + pL - (a1 * (q - c) + a3 * q + a5 * (q + c))),
         0.5 * (rR * tR * q + rL * tL * q - ((a1 + a3 + a5) * t + a4 * dt_)),
         0.5 * (rR * HR * q + rL * HL * q -
                (a1 * (H - c * q) + a3 * k + a4 * (t * dt_) + a5 * (H + c * q)))]
    # the shear correction where a pressure sensor of the neighbourhood fires
    jump = torch.zeros_like(c, dtype=torch.bool)
    for (n0, t0), (n1, t1) in _ROE_PAIRS[P.axis]:
        x, y = P(n0, t0), P(n1, t1)
        jump |= ~((y - x).abs() / (torch.minimum(x, y) + 1e-16) < 1.0)
    f = 0.5 * jump.double() * ra * c
    F[1] = F[1] - f * ((cR - cL).abs() / torch.maximum(cR, cL)) * dq
    # along an x edge the tangential term is +dv, along a y edge -du
    F[2] = F[2] - f * (dt_ if P.axis == 0 else -dt_)
    return F


# pairs of cells ((n, t), (n, t)) of the sensor, along x edges and along y edges
_ROE_PAIRS = (
    (((0, 0), (1, 0)), ((0, 0), (0, 1)), ((0, 0), (0, -1)), ((0, 1), (1, 1)), ((0, -1), (1, -1))),
    (((0, 0), (1, 0)), ((0, 0), (0, -1)), ((0, 0), (0, 1)), ((1, 0), (1, -1)), ((1, 0), (1, 1))),
)


def _flux_ausmpw(L, R, P=None, **_):
    (rL, qL, tL, pL), (rR, qR, tR, pR) = L, R
    UL, UR = qL, qR
    VL, VR = tL, tR
    ML = (qL * qL + tL * tL).sqrt() / (_GAMMA * pL / rL).sqrt()
    MR = (qR * qR + tR * tR).sqrt() / (_GAMMA * pR / rR).sqrt()
    low = (ML < 0.1) | (MR < 0.1)  # the low-Mach velocity blend
    f = torch.maximum(ML, MR).clamp(max=1.0)

    def blend(a, b):
        m, d = 0.5 * (a + b), 0.5 * f * (a - b)
        return torch.where(low, m + d, a), torch.where(low, m - d, b)

    qL, qR = blend(qL, qR)
    tL, tR = blend(tL, tR)
    HL = _HQ * pL / rL + 0.5 * (qL * qL + tL * tL)
    HR = _HQ * pR / rR + 0.5 * (qR * qR + tR * tR)
    Hn = torch.minimum(HL - 0.5 * VL * VL, HR - 0.5 * VR * VR)
    cs = (2.0 * (_GM1 / (_GAMMA + 1.0)) * Hn).sqrt()
    c = cs * cs / torch.where(UL + UR < 0, torch.maximum(UR.abs(), cs), torch.maximum(UL.abs(), cs))
    ML, MR = UL / c, UR / c
    one = torch.ones_like(ML)
    Mp = torch.where(ML.abs() > 1, 0.5 * (ML + ML.abs()), 0.25 * (ML + 1.0) ** 2)
    Mm = torch.where(MR.abs() > 1, 0.5 * (MR - MR.abs()), -0.25 * (MR - 1.0) ** 2)
    Pp = torch.where(ML.abs() > 1, 0.5 * (1.0 + torch.copysign(one, ML)),
                     0.25 * (ML + 1.0) ** 2 * (2.0 - ML) + 0.125 * ML * (ML * ML - 1.0) ** 2)
    Pm = torch.where(MR.abs() > 1, 0.5 * (1.0 - torch.copysign(one, MR)),
                     0.25 * (MR - 1.0) ** 2 * (2.0 + MR) - 0.125 * MR * (MR * MR - 1.0) ** 2)
    ps = pL * Pp + pR * Pm
    w = 1.0 - torch.minimum(pL / pR, pR / pL) ** 3
    if P.axis == 0:
        near = (P(0, -1), P(1, -1), P(0, 1), P(1, 1))
    else:
        near = (P(0, 1), P(1, 1), P(0, -1), P(1, -1))
    least = torch.minimum(torch.minimum(near[0], near[1]), torch.minimum(near[2], near[3]))
    m = (least / torch.minimum(pL, pR)).clamp(max=1.0) ** 2
    fL, fR = (pL / ps - 1.0) * m, (pR / ps - 1.0) * m
    back = Mp + Mm < 0
    aL = torch.where(back, Mp * w * (1.0 + fL), Mp + Mm * ((1.0 - w) * (1.0 + fR) - fL))
    aR = torch.where(back, Mm + Mp * ((1.0 - w) * (1.0 + fL) - fR), Mm * w * (1.0 + fR))
    mL, mR = aL * c * rL, aR * c * rR
    return [mL + mR, mL * qL + mR * qR + ps, mL * tL + mR * tR, mL * HL + mR * HR]


def _flux_ausm_up(L, R, **_):
    (rL, qL, tL, pL), (rR, qR, tR, pR) = L, R
    gf = 2.0 * _GM1 / (_GAMMA + 1.0)
    HL = _HQ * pL / rL + 0.5 * (qL * qL + tL * tL)
    HR = _HQ * pR / rR + 0.5 * (qR * qR + tR * tR)
    aL, aR = (gf * HL.abs()).sqrt(), (gf * HR.abs()).sqrt()
    a = torch.minimum(aL * aL / torch.maximum(aL, qL), aR * aR / torch.maximum(aR, -qR))
    ML, MR = qL / a, qR / a
    p2L, m2L = 0.25 * (ML + 1.0) ** 2, -0.25 * (ML - 1.0) ** 2
    p2R, m2R = 0.25 * (MR + 1.0) ** 2, -0.25 * (MR - 1.0) ** 2
    beta, alpha = 1.0 / 8.0, 3.0 / 16.0
    Mp = torch.where(ML.abs() >= 1, 0.5 * (ML + ML.abs()), p2L * (1.0 - 16.0 * beta * m2L))
    Mm = torch.where(MR.abs() >= 1, 0.5 * (MR - MR.abs()), m2R * (1.0 + 16.0 * beta * p2R))
    dp = _flushed(pR - pL)
    Mpr = -0.25 * (1.0 - 0.5 * (ML + MR)).clamp(min=0.0) * dp / (0.5 * (rL + rR) * a * a)
    M = Mp + Mm + Mpr
    M = torch.where(M.abs() < 1e-13, torch.zeros_like(M), M)
    Pp = torch.where(ML.abs() >= 1, 0.5 * (ML + ML.abs()) / ML,
                     p2L * ((2.0 - ML) - 16.0 * alpha * ML * m2L))
    Pm = torch.where(MR.abs() >= 1, 0.5 * (MR - MR.abs()) / MR,
                     m2R * ((-2.0 - MR) + 16.0 * alpha * MR * p2R))
    ph = Pp * pL + Pm * pR - 0.75 * Pp * Pm * (rL + rR) * a * (qR - qL)
    left = M > 0
    r, q, t, H = (torch.where(left, x, y) for x, y in ((rL, rR), (qL, qR), (tL, tR), (HL, HR)))
    mf = M * a * r
    return [mf, mf * q + ph, mf * t, mf * H]


_FLUXES = {"HLLC": _flux_hllc, "Roe": _flux_roe, "AUSMPW+": _flux_ausmpw,
           "AUSM+-up": _flux_ausm_up, "SLAU": _flux_slau, "SLAU2": _flux_slau,
           "SD-SLAU": _flux_slau}


def _edge_fluxes(cfg, P, axis):
    nj, ni = P.shape[1] - 2 * _G, P.shape[2] - 2 * _G

    def Q(n, t):
        if axis == 0:
            return P[:, _G + t:_G + t + nj, _G - 1 + n:_G + n + ni]
        return P[:, _G - 1 + n:_G + n + nj, _G + t:_G + t + ni]

    L, R = _edge_states(cfg.limiter, Q)
    normal = (0, 1, 2, 3) if axis == 0 else (0, 2, 1, 3)

    def pressure(n, t):
        return Q(n, t)[3]

    pressure.axis = axis
    F = _FLUXES[cfg.flux_solver]([L[k] for k in normal], [R[k] for k in normal], P=pressure,
                                 variant=cfg.flux_solver, harten=cfg.roe_entropy_fix == "harten")
    return torch.stack([F[k] for k in normal])


def _residual(cfg, W, wx, wy):
    P = _padded(W, cfg.bc)
    Fi, Fj = _edge_fluxes(cfg, P, 0), _edge_fluxes(cfg, P, 1)
    return -((Fi[:, :, 1:] - Fi[:, :, :-1]) / wx + (Fj[:, 1:] - Fj[:, :-1]) / wy)


def _conserved(W):
    r, u, v, p = W
    return torch.stack([r, r * u, r * v, p / _GM1 + 0.5 * r * (u * u + v * v)])


def _primitive(U):
    r, ru, rv, E = U
    u, v = ru / r, rv / r
    return torch.stack([r, u, v, _GM1 * (E - 0.5 * r * (u * u + v * v))])


_ALPHAS = {"rk(1,3)": (0.1481, 0.4, 1.0), "rk(2,4)": (0.1084, 0.2602, 0.5052, 1.0)}


def _advance(cfg, W, steps, wx, wy):
    U, dts = _conserved(W), []
    for _ in range(steps):
        cs = (_GAMMA * W[3] / W[0]).sqrt()
        dt = (cfg.cfl / ((W[1].abs() + cs) / wx + (W[2].abs() + cs) / wy)).min()
        dts.append(dt)
        if cfg.integration_strategy in _ALPHAS:
            V = U
            for a in _ALPHAS[cfg.integration_strategy]:
                V = U + (dt * a) * _residual(cfg, W, wx, wy)
                W = _primitive(V)
            U = V
            continue
        V = U + dt * _residual(cfg, W, wx, wy)
        if cfg.integration_strategy == "ssp_rk2":
            U = 0.5 * U + 0.5 * V + 0.5 * dt * _residual(cfg, _primitive(V), wx, wy)
        else:
            V = 0.75 * U + 0.25 * V + 0.25 * dt * _residual(cfg, _primitive(V), wx, wy)
            U = U / 3.0 + 2.0 * V / 3.0 + (2.0 / 3.0) * dt * _residual(cfg, _primitive(V), wx, wy)
        W = _primitive(U)
    return U, dts


def _field(cfg, a):
    g = cfg.ghost_layers()
    out = torch.zeros((cfg.nj + 2 * g, cfg.ni + 2 * g), dtype=torch.float64)
    out[g:g + cfg.nj, g:g + cfg.ni] = a.cpu()
    return out.numpy().T


def exact(case, seed):
    # a stage of the torch integration is about 500 kernels, 60 ns a cell of a large grid
    inst = _instances(case, seed)
    ns = RK_STAGES[case["rk"]]
    if sum(n * ns * (8e-3 + 6e-9 * 10 * c.ni * c.nj) for c, _, n in inst) > 60.0:
        return None
    out = []
    for cfg, W, steps in inst:
        if case["layered"]:
            xn, yn = (torch.from_numpy(np.diff(a)).cuda() for a in _nodes(case, cfg))
            wx, wy = xn[None, :], yn[:, None]
        else:
            wx, wy = cfg.dx, cfg.dy
        if case["kind"] == "residual":
            return tuple(_field(cfg, a) for a in _residual(cfg, W, wx, wy))
        U, dts = _advance(cfg, W, steps, wx, wy)
        fields = {k: _field(cfg, a) for k, a in zip(FIELDS, U)}
        if case["kind"] == "solve":
            return fields
        if case["kind"] == "loop":
            return {"dt": [float(d) for d in dts], "code": [None] * steps, **fields}
        out.append(fields)
    return out
