"""The mixed form takes densities and pressures over FP32's range, each by
itself: a member whose conserved densities are all scaled by a power of two
gives the scaled values of the unscaled one, and a thin, cold gas has finite
wave speeds."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu

STEPS = 30


@pytest.mark.parametrize("prec,model,case,limiter,flux",
                         [(prec, G.EULER, *c) for prec in (G.MIXED, G.FP64_FAST)
                          for c in (("cross", 0, "MUSCL"), ("totem_pole_1", 2, "MUSCL"),
                                    ("cross", 0, "Godunov"))] +
                         [(G.MIXED, G.ALLAIRE, "shocked_helium_bubble", 0, flux)
                          for flux in ("MUSCL", "Godunov")])
def test_scaled_densities_give_scaled_values(model, case, limiter, flux, prec):
    """By 2^70: p rho grows by 2^140, beyond FP32's 2^128.  Everything moves, so
    that no momentum falls off to where FP32 flushes to zero, 2^-126 unscaled
    and 2^-196 scaled, and the Euler values are the scaled bits.  A material's
    partial density does fall off: what is flushed there is below 2^-126 an
    operation, and 2^-110 allows for 30 steps of them.  The fast form snaps
    partial densities below 1e-12, which a scale changes: Euler only."""
    cfg = G.case_config(model, case, 75, 62, flux)
    cfg.precision, cfg.limiter, cfg.fix_dy_halfstep, cfg.cfl = prec, limiter, 1, 0.5
    for k in range(4):
        cfg.bc[k] = 0
    ic = G.case_ic(cfg, case)
    g = cfg.ghosts
    inner, im = ic[g:-g, g:-g], 1 if model == G.EULER else 2
    rho = inner[..., 0] if model == G.EULER else inner[..., 0] + inner[..., 1]
    e = inner[..., im + 2] - 0.5 * (inner[..., im] ** 2 + inner[..., im + 1] ** 2) / rho
    speed = np.sqrt(e / rho).mean()
    inner[..., im] += 0.21 * speed * rho
    inner[..., im + 1] += 0.17 * speed * rho
    inner[..., im + 2] = e + 0.5 * (inner[..., im] ** 2 + inner[..., im + 1] ** 2) / rho
    scale = np.full(ic.shape[-1], 2.0**70)
    if model == G.ALLAIRE:
        scale[5] = 1.0  # the volume fraction

    def run(x):
        with G.Batch() as b:
            m = b.add(cfg, x, max_steps=STEPS)
            b.step(STEPS)
            return b.download(m)[g:-g, g:-g], b.status(m)

    want, st = run(ic)
    got, st2 = run(ic * scale)
    assert st.n == st2.n == STEPS and np.isfinite(want).all()
    assert (st.t, st.maxu, st.maxv) == (st2.t, st2.maxu, st2.maxv)
    assert np.abs(got / scale - want).max() <= (0.0 if model == G.EULER else 2.0**-110)


@pytest.mark.parametrize("rho,p,prec", [(1e-9, 0.0, G.MIXED), (1.0, 0.0, G.MIXED),
                                        (1e-9, 1e-20, G.MIXED), (1e-11, 1e-29, G.MIXED),
                                        (1e-9, 1e-20, G.FP64_FAST), (1e-11, 1e-29, G.FP64_FAST)])
def test_thin_cold_gas_has_finite_speeds(rho, p, prec):
    """p rho is below FP32's least normal number, or 0.  (Where p is 0 the
    forms in FP64 have S_L = S_R = 0 and a flux of 0/0, as the reference.)"""
    cfg = G.case_config(G.EULER, "cross", 40, 36)
    cfg.precision, cfg.fix_dy_halfstep, cfg.cfl = prec, 1, 0.5
    for k in range(4):
        cfg.bc[k] = 0
    ic = G.case_ic(cfg, "cross")
    g = cfg.ghosts
    # a gas of sound speed c beside a thin one at rest
    ic[g:-g, g:-g] = [1.0, 0.3, 0.0, 1.0 / (cfg.gamma1 - 1) + 0.045]
    ic[g:g + 18, g:-g] = [rho, 0.0, 0.0, p / (cfg.gamma1 - 1)]
    c = np.sqrt(cfg.gamma1)
    with G.Batch() as b:
        m = b.add(cfg, ic, max_steps=3)
        b.step(1)
        st = b.status(m)
        assert np.isfinite(b.download(m)[g:-g, g:-g]).all()
    assert 0 < st.t and np.isfinite([st.t, st.dt_next, st.maxu, st.maxv]).all()
    # nothing is faster than the gas expanding into a vacuum, 2 c/(gamma - 1), and c
    assert max(st.maxu, st.maxv) <= 0.3 + 2 * c / (cfg.gamma1 - 1) + c
