"""The plain FP64 form where its shared-reciprocal arithmetic and its segment
tiling can go wrong, against the CPU oracle, bit for bit (equal values; only
the sign of an exact zero may differ)."""
import numpy as np
import pytest

import cfdgpu as G
import oracle_py as O
from cfdtest import params_from_config

pytestmark = pytest.mark.gpu


def _states(model, rng, n):
    """Stencils whose divisors and numerators sit at the edges of the method:
    mantissas of all ones or a few below (densities just under a power of two,
    and products (gamma - 1) rho there), momenta that are zero, denormal or
    below its range, and pressures that cancel."""
    ulps = rng.integers(0, 20, (n, 4))
    base = rng.choice([1.0, 2.0, 0.5, 2.5, 5.0, 1.5], (n, 4))
    rho = base - ulps * np.spacing(base / 2)
    tiny = rng.choice([0.0, -0.0, 5e-324, -3e-320, 1e-310, 2.5e-308, 1e-300, -1e-265, 1e-150, 0.3],
                      (n, 4))
    tinv = rng.choice([0.0, 1e-312, -1e-290, 1e-262, 0.7], (n, 4))
    p = rng.choice([1.0, 1.0 - 2.0**-53, 0.029, 1e-3], (n, 4)) * rng.choice([1.0, 1.0 + 2.0**-40], (n, 4))
    if model == "euler":
        E = p / (1.4 - 1.0) + 0.5 * rho * (tiny * tiny + tinv * tinv)
        return np.stack([rho, rho * tiny, rho * tinv, E], -1)
    z = rng.choice([0.0, 1.0, 1e-6, 1.0 - 1e-6, 0.5, 1e-13, 0.3], (n, 4))
    p = p * 1e5
    eps = z / 3.4 + (1 - z) / 0.4
    kn = z * 4.4 * 6e8 / 3.4
    r1, r2 = z * 1000.0 * rho, (1 - z) * rho
    R = r1 + r2
    return np.stack([r1, r2, R * tiny, R * tinv,
                     p * eps + kn + 0.5 * R * (tiny * tiny + tinv * tinv), z], -1)


@pytest.mark.parametrize("model,flux,limiter,ws", [
    ("euler", "MUSCL", "minmod", "davis"), ("euler", "MUSCL", "vanleer", "davis"),
    ("euler", "Godunov", "minmod", "davis"), ("allaire", "MUSCL", "minmod", "pvrs"),
    ("allaire", "MUSCL", "vanleer", "davis"), ("allaire", "Godunov", "minmod", "pvrs")])
def test_faces_at_the_edges_of_the_shared_reciprocals(model, flux, limiter, ws):
    rng = np.random.default_rng(77)
    n = 3000
    st = _states(model, rng, n)
    if flux == "Godunov":
        st = st[:, :2].copy()
    name = "four_quadrant" if model == "euler" else "water_shock_air_bubble"
    cfg = G.recipe_config(name, 8, 8)
    cfg.flux_solver, cfg.limiter, cfg.wavespeed = G.FLUX[flux], G.LIMITERS[limiter], G.WAVESPEED[ws]
    p, _ = params_from_config(cfg)
    dt, dx = (2e-3, 1e-2) if model == "euler" else (2e-7, 1e-2)
    got, us, zs = G.face_flux(cfg, st, dt, dx)
    for f in range(n):
        rf, ru, rz = O.port_face_flux(model, p, st[f], dt, dx)
        assert np.array_equal(got[f], rf, equal_nan=True), (f, st[f].tolist(), got[f], rf)
        assert us[f] == ru or (np.isnan(ru) and np.isnan(us[f]))
        if model == "allaire" and not np.isnan(rz):
            assert zs[f] == rz


@pytest.mark.parametrize("nx,ny", [(27, 9), (28, 8), (29, 7), (30, 10), (31, 16), (57, 28),
                                   (3, 29), (8, 57), (112, 5), (113, 33)])
@pytest.mark.parametrize("strang", [0, 1])
def test_segment_edges_match_oracle(nx, ny, strang):
    """Grids one cell around the multiples of a segment's 28 outputs and of a
    tile's 4 rows or 8 columns, walls on two sides, both splittings (the
    reduction rides on the y sweep or on the last x sweep)."""
    cfg = G.case_config(G.EULER, "circular_explosion", nx, ny)
    cfg.splitting, cfg.cfl = strang, 0.7
    cfg.bc[1] = G.REFLECTIVE  # right
    cfg.bc[2] = G.REFLECTIVE             # bottom
    ic = G.case_ic(cfg, "circular_explosion")
    p, model = params_from_config(cfg)
    ref = ic.copy()
    taken, n, t, _ = O.port_run(model, p, ref, 25)
    with G.Solver(cfg) as s:
        s.upload(ic)
        s.advance(25)
        st = s.status()
        out = s.download()
    assert (st.n, st.t) == (n, t)
    assert np.array_equal(out[2:-2, 2:-2], ref[2:-2, 2:-2])


@pytest.mark.parametrize("strang", [0, 1])
@pytest.mark.parametrize("ws", ["davis", "pvrs"])
@pytest.mark.parametrize("limiter", ["minmod", "vanleer", "mc", "unlimited"])
@pytest.mark.parametrize("case", ["shocked_helium_bubble", "underwater_explosion_modified"])
def test_two_material_options_match_oracle(case, limiter, ws, strang):
    """The sweeps compiled for a limiter and a wave-speed estimate, and the
    general ones."""
    cfg = G.case_config(G.ALLAIRE, case, 45, 31)
    cfg.limiter, cfg.wavespeed, cfg.splitting = G.LIMITERS[limiter], G.WAVESPEED[ws], strang
    ic = G.case_ic(cfg, case)
    p, model = params_from_config(cfg)
    ref = ic.copy()
    taken, n, t, _ = O.port_run(model, p, ref, 12)
    with G.Solver(cfg) as s:
        s.upload(ic)
        s.advance(12)
        st = s.status()
        out = s.download()
    assert (st.n, st.t) == (n, t)
    assert np.array_equal(out[2:-2, 2:-2], ref[2:-2, 2:-2], equal_nan=True)
