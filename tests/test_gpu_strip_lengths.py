"""A member's bits do not depend on the strip length of the marching y sweep
(which its company in the batch sets), for odd lengths too, nor on whether the
launch is compiled for its options: every limiter and flux, walls and open
sides, gas and stiffened gas, both wave-speed estimates, both forms."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu

MATERIALS = [("gas", G.EULER, "cross", {}), ("stiffened gas", G.EULER, "cross", {"pinf1": 0.3}),
             ("two gases", G.ALLAIRE, "shocked_helium_bubble", {}),
             ("water and gas", G.ALLAIRE, "underwater_explosion_modified", {}),
             ("water and gas PVRS", G.ALLAIRE, "underwater_explosion_modified", {"wavespeed": 1})]


@pytest.mark.parametrize("prec", [G.MIXED, G.FP64_FAST], ids=["mixed", "fast"])
@pytest.mark.parametrize("flux", ["MUSCL", "Godunov"])
@pytest.mark.parametrize("limiter", range(4), ids=["minmod", "vanleer", "mc", "unlimited"])
@pytest.mark.parametrize("wall", [0, 1], ids=["open", "walls"])
@pytest.mark.parametrize("name,model,case,over", MATERIALS, ids=[m[0] for m in MATERIALS])
def test_bits_do_not_depend_on_strip_lengths(name, model, case, over, wall, limiter, flux, prec):
    def config(nx, ny, lim):
        cfg = G.case_config(model, case, nx, ny, flux)
        cfg.precision, cfg.limiter, cfg.fix_dy_halfstep, cfg.cfl = prec, lim, 1, 0.5
        for k in range(4):
            cfg.bc[k] = wall
        for k, v in over.items():
            setattr(cfg, k, v)
        return cfg, G.case_ic(cfg, case)

    cfg, ic = config(131, 97, limiter)
    other, other_ic = config(40, 30, (limiter + 1) % 3)
    want = None
    for company in (False, True):
        for rows in (16, 17, 20, 33, 64):
            with G.Batch() as b:
                m = b.add(cfg, ic, max_steps=12)
                if company:
                    b.add(other, other_ic, max_steps=12)
                b.set_march_rows(model, rows)
                b.step(12)
                st = b.status(m)
                got = (repr((st.n, st.t, st.dt_next, st.maxu, st.maxv)), b.download(m).tobytes())
            want = want or got
            assert got == want, (company, rows)
