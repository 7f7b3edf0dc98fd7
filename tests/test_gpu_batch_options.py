"""Launches compiled for one set of options against the general one: a member
alone in a batch runs the instantiation of its own options, beside a member of
other options the general one, and its result must be the same bits."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu



def _member(precision, model, case, nx, ny, over):
    if case in G.RECIPE:
        cfg = G.recipe_config(case, nx, ny)
        ic = None
    else:
        cfg = G.case_config(model, case, nx, ny)
        ic = True
    cfg.precision, cfg.cfl = precision, 0.6
    for k, v in over.items():
        setattr(cfg, k, v)
    ic = G.case_ic(cfg, case) if ic else G.recipe_ic(cfg, case, nbubbles=6)
    return cfg, ic


CASES = [
    ("euler minmod", G.EULER, "shock_bubbles", {"limiter": 0}, {"limiter": 2}),
    ("euler van Leer", G.EULER, "shock_bubbles", {"limiter": 1}, {"limiter": 0}),
    ("euler MC", G.EULER, "shock_bubbles", {"limiter": 2}, {"limiter": 1}),
    ("euler unlimited", G.EULER, "four_quadrant", {"limiter": 3}, {"limiter": 1}),
    ("euler first order", G.EULER, "shock_bubbles", {"flux_solver": 1, "limiter": 1}, {"limiter": 2}),
    ("allaire stiff PVRS", G.ALLAIRE, "water_shock_air_bubble", {"limiter": 0}, {"limiter": 1}),
    ("allaire gas", G.ALLAIRE, "shocked_helium_bubble", {"limiter": 0}, {"limiter": 1}),
]


@pytest.mark.parametrize("name,model,case,over,other", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("precision", [G.MIXED, G.FP64_FAST], ids=["mixed", "fast"])
@pytest.mark.parametrize("nx,ny", [(61, 17), (28, 70), (200, 131)])
def test_options_compiled_in_equal_the_general_launch(precision, name, model, case, over, other, nx, ny):
    cfg, ic = _member(precision, model, case, nx, ny, over)
    with G.Batch() as b:
        m = b.add(cfg, ic, 40)
        b.step(40)
        alone = b.download(m)
        st = b.status(m)
    cfg2, ic2 = _member(precision, model, case, 45, 38, other)
    with G.Batch() as b:
        m = b.add(cfg, ic, 40)
        b.add(cfg2, ic2, 40)
        b.step(40)
        mixed = b.download(m)
        st2 = b.status(m)
    assert np.isfinite(alone).all()
    assert st.n == st2.n == 40 and st.t == st2.t
    assert np.array_equal(alone, mixed)
