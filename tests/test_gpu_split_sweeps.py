"""Divided tiles and the two ways a step is closed: a small grid alone runs its
tiles divided among warps and is closed by its last warp or, with many
reduction slots, by a kernel of its own; beside a large member that fills the
device it runs undivided.  The member's bits and times are the same."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [G.MIXED, G.FP64_FAST], ids=["mixed", "fast"])
@pytest.mark.parametrize("recipe", ["shock_bubbles", "water_shock_air_bubble"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (5, 3), (64, 64), (31, 17), (33, 15), (300, 200), (700, 20)])
def test_divided_small_grid_equals_undivided(prec, recipe, nx, ny):
    cfg = G.recipe_config(recipe, nx, ny)
    cfg.precision, cfg.fix_dy_halfstep = prec, 1
    ic = G.recipe_ic(cfg, recipe, nbubbles=6)
    with G.Batch() as b:
        m = b.add(cfg, ic, 30)
        b.step(30)
        alone, st = b.download(m), b.status(m)
    big = G.recipe_config(recipe, 2048, 1024)
    big.precision = prec
    with G.Batch() as b:
        b.add_recipe(big, recipe, max_steps=30)
        m = b.add(cfg, ic, 30)
        b.step(30)
        mixed, st2 = b.download(m), b.status(m)
    assert np.isfinite(alone).all()
    assert st.n == st2.n == 30 and st.t == st2.t and st.maxu == st2.maxu and st.maxv == st2.maxv
    assert np.array_equal(alone, mixed)
    # the mass sums are grouped by strip: equal to the rounding of their sums
    assert abs(st.mass1 - st2.mass1) <= 1e-12 * abs(st.mass1)
