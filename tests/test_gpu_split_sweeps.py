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


@pytest.mark.parametrize("prec", [G.MIXED, G.FP64_FAST], ids=["mixed", "fast"])
def test_replayed_ticks_equal_ticks_launched_one_by_one(prec):
    """31 ticks are launched one by one, 32 and more in one call replay a
    graph, and so do later calls of 8; the states are the same."""
    cfg = G.recipe_config("shock_bubbles", 40, 33)
    cfg.precision = prec
    states = []
    for calls in [(31, 33), (1,) * 64, (64,), (7,) * 8 + (8,), (40, 8, 8, 8)]:
        with G.Batch() as b:
            m = b.add_recipe(cfg, "shock_bubbles", max_steps=64)
            for ticks in calls:
                b.step(ticks)
            st = b.status(m)
            states.append((st.n, st.t, st.mass1, b.download(m).tobytes()))
    assert states[0][0] == 64 and all(s == states[0] for s in states)


@pytest.mark.parametrize("ticks", [(1, 2, 17), (70,)], ids=["launched", "replayed"])
@pytest.mark.parametrize("sizes", [[(40, 33)] * 4, [(300, 200), (5, 3), (1024, 700), (64, 64)]],
                         ids=["small", "uneven"])
def test_models_and_forms_side_by_side_equal_each_alone(sizes, ticks):
    """Chains of launches of different models and forms run at the same time."""
    members = []
    for (nx, ny), (recipe, prec) in zip(sizes, [("shock_bubbles", G.MIXED),
                                                ("water_shock_air_bubble", G.FP64_FAST),
                                                ("water_shock_air_bubble", G.MIXED),
                                                ("shock_bubbles", G.FP64_FAST)]):
        cfg = G.recipe_config(recipe, nx, ny)
        cfg.precision = prec
        members.append((cfg, recipe))

    def solve(some):
        with G.Batch() as b:
            ids = [b.add_recipe(c, r, max_steps=sum(ticks) - 3 * k)
                   for k, (c, r) in some]
            for n in ticks:
                b.step(n)
            out = []
            for i in ids:
                st = b.status(i)
                out.append((st.n, st.t, st.mass1, st.maxu, st.maxv, b.download(i).tobytes()))
            return out

    numbered = list(enumerate(members))
    together = solve(numbered)
    for k, m in numbered:
        assert together[k][0] == sum(ticks) - 3 * k
        assert together[k] == solve([(k, m[:2])])[0]


@pytest.mark.parametrize("ticks", [(5, 12), (40,)], ids=["launched", "replayed"])
@pytest.mark.parametrize("recipe,prec", [("shock_bubbles", G.MIXED), ("shock_bubbles", G.FP64_FAST),
                                         ("water_shock_air_bubble", G.FP64_FAST)])
def test_strands_of_one_form_equal_each_member_alone(recipe, prec, ticks):
    """7.7e5 cells in all step in three strands, one member finishing early."""
    members = []
    for k, (nx, ny) in enumerate([(64, 64), (700, 500), (300, 411), (512, 512), (129, 257)]):
        cfg = G.recipe_config(recipe, nx, ny)
        cfg.precision = prec
        members.append((cfg, sum(ticks) - 9 * (k == 2)))

    def solve(some):
        with G.Batch() as b:
            ids = [b.add_recipe(c, recipe, max_steps=n) for c, n in some]
            for n in ticks:
                b.step(n)
            return [(b.status(i), b.download(i)) for i in ids]

    for (st, grid), m in zip(solve(members), members):
        st1, alone = solve([m])[0]
        assert st.n == st1.n == m[1]
        assert (st.t, st.maxu, st.maxv) == (st1.t, st1.maxu, st1.maxv)
        assert np.array_equal(grid, alone)
        assert abs(st.mass1 - st1.mass1) <= 1e-12 * abs(st1.mass1)


@pytest.mark.parametrize("prec", [G.MIXED, G.FP64_FAST], ids=["mixed", "fast"])
@pytest.mark.parametrize("recipe", ["shock_bubbles", "water_shock_air_bubble"])
def test_many_x_tiles_of_twenty_rows(recipe, prec):
    """Beside a grid of many tiles a small one's segments have 20 rows, alone
    others; its bits are the same."""
    small = G.recipe_config(recipe, 333, 217)
    large = G.recipe_config(recipe, 2400, 2400)
    small.precision = large.precision = prec
    states, rows = [], []
    for beside in (False, True):
        with G.Batch() as b:
            m = b.add_recipe(small, recipe, max_steps=4)
            if beside:
                b.add_recipe(large, recipe, max_steps=4)
            b.step(4)
            st = b.status(m)
            states.append((st.n, st.t, st.maxu, st.maxv, b.download(m).tobytes()))
        with G.Batch() as b:
            b.add_recipe(small, recipe, max_steps=4)
            if beside:
                b.add_recipe(large, recipe, max_steps=4)
            rows.append(b.segment_rows(small.model, prec))
    assert rows[1] == 20 and rows[0] != 20
    assert states[0] == states[1]
