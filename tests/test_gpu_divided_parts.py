"""Strips divided among warps so that some parts have no rows (a last strip no
longer than its first part, rows that do not divide evenly): such a part copies
no rows, so whichever part its warp takes next finds its staging slots free.
The member's bits are those of other strip lengths and of a batch of its own
copies, whose strips are divided otherwise or not at all."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu

STEPS = 24


def _run(cfg, recipe, copies=1, rows=0):
    with G.Batch() as b:
        ids = [b.add_recipe(cfg, recipe, max_steps=STEPS) for _ in range(copies)]
        if rows:
            b.set_march_rows(cfg.model, rows)
        b.step(STEPS)
        out = []
        for i in (ids[0], ids[-1]):
            st = b.status(i)
            out.append((st.n, st.t, st.maxu, st.maxv, b.download(i).tobytes()))
        return out


@pytest.mark.parametrize("recipe,prec", [("water_shock_air_bubble", G.FP64_FAST),
                                         ("water_shock_air_bubble", G.MIXED),
                                         ("shock_bubbles", G.FP64_FAST), ("shock_bubbles", G.MIXED)])
@pytest.mark.parametrize("nx,ny", [(700, 500), (640, 612), (900, 900), (64, 65), (200, 49)])
def test_parts_without_rows(recipe, prec, nx, ny):
    cfg = G.recipe_config(recipe, nx, ny)
    cfg.precision = prec
    want = _run(cfg, recipe)[0]
    assert want[0] == STEPS and np.isfinite(np.frombuffer(want[-1])).all()
    assert _run(cfg, recipe, copies=6) == [want, want]
    for rows in (16, 20, 33, 64):
        assert _run(cfg, recipe, rows=rows)[0] == want


@pytest.mark.parametrize("rows", [0, 16, 20, 36, 64])
@pytest.mark.parametrize("recipe,prec", [("water_shock_air_bubble", G.FP64_FAST),
                                         ("water_shock_air_bubble", G.MIXED),
                                         ("shock_bubbles", G.FP64_FAST), ("shock_bubbles", G.MIXED)])
def test_parts_fit_on_the_device(recipe, prec, rows):
    """A divided y sweep has no more parts than warps that fit at once: 8 per
    SM for the two-material fast FP64 sweep, 16 for the others."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    model = G.recipe_config(recipe, 64, 64).model
    fit = (8 if (model, prec) == (G.ALLAIRE, G.FP64_FAST) else 16) * sms
    for nx, ny in [(64, 64), (300, 200), (512, 512), (640, 612), (700, 500), (900, 900), (1024, 512),
                   (1536, 768), (2048, 1024)]:
        cfg = G.recipe_config(recipe, nx, ny)
        cfg.precision = prec
        with G.Batch() as b:
            b.add_recipe(cfg, recipe, max_steps=1)
            b.set_march_rows(model, rows)
            _, y = b.split(model, prec)
            if rows:
                parts = (nx + 31) // 32 * -(-ny // rows) * y
                assert y == 1 or parts <= fit, (nx, ny, y)
            elif fit == 8 * sms and nx >= 640:  # its strips fill the device by themselves
                assert y == 1, (nx, ny, y)
            if nx == 64:
                assert y > 1


@pytest.mark.parametrize("recipe,prec", [("water_shock_air_bubble", G.FP64_FAST),
                                         ("water_shock_air_bubble", G.MIXED),
                                         ("shock_bubbles", G.FP64_FAST), ("shock_bubbles", G.MIXED)])
@pytest.mark.parametrize("nx,ny", [(5, 3), (64, 64), (31, 17), (300, 200), (700, 20)])
def test_divided_member_equals_undivided(recipe, prec, nx, ny):
    """Alone a small member's tiles are divided; among enough others of its
    form, which fill the warps, they are not.  64x64 is closed by its last
    warp then, and by a kernel of its own alone (32 slots and fewer, more)."""
    cfg = G.recipe_config(recipe, nx, ny)
    filler = G.recipe_config(recipe, 64, 64)
    cfg.precision = filler.precision = prec
    want = None
    for fillers in (0, 165):
        with G.Batch() as b:
            m = b.add_recipe(cfg, recipe, max_steps=STEPS)
            for _ in range(fillers):
                b.add_recipe(filler, recipe, max_steps=STEPS)
            b.set_march_rows(cfg.model, 16)
            x, y = b.split(cfg.model, prec)
            if fillers:
                assert (x, y) == (1, 1)
            else:
                assert x > 1 and y > 1
                if (nx, ny) == (64, 64):
                    assert 8 <= 32 < 8 * y
            b.step(STEPS)
            st = b.status(m)
            got = (st.n, st.t, st.maxu, st.maxv, b.download(m).tobytes())
        want = want or got
        assert got == want
    assert want[0] == STEPS and np.isfinite(np.frombuffer(want[-1])).all()
