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
