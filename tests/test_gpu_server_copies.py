"""Grids the server copies in parts on several threads (from 4 MiB on) arrive
and return whole, also when two threads wait for one request."""
import threading

import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [0, 256 << 20], ids=["pageable", "pinned"])
@pytest.mark.parametrize("nx,ny", [(358, 358), (508, 254), (509, 254), (1021, 517), (2043, 1025)])
def test_served_grid_equals_batch(nx, ny, pinned):
    cfg = G.recipe_config("shock_bubbles", nx, ny)
    ic = G.recipe_ic(cfg, "shock_bubbles", nbubbles=6)
    with G.Batch() as b:
        m = b.add(cfg, ic, 3)
        b.step(3)
        want = b.download(m)
    outs = [np.zeros_like(want), np.zeros_like(want)]
    with G.Server(host_pinned_bytes=pinned) as s:
        rid = s.submit(cfg, ic, 3)
        ts = [threading.Thread(target=s.wait, args=(rid,), kwargs={"out": o}) for o in outs]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        s.release(rid)
    for o in outs:
        assert np.array_equal(o, want)
