"""Every way of handing a solver its state gives the same state, wave speeds and
masses, bit for bit: a ghosted host grid, host planes, device planes read in
place, and device planes that have to be copied (off an 8-byte boundary)."""
import numpy as np
import pytest

import cfdgpu as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ghosts", [False, True], ids=["plain", "frame"])
@pytest.mark.parametrize("recipe", ["shock_bubbles", "water_shock_air_bubble"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (2, 7), (31, 5), (64, 64), (257, 129), (700, 433),
                                   (2, 4000), (4000, 3)])
def test_uploads_agree(nx, ny, recipe, ghosts):
    cfg = G.recipe_config(recipe, nx, ny)
    ic = G.recipe_ic(cfg, recipe, nbubbles=4)
    g = cfg.ghosts
    planes = np.ascontiguousarray(ic[g:-g, g:-g].transpose(2, 0, 1))
    dev = torch.from_numpy(planes).cuda()
    shifted = torch.empty(planes.nbytes + 12, dtype=torch.uint8, device="cuda")
    by4, by8 = shifted[4:-8], shifted[8:-4]
    torch.cuda.synchronize()

    def state(put):
        with G.Solver(cfg) as s:
            if ghosts:
                s.set_reference_ghosts(True)
            put(s)
            st0 = s.status()
            s.advance(2)
            st = s.status()
            return ([getattr(x, f) for x in (st0, st) for f in ("n", "t", "dt_next", "maxu", "maxv",
                                                                "mass1", "mass2")],
                    s.download().tobytes())

    by4.copy_(dev.flatten().view(torch.uint8))
    torch.cuda.synchronize()
    want = state(lambda s: s.upload_device(by4.data_ptr()))
    assert np.isfinite(want[0]).all()
    assert state(lambda s: s.upload_device(dev.data_ptr())) == want
    by8.copy_(dev.flatten().view(torch.uint8))
    torch.cuda.synchronize()
    assert state(lambda s: s.upload_device(by8.data_ptr())) == want
    assert state(lambda s: s.upload(planes, layout=G.SOA)) == want
    if not ghosts:  # with a frame the grid's own ghost cells are kept
        assert state(lambda s: s.upload(ic)) == want
