"""An upload that is refused leaves the solver as it was.  The planes handed over
are larger than the allocation they lie in, which the driver's copies refuse.
(The next allocation follows it directly, so the memory past its end exists.)"""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import cfdgpu as G
from cfdtest import ROOT

pytestmark = pytest.mark.gpu

FIELDS = ("n", "t", "dt_next", "maxu", "maxv", "mass1", "mass2")


def _adjacent(driver, size):
    """Device allocations of `size` bytes, and one of them whose end another begins at."""
    got = []
    for _ in range(16):
        p = ctypes.c_uint64()
        assert driver.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        got.append(p.value)
    return got, next((p for p in got if p + size in got), None)


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("offset", [4, 0], ids=["copied", "aligned"])
def test_refused_upload_changes_nothing(offset, steps):
    cfg = G.recipe_config("shock_bubbles", 64, 64)
    cfg.splitting = 1  # an odd number of sweeps a step: the current buffer alternates
    ic = G.recipe_ic(cfg, "shock_bubbles", nbubbles=4)
    driver = ctypes.CDLL("libcuda.so.1")
    with G.Solver(cfg) as s, G.Solver(cfg) as untouched:
        for x in (s, untouched):
            x.upload(ic)
            x.advance(steps)
        before = [getattr(s.status(), f) for f in FIELDS]
        state = s.download()
        size = 64 * 64 * 8 * 3 // 2  # a plane and a half of four
        all_, small = _adjacent(driver, size)
        try:
            if small is None:
                pytest.skip("no two adjacent allocations")
            with pytest.raises(G.CfdError):
                s.upload_device(small + offset, n=70, t=0.5)
        finally:
            for p in all_:
                driver.cuMemFree_v2(ctypes.c_uint64(p))
        assert [getattr(s.status(), f) for f in FIELDS] == before
        if steps % 2:  # the copy goes to the other buffer then, as far as it got
            assert np.array_equal(s.download(), state)
            s.advance(3)
            untouched.advance(3)
            assert np.array_equal(s.download(), untouched.download())


SEGMENTS = r"""
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
import cfdgpu as G
cfg = G.recipe_config("shock_bubbles", 1500, 1100)
ic = G.recipe_ic(cfg, "shock_bubbles", nbubbles=4)
planes = np.ascontiguousarray(ic[2:-2, 2:-2].transpose(2, 0, 1))
dev = torch.from_numpy(planes).cuda()
torch.cuda.synchronize()
out = []
for put in (lambda s: s.upload_device(dev.data_ptr()), lambda s: s.upload(planes, layout=G.SOA)):
    with G.Solver(cfg) as s:
        put(s)
        s.advance(2)
        out.append(s.download().tobytes())
assert out[0] == out[1]
print("same")
"""


def test_planes_in_mapped_pieces():
    """53 MB of an allocator that maps its memory in pieces."""
    pytest.importorskip("torch")
    env = dict(os.environ, PYTORCH_CUDA_ALLOC_CONF="expandable_segments:True")
    out = subprocess.run([sys.executable, "-c", SEGMENTS, str(ROOT / "cfd-art_b200")], capture_output=True,
                         text=True, timeout=300, env=env)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
