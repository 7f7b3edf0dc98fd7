"""Solvers and batches of several threads, whose sweeps are launched for the
first time at once (in a process of their own), give the results they give one
after the other."""
import subprocess
import sys

import pytest

from cfdtest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys, threading
sys.path.insert(0, sys.argv[1])
import cfdgpu as G
jobs = [(r, p) for r in ("shock_bubbles", "water_shock_air_bubble")
        for p in (G.FP64, G.MIXED, G.FP64_FAST)] * 2
def solve(recipe, prec):
    cfg = G.recipe_config(recipe, 150, 90)
    if prec == G.FP64:
        with G.Solver(cfg) as s:
            s.upload_recipe(recipe, nbubbles=4)
            s.advance(12)
            return s.download().tobytes()
    cfg.precision = prec
    with G.Batch() as b:
        m = b.add_recipe(cfg, recipe, max_steps=12)
        b.step(12)
        return b.download(m).tobytes()
got = [None] * len(jobs)
start = threading.Barrier(len(jobs))
def run(k):
    start.wait()
    got[k] = solve(*jobs[k])
ts = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
for t in ts: t.start()
for t in ts: t.join()
assert all(got) and got == [solve(*j) for j in jobs]
print("same")
"""


def test_first_launches_of_several_threads():
    out = subprocess.run([sys.executable, "-c", SCRIPT, str(ROOT / "cfd-art_b200")], capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
