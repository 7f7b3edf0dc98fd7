"""Shared test setup: the `gpu` marker, import paths, fixture loaders."""
import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
for p in (ROOT / "oracle", ROOT / "cfd-art_b200", ROOT / "tests"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))

# A `reference` directory that holds no sources is no reference checkout.
if not (ROOT.parent / "reference" / "euler_equations").is_dir():
    os.environ.setdefault("CFD_REFERENCE_DIR", str(ROOT.parent / "reference" / "absent"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
