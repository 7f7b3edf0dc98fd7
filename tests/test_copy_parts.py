"""The parts of a cut copy cover every byte once, for sizes whose quotient is a
multiple of the step with a remainder too."""
import shutil
import subprocess

import pytest

from cfdtest import ROOT

CXX = shutil.which("g++")

PROGRAM = r"""
#include "cfd_copy.h"
#include <cstdio>
int main() {
    int bad = 0;
    for (size_t parts = 1; parts <= 16; ++parts)
        for (size_t pages = 0; pages <= 9; ++pages)
            for (long off = -17; off <= 17; ++off) {
                const long total = (long)(parts * pages * 4096) + off;
                if (total < 0) continue;
                const size_t bytes = (size_t)total;
                size_t at = 0;
                for (size_t k = 0; k < parts; ++k) {
                    const cfd::CopyPart p = cfd::copy_part(bytes, parts, k);
                    bad += p.lo != at || p.n > bytes - p.lo;
                    at = p.lo + p.n;
                }
                bad += at != bytes;
            }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(CXX is None, reason="no g++")
def test_parts_cover_every_byte_once(tmp_path):
    src, exe = tmp_path / "parts.cpp", tmp_path / "parts"
    src.write_text(PROGRAM)
    subprocess.run([CXX, "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'cfd-art_b200' / 'csrc'}", str(src),
                    "-o", str(exe)], check=True, timeout=120)
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout == "0\n"
