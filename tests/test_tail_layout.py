"""The layout of the fused stage tail's tile lists, compiled for the host: what a block's threads load
ahead of knowing the tile stays inside the tile's own lists."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "afar_cudaeuler2dmixo3rk3solver_gb300", "csrc")


def _run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include "afar_tail_layout.h"\nusing namespace afar;\nint main() {\n' + body + "}\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("cells", [1, 95, 96, 97, 127, 128, 129, 152, 192])
def test_halo_entries_loaded_ahead_are_the_tiles_own(tmp_path, cells):
    got = _run(tmp_path, 'std::printf("%%d\\n", kTailHalo);\n'
               'for (int t = %d; t < kTailThreads; ++t) std::printf("%%d\\n", tail_first_halo(t, %d));\n' % (cells, cells))
    halo, first = int(got[0]), [int(x) for x in got[1:]]
    assert len(first) == 256 - cells
    assert all(0 <= h < halo for h in first)
    # the entries that a tile can have are each their own thread's
    assert first[:halo] == list(range(min(halo, len(first))))
