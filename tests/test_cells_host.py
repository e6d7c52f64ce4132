"""Index arithmetic of the cell gathers, run on the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def reach(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    exe = tmp_path_factory.mktemp("cells") / "cells_reach"
    subprocess.run([nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-I{ROOT / 'wake_b200' / 'csrc'}", f"-I{ROOT / 'include'}", str(ROOT / "tests" / "cells_reach.cu"),
                    "-o", str(exe)], check=True)
    return exe


# Node counts that are a multiple of the plane's padding (64), where the last plane ends with its last node, rows
# longer and shorter than a cell, and rows of which a cell ends one node before or after the end.
@pytest.mark.parametrize("q,nx,ny,nz", [(9, 72, 64, 1), (9, 80, 64, 1), (9, 65, 64, 1), (9, 64, 16, 1), (9, 66, 33, 1),
                                        (9, 300, 16, 1), (19, 80, 16, 12), (19, 81, 15, 13), (27, 80, 13, 12),
                                        (27, 72, 8, 8)])
def test_inside_cells_read_their_plane_only(reach, q, nx, ny, nz):
    r = subprocess.run([str(reach), str(q), str(nx), str(ny), str(nz)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
