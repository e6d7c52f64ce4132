"""Arithmetic of the step kernels that runs on the host too: the cells' indexes, the division of the Zou-He faces,
the stress behind the packed BGK kernel's Smagorinsky tau."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def _compile(source, folder):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    exe = folder / source
    subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-I{ROOT / 'wake_b200' / 'csrc'}", f"-I{ROOT / 'include'}", str(ROOT / "tests" / f"{source}.cu"),
                    "-o", str(exe)], check=True)
    return exe


@pytest.fixture(scope="module")
def reach(tmp_path_factory):
    return _compile("cells_reach", tmp_path_factory.mktemp("cells"))


# Node counts that are a multiple of the plane's padding (64), where the last plane ends with its last node, rows
# longer and shorter than a cell, and rows of which a cell ends one node before or after the end.
@pytest.mark.parametrize("q,nx,ny,nz", [(9, 72, 64, 1), (9, 80, 64, 1), (9, 65, 64, 1), (9, 64, 16, 1), (9, 66, 33, 1),
                                        (9, 300, 16, 1), (19, 80, 16, 12), (19, 81, 15, 13), (27, 80, 13, 12),
                                        (27, 72, 8, 8)])
def test_inside_cells_read_their_plane_only(reach, q, nx, ny, nz):
    r = subprocess.run([str(reach), str(q), str(nx), str(ny), str(nz)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def test_division_by_a_constant(tmp_path):
    """By 3 and 6 over every 251st float (every 7th of the smallest), the zeros, the largest, infinity and NaN."""
    r = subprocess.run([str(_compile("by_const", tmp_path))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def test_stress_of_the_packed_bgk_kernel(tmp_path):
    """Its error against FP64 is no larger than the one-node kernels' on the same nodes."""
    r = subprocess.run([str(_compile("bgk_stress", tmp_path))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
