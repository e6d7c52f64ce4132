"""The device memory of a lattice against its estimate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wb = pytest.importorskip("wake_b200")


@pytest.mark.parametrize("q,nx,ny,nz,storage", [(9, 64, 60000, 1, "f16"), (19, 64, 192, 192, "f16"),
                                                (19, 65, 192, 192, "f32")])
def test_estimate_covers_a_lattice_of_obstacles(q, nx, ny, nz, storage):
    """Every segment general: a record per node, lists and force slots for every cell."""
    types = np.zeros((nz, ny, nx), np.uint8)
    types[:, 1::3, 1::4] = wb.SOLID
    wb.lib.wake_gpu_cache_trim()
    g = wb.LatticeGrid2D(nx, ny, 0.6, storage=storage) if q == 9 else wb.LatticeGrid3D(nx, ny, nz, 0.6, storage=storage)
    g.set_cell_types(types)
    g.enable_forces(nx / 2, ny / 2, nz / 2)
    g.step(wb.TRT, n=2)
    g.synchronize()
    held = wb.lib.wake_grid_device_bytes(g.handle)
    estimate = wb.lib.wake_grid_estimate_bytes(q, nx, ny, nz, {"f32": 0, "f16": 1}[storage], 0)
    print(f"[memory] {held / 1e6:.1f} MB held, {estimate / 1e6:.1f} MB estimated")
    assert held <= estimate
