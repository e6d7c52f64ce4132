"""A batch whose members' model or parameters change between replays of its graph.

Results are the single lattice's, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wb = pytest.importorskip("wake_b200")
from wake_b200 import workloads as W  # noqa: E402
from wake_b200.batch import Batch  # noqa: E402


@pytest.mark.parametrize("q,storage", [(9, "f32"), (19, "f32"), (9, "f16")])
def test_graph_follows_a_change_of_model(q, storage):
    """Collision model, then the LES switch, changed on every member after the graph was captured."""
    if q == 9:
        cases = [W.cylinder_channel(80, 32, 6, 20, 16), W.cylinder_channel(65, 24, 6, 20, 12)]
    else:
        cases = [W.sphere_channel(32, 16, 16, 4.0, (10.0, 8.0, 8.0), tau=0.55)]
    models = [(wb.BGK, False), (wb.MRT, False), (wb.MRT, True), (wb.TRT, True)]
    with Batch(q, storage) as batch:
        grids = [W.build_grid(c, storage=storage) for c in cases]
        for g in grids:
            batch.add(g, *models[0], 0.17)
        batch.use_graph(4)
        batch.step(8)  # the buffers are the same ones again
        for model in models[1:]:
            for g in grids:
                g._apply_model(*model, 0.17)
            batch.step(8)
        batch.synchronize()
        for g, case in zip(grids, cases):
            alone = W.build_grid(case, storage=storage)
            for collision, les in models:
                alone.step(collision, use_les=les, smag_const=0.17, n=8)
            assert np.array_equal(g.f_src_data(), alone.f_src_data())
            assert np.array_equal(g.force_history(), alone.force_history())


def test_graph_follows_a_change_of_a_member_beyond_32_bit_offsets():
    """A member of 2^32 or more values steps by its own launches, whose arguments a graph holds by value."""
    nx = ny = 21846
    assert 9 * nx * ny >= 1 << 32

    def flow():
        g = wb.LatticeGrid2D(nx, ny, 0.6, storage="f16")
        wb.check(wb.lib.wake_grid_initialize_noise(g.handle, 1.0, 0.04, 0.0, 0.0, 0.02, 7, 0))
        return g

    with Batch(9, "f16") as batch:
        g = flow()
        batch.add(g, wb.BGK)
        assert batch.info()["launches_per_step"] == 1
        batch.use_graph(2)
        batch.step(2)
        g.set_relaxation_time(0.9)
        batch.step(2)
        batch.synchronize()
        got = g._diag()
        batch.remove(g)
        g.close()
    alone = flow()
    alone.step(wb.BGK, n=2)
    alone.set_relaxation_time(0.9)
    alone.step(wb.BGK, n=2)
    want = alone._diag()
    alone.close()
    wb.lib.wake_gpu_cache_trim()
    assert got == want
