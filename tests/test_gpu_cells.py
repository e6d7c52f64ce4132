"""The step over 64-node cells where its cells, segments and lists have edges.

Rows that are no multiple of 64 nodes (cells run over row ends), rows shorter than a cell, lattices smaller than one,
odd node counts (16-bit pairs start on odd nodes), short runs of pure gathers between obstacles, more curved links in a
cell than a warp takes at once. Tolerances are those of the other oracle comparisons: velocity within twice an FP32
CPU implementation's error against FP64 (or 1e-5), density 1e-5, force history 1e-4, and 1e-3 / 1e-2 for 16-bit
storage (one stored value is rounded to 2^-11 / 2^-8 of its deviation each step).
"""
import numpy as np
import pytest

from conftest import rel_l2, vel_rel_l2
from test_gpu_grid import FORCE_TOL, RHO_TOL, U_TOL, _run_case_gpu, _run_case_oracle

pytestmark = pytest.mark.gpu

wb = pytest.importorskip("wake_b200")
from wake_b200 import workloads as W  # noqa: E402

STEPS = 20
SPHERES = {  # (nx, ny, nz, radius, center)
    "under_a_cell": (20, 12, 12, 3.0, (8.0, 6.0, 6.0)),
    "one_segment": (64, 14, 12, 3.0, (20.0, 7.0, 6.0)),
    "one_node_over": (65, 13, 12, 3.0, (20.0, 6.0, 6.0)),
    "odd": (81, 15, 13, 4.0, (30.0, 7.0, 6.0)),
    "two_segments": (128, 12, 12, 3.0, (64.0, 6.0, 6.0)),
    "short_runs": (200, 12, 12, 4.0, (100.0, 6.0, 6.0)),
    "many_links": (64, 24, 12, 300.0, (32.0, -290.0, 6.0)),
}
CYLINDERS = {  # (nx, ny, diameter, cx, cy)
    "under_a_cell": (24, 16, 4, 8, 8),
    "one_node_over": (65, 24, 6, 20, 12),
    "odd": (99, 33, 8, 30, 16),
    "short_runs": (200, 40, 10, 100, 20),
    "long_rows": (1100, 20, 6, 300, 10),
}


def _check(case, storage, u_tol, rho_tol, force_tol):
    g = _run_case_gpu(case, STEPS, storage)
    links = g.curved_links() if case.q == 19 else None
    m, hist = g.macro(), g.force_history()
    o32, h32 = _run_case_oracle(case, STEPS, 32, links)
    o64, _ = _run_case_oracle(case, STEPS, 64, links)
    keys = ("ux", "uy", "uz") if case.q != 9 else ("ux", "uy")
    m32, m64 = o32.macro(), o64.macro()
    e64, e_o64 = vel_rel_l2(m, m64, keys), vel_rel_l2(m32, m64, keys)
    assert e64 <= max(u_tol, 2.0 * e_o64)
    assert rel_l2(m["rho"], m32["rho"]) <= rho_tol
    assert hist.shape[0] == STEPS and rel_l2(hist, h32) <= force_tol


@pytest.mark.parametrize("collision", [wb.BGK, wb.TRT, wb.MRT])
@pytest.mark.parametrize("shape", sorted(SPHERES))
def test_sphere_shapes_match_oracle(shape, collision):
    nx, ny, nz, r, c = SPHERES[shape]
    case = W.sphere_channel(nx, ny, nz, r, c, tau=0.55, collision=collision, les=collision == wb.TRT)
    _check(case, "f32", U_TOL, RHO_TOL, FORCE_TOL)


@pytest.mark.parametrize("collision", [wb.BGK, wb.TRT, wb.MRT])
@pytest.mark.parametrize("shape", sorted(CYLINDERS))
def test_cylinder_shapes_match_oracle(shape, collision):
    nx, ny, d, cx, cy = CYLINDERS[shape]
    _check(W.cylinder_channel(nx, ny, d, cx, cy, collision=collision), "f32", U_TOL, RHO_TOL, FORCE_TOL)


@pytest.mark.parametrize("storage,tol", [("f16", 1e-3), ("bf16", 1e-2), ("f16c", 1e-3)])
@pytest.mark.parametrize("shape", ["one_node_over", "odd", "short_runs"])
def test_16bit_shapes_against_fp64(shape, storage, tol):
    nx, ny, nz, r, c = SPHERES[shape]
    case = W.sphere_channel(nx, ny, nz, r, c, tau=0.55, collision=wb.TRT)
    g = _run_case_gpu(case, STEPS, storage)
    o64, _ = _run_case_oracle(case, STEPS, 64, g.curved_links())
    assert vel_rel_l2(g.macro(), o64.macro(), ("ux", "uy", "uz")) <= tol


@pytest.mark.parametrize("variant", [1, 3])
def test_force_history_does_not_depend_on_the_reads(variant):
    """The force of a step is appended by the next step's launch or by a read: reads and changes of kernel between
    steps, and steps replayed from a graph, leave the same history."""
    case = W.sphere_channel(128, 16, 16, 4.0, (40.0, 8.0, 8.0), tau=0.55, collision=wb.TRT)
    model = dict(use_les=case.les, smag_const=case.cs_smag)
    a, b, c = (W.build_grid(case) for _ in range(3))
    for g in (a, b, c):
        wb.check(wb.lib.wake_grid_set_kernel(g.handle, variant))
    a.step(case.collision, n=24, **model)
    for k in range(24):
        wb.check(wb.lib.wake_grid_set_kernel(b.handle, variant if k % 3 else 4 - variant))
        b.step(case.collision, n=1, **model)
        if k % 2:
            assert b.force_history().shape[0] == k + 1
    c.use_graph(4)
    c.step(case.collision, n=10, **model)
    assert c.force_history().shape[0] == 10
    c.step(case.collision, n=14, **model)
    want = a.force_history()
    assert want.shape[0] == 24 and np.all(np.any(want != 0.0, axis=1))
    assert np.array_equal(want, b.force_history()) and np.array_equal(want, c.force_history())


def test_members_of_all_shapes_equal_single_lattices():
    """One launch over members whose cells end differently gives each member its single-lattice result."""
    from wake_b200.batch import Batch

    cases = [W.cylinder_channel(*CYLINDERS[k], collision=wb.TRT) for k in sorted(CYLINDERS)]
    batch = Batch(q=9)
    grids = [W.build_grid(case) for case in cases]
    for g in grids:
        batch.add(g, wb.TRT)
    batch.step(STEPS)
    batch.synchronize()
    for case, g in zip(cases, grids):
        alone = W.build_grid(case)
        alone.step(wb.TRT, n=STEPS)
        m, want = g.macro(), alone.macro()
        assert np.array_equal(m["ux"], want["ux"]) and np.array_equal(m["rho"], want["rho"])
        assert np.array_equal(g.force_history(), alone.force_history())


def test_moments_reach_every_kind_of_buffer():
    """Moments go straight to aligned device memory and by way of a copy elsewhere: the same values either way,
    whatever is left out, and the later field where two share a buffer."""
    import ctypes

    import torch

    case = W.cylinder_channel(*CYLINDERS["odd"], collision=wb.TRT)
    g = _run_case_gpu(case, STEPS)
    n = case.nx * case.ny
    names = ("rho", "ux", "uy", "speed")
    host = {k: np.zeros(n, np.float32) for k in names}
    g.macroscopic_into(**host)
    device = {k: torch.zeros(n, dtype=torch.float32, device="cuda") for k in names}
    torch.cuda.synchronize()
    g.macroscopic_into(**device)
    for k in names:
        assert np.array_equal(device[k].cpu().numpy(), host[k])
        one = torch.zeros(n, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        g.macroscopic_into(**{k: one})
        assert np.array_equal(one.cpu().numpy(), host[k])
    both = torch.zeros(n + 7, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g.macroscopic_into(rho=both[:n], uy=both[7:])  # uy is written after rho
    want = np.concatenate([host["rho"][:7], host["uy"]])
    assert np.array_equal(both.cpu().numpy(), want)
    raw = torch.zeros(4 * n + 1, dtype=torch.uint8, device="cuda")  # no float's alignment
    torch.cuda.synchronize()
    wb.check(wb.lib.wake_grid_get_macroscopic(g.handle, ctypes.c_void_p(raw.data_ptr() + 1), None, None, None, None))
    assert np.array_equal(raw.cpu().numpy()[1:].view(np.float32), host["rho"])
