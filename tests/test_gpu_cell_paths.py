"""Steps over geometry, models and options that the scenario tests do not combine, against the oracle.

Tolerances are those of the other oracle comparisons: velocity within twice an FP32 CPU implementation's error against
FP64 (or 1e-5), density 1e-5, force history 1e-4.
"""
import numpy as np
import pytest

from conftest import rel_l2, vel_rel_l2
from test_gpu_grid import FORCE_TOL, RHO_TOL, U_TOL

pytestmark = pytest.mark.gpu

wb = pytest.importorskip("wake_b200")
import oracle  # noqa: E402

STEPS = 20
TAU = 0.56
SMAG = 0.6  # the eddy viscosity is then a few per cent of the flow's
GRIDS = {9: wb.LatticeGrid2D, 19: wb.LatticeGrid3D, 27: wb.LatticeGrid3DQ27}


def _waves(q, nx, ny, nz):
    """Density and velocity of a few long waves, every component non-zero, as float32 arrays."""
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    a, b, c = (2.0 * np.pi * v / n for v, n in ((x, nx), (y, ny), (z, nz)))
    u = (0.04 + 0.02 * np.sin(a + b + 0.3), 0.02 * np.cos(a - c) + 0.01 * np.sin(b), 0.015 * np.sin(c + a + 1.0))
    rho = 1.0 + 0.01 * np.sin(a + 2.0 * b)
    out = [np.ascontiguousarray(v, np.float32).ravel() for v in (rho, *u)]
    if q == 9:
        out[3] = np.zeros_like(out[3])
    return out


def _step_both(q, size, types, collision, les=False, force=(0.0, 0.0, 0.0), wall=None, periodic=(False, False), links=None,
               mem=None, tau=TAU, steps=STEPS):
    """(grid, oracle FP32, oracle FP64, its FP32 force history) after the same steps from the same populations.
    wall: velocity of the MOVING_WALL cells; links: (node, direction, delta, velocity)."""
    nx, ny, nz = size
    types = np.ascontiguousarray(types, np.uint8).ravel()
    f0 = oracle.equilibrium(q, *_waves(q, nx, ny, nz), prec=32).astype(np.float32)
    g = GRIDS[q](nx, ny, tau) if q == 9 else GRIDS[q](nx, ny, nz, tau)
    if wall is not None:
        wb.check(wb.lib.wake_grid_set_moving_wall(g.handle, *wall))
    g.set_cell_types(types)
    if q != 9:
        g.set_periodic_axes(*periodic)
    if links is not None:
        g.set_curved_links(*links)
    g.set_populations(f0)
    if mem is not None:
        g.enable_forces(*mem)
    gz = {} if q == 9 else {"gz": force[2]}
    g.step(collision, gx=force[0], gy=force[1], use_les=les, smag_const=SMAG, n=steps, **gz)
    g.synchronize()
    out = [g]
    for prec in (32, 64):
        o = oracle.OracleGrid(q, nx, ny, nz, prec)
        kw = {} if wall is None else {"u_wall": wall}
        if mem is not None:
            kw.update(mem=1, center=mem[:3], r_max=mem[3])
        o.configure(collision=collision, tau=tau, les=int(les), cs_smag=SMAG, g=force, periodic_y=int(periodic[0]),
                    periodic_z=int(periodic[1]), **kw)
        o.set_cell_types(types)
        o.set_state(f0)
        if links is not None:
            o.set_links(*links)
        hist = o.step(steps, forces=mem is not None)
        out.append(o)
        if prec == 32:
            h32 = hist
    return (*out, h32)


def _check(q, *args, **kw):
    g, o32, o64, h32 = _step_both(q, *args, **kw)
    keys = ("ux", "uy") if q == 9 else ("ux", "uy", "uz")
    m, m32, m64 = g.macro(), o32.macro(), o64.macro()
    e64, e_o64 = vel_rel_l2(m, m64, keys), vel_rel_l2(m32, m64, keys)
    print(f"[D?Q{q}] u vs FP64 {e64:.2e} (oracle-fp32 {e_o64:.2e}), rho vs oracle-fp32 {rel_l2(m['rho'], m32['rho']):.2e}")
    assert e64 <= max(U_TOL, 2.0 * e_o64)
    assert rel_l2(m["rho"], m32["rho"]) <= RHO_TOL
    if kw.get("mem") is not None:
        hist = g.force_history()
        assert hist.shape[0] == STEPS and np.any(h32 != 0.0) and rel_l2(hist, h32) <= FORCE_TOL


@pytest.mark.parametrize("collision", [wb.BGK, wb.TRT, wb.MRT])
@pytest.mark.parametrize("q,size,solid", [(9, (72, 64, 1), (68, 63, 0)), (19, (80, 16, 12), (72, 15, 11)),
                                          (27, (80, 16, 12), (72, 15, 11))])
def test_pure_run_ends_within_the_last_inner_row(q, size, solid, collision):
    """A cell shorter than 64 nodes at the end of the last rows whose pulls stay inside, in a lattice whose node count
    leaves no padding behind the planes."""
    nx, ny, nz = size
    types = np.zeros((nz, ny, nx), np.uint8)
    types[solid[2], solid[1], solid[0]] = wb.SOLID
    _check(q, size, types, collision)


def _walls(nx, ny, nz):
    """A block of solid cells inside and one that crosses the x faces."""
    types = np.zeros((nz, ny, nx), np.uint8)
    types[nz // 3:nz // 3 + 3, ny // 2:ny // 2 + 3, nx // 4:nx // 4 + 5] = wb.SOLID
    types[0, 0, -1] = types[0, 0, 0] = wb.SOLID
    return types


MODELS = [(wb.BGK, False), (wb.BGK, True), (wb.TRT, True), (wb.MRT, False), (wb.MRT, True)]


@pytest.mark.parametrize("collision,les", MODELS)
@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (2e-5, -1e-5, 3e-5)])
def test_models_over_walls(q, force, collision, les):
    """Every collision model with and without Smagorinsky and body force, over general cells of the 3D lattices."""
    size = (70, 12, 9)
    _check(q, size, _walls(*size), collision, les=les, force=force, mem=(19.0, 7.0, 4.0, 8.0))


@pytest.mark.parametrize("collision,les", MODELS)
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (2e-5, -1e-5, 0.0)])
def test_models_over_walls_2d(force, collision, les):
    size = (99, 33, 1)
    types = np.zeros((1, 33, 99), np.uint8)
    types[0, 12:17, 30:34] = wb.SOLID
    _check(9, size, types, collision, les=les, force=force, mem=(31.0, 14.0, 0.0, 8.0))


@pytest.mark.parametrize("collision", [wb.BGK, wb.TRT, wb.MRT])
@pytest.mark.parametrize("q", [9, 19, 27])
def test_moving_wall(q, collision):
    size = (70, 12, 1 if q == 9 else 9)
    types = _walls(*size) if q != 9 else np.zeros(size[::-1], np.uint8)
    types[:, -1, :] = wb.MOVING_WALL
    _check(q, size, types, collision, wall=(0.05, 0.0, 0.0 if q == 9 else 0.02), periodic=(False, q != 9))


@pytest.mark.parametrize("collision", [wb.BGK, wb.TRT, wb.MRT])
def test_moving_curved_links(collision):
    """Links of a sphere that turns: their moving-wall terms, for delta below and above one half."""
    size = nx, ny, nz = 66, 14, 12
    at, radius = (20.0, 7.0, 6.0), 3.3
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    types = ((x - at[0]) ** 2 + (y - at[1]) ** 2 + (z - at[2]) ** 2 <= radius ** 2).astype(np.uint8) * wb.SOLID
    g = wb.LatticeGrid3D(nx, ny, nz, TAU)
    g.set_cell_types(types)
    g.build_curved_sphere_links(*at, radius)
    node, direction, delta = g.curved_links()
    g.close()
    assert (delta < 0.5).any() and (delta >= 0.5).any()
    rx, ry = node % nx - at[0], (node // nx) % ny - at[1]
    uw = np.stack([-0.01 * ry, 0.01 * rx, np.full(len(node), 0.005)], axis=1).astype(np.float32)
    uw[::3] = 0.0  # and links at rest among them
    _check(19, size, types, collision, links=(node, direction, delta, uw), periodic=(True, True), mem=(*at, 6.0))


def test_moments_into_a_buffer_that_is_too_short_are_refused():
    """A device buffer whose allocation ends before the field does: an error from the host, as from a copy to it."""
    import ctypes

    import torch

    torch.cuda.synchronize()
    g = wb.LatticeGrid2D(65, 33, TAU)
    g.step(wb.TRT, n=2)
    cuda = ctypes.CDLL("libcuda.so.1")
    p = ctypes.c_uint64()
    assert cuda.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(4096)) == 0  # 65 x 33 floats take 8,580 B
    try:
        with pytest.raises(RuntimeError):
            wb.check(wb.lib.wake_grid_get_macroscopic(g.handle, None, ctypes.c_void_p(p.value), None, None, None))
    finally:
        assert cuda.cuMemFree_v2(p) == 0
    wb.lib.wake_gpu_clear_error()
    whole = torch.zeros(65 * 33, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g.macroscopic_into(ux=whole)
    assert np.array_equal(whole.cpu().numpy(), g.macro()["ux"])


def test_outlet_face_keeps_an_infinite_correction():
    """Where the outlet's density sum overflows, its unknown populations are a finite value minus infinity."""
    nx, ny, nz = 16, 8, 8
    types = np.zeros((nz, ny, nx), np.uint8)
    types[:, :, -1] = wb.OUTFLOW
    f0 = oracle.equilibrium(19, *_waves(19, nx, ny, nz), prec=32).astype(np.float32).reshape(19, nz, ny, nx)
    f0[:, :, :, -2] = 0.0
    f0[1, :, :, -2] = 2.5e38  # u = 1: BGK at tau = 1 sends 7/18 of it and 7/36 along each diagonal to the face
    g = wb.LatticeGrid3D(nx, ny, nz, 1.0)
    g.set_outflow_east(1.0)
    g.set_cell_types(types)
    g.set_periodic_axes(True, True)
    g.set_populations(f0.reshape(19, -1))
    g.step(wb.BGK, n=1)
    got = g.f_src_data()
    o = oracle.OracleGrid(19, nx, ny, nz, 32)
    o.configure(collision=wb.BGK, tau=1.0, outflow=1, rho_out=1.0, periodic_y=1, periodic_z=1)
    o.set_cell_types(types)
    o.set_state(f0.reshape(19, -1))
    o.step(1)
    want = o.f()
    assert np.count_nonzero(np.isneginf(want)) == 5 * ny * nz  # directions 2, 8, 10, 12, 14 of the face
    assert np.array_equal(np.isneginf(got), np.isneginf(want)) and np.array_equal(np.isnan(got), np.isnan(want))


def test_forces_of_a_callers_graph_between_steps_of_another_kernel():
    """Replays of a graph the caller captured with one kernel and steps with another leave one history in order."""
    import torch

    from wake_b200 import workloads as W

    case = W.sphere_channel(64, 16, 16, 4.0, (20.0, 8.0, 8.0), tau=0.55, collision=wb.TRT)
    model = dict(use_les=case.les, smag_const=case.cs_smag)
    g, alone = W.build_grid(case, storage="f16"), W.build_grid(case, storage="f16")
    stream = torch.cuda.Stream()
    g.set_stream(stream.cuda_stream)
    g.step(case.collision, n=2, **model)
    assert wb.lib.wake_grid_get_kernel(g.handle) == 4
    g.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        g.step(case.collision, n=2, **model)
    with torch.cuda.stream(stream):
        graph.replay()
        for _ in range(3):
            wb.check(wb.lib.wake_grid_set_kernel(g.handle, 1))
            g.step(case.collision, n=2, **model)
            graph.replay()
    got = g.force_history()
    alone.step(case.collision, n=16, **model)
    want = alone.force_history()
    assert want.shape[0] == 16 and np.all(np.any(want != 0.0, axis=1))
    assert np.array_equal(got, want)
