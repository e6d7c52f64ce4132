"""Performance cases of the lattice update: what programs that use this package have it do.

Each case is one pass of such a program through the public entry points (the grid classes,
``Batch``, ``FieldAnalytics`` and the drop-in C functions), with the read-out that follows it.
``exact`` gives the same outputs from a plain FP64 restatement of the scheme in torch.

The initial velocity of every flow is its mean flow plus a few long waves with phases from the
seed (a developed, not a uniform, state): all velocity components matter.
"""
import math

import numpy as np
import torch

import wake_b200 as wb
from wake_b200.batch import Batch

BGK, TRT, MRT = 0, 1, 2
FLUID, SOLID, INFLOW, OUTFLOW = 0, 1, 2, 3
DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: an interactive loop that advances a small forced channel by one step with
        # the default model (MRT) and shows the fields; odd sizes
        {"name": "channel2d_step_and_show", "kind": "channel2d", "nx": 65, "ny": 33, "coll": MRT, "steps": 1},
        # the vortex-street scenario: BGK cylinder channel with lift and drag every step, plain stepping
        {"name": "cylinder2d_bgk", "kind": "cylinder2d", "nx": 400, "ny": 160, "coll": BGK, "steps": 50},
        # the package's headline flow: sphere channel, TRT + Smagorinsky, curved links, Zou-He faces,
        # forces every step, 20-step graphs
        {"name": "sphere_f32", "kind": "sphere", "nx": 256, "ny": 128, "nz": 128, "storage": "f32", "graph": 20, "steps": 20},
        # the same with IEEE half storage, the resident state handed over as it is
        {"name": "sphere_f16", "kind": "sphere", "nx": 256, "ny": 128, "nz": 128, "storage": "f16", "graph": 20, "steps": 20},
        # the storage for long 16-bit runs, on a lattice whose rows are no multiple of 64, plain stepping
        {"name": "sphere_f16c", "kind": "sphere", "nx": 200, "ny": 100, "nz": 100, "storage": "f16c", "graph": 0, "steps": 20},
        # one served job from its fields to its results: grid, geometry, links, steps, read-out; odd edge
        {"name": "sphere_job", "kind": "job", "n": 81, "steps": 200},
        # the 3D scenario in the form the reference host has: MRT (the default), x-periodic, walls in y and z
        {"name": "sphere_mrt_walls", "kind": "duct", "nx": 192, "ny": 96, "nz": 96, "coll": MRT, "steps": 20},
        # the largest: Taylor-Green vortex on D3Q27, MRT
        {"name": "taylor_green_d3q27", "kind": "tgv", "edge": 384, "q": 27, "coll": MRT, "storage": "f32", "steps": 10},
        # a parameter sweep: many 2D ellipse channels of uneven sizes advanced together, 20-step graphs
        {"name": "ellipse_batch", "kind": "batch", "members": 60, "layout": 1, "steps": 100},
        # natural convection: D2Q9 flow with a coupled temperature
        {"name": "thermal_cell", "kind": "thermal", "nx": 384, "ny": 192, "steps": 50},
        # one time step of a host program that keeps its own device buffers and calls the drop-in kernels
        {"name": "dropin_d3q19", "kind": "dropin", "nx": 128, "ny": 128, "nz": 128},
        # a visualisation frame: vorticity and Q-criterion of a resident 3D flow
        {"name": "snapshot_3d", "kind": "snapshot", "nx": 256, "ny": 128, "nz": 128, "storage": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel2d", "cylinder2d", "sphere", "sphere", "job", "duct", "tgv", "batch", "thermal",
                       "dropin", "snapshot"])
    if kind == "channel2d":
        return {"kind": kind, "nx": _log(rng, 16, 1024), "ny": _log(rng, 8, 512), "coll": rng.choice([BGK, TRT, MRT]),
                "steps": _log(rng, 1, 20)}
    if kind == "cylinder2d":
        nx = rng.randint(200, 1200)
        return {"kind": kind, "nx": nx, "ny": rng.randint(2 * nx // 5, nx // 2), "coll": rng.choice([BGK, TRT, MRT]),
                "steps": rng.randint(20, 100)}
    if kind == "sphere":
        return {"kind": kind, "nx": rng.randint(64, 320), "ny": rng.randint(48, 160), "nz": rng.randint(48, 160),
                "storage": rng.choice(["f32", "f32", "f16", "bf16", "f16c"]), "graph": rng.choice([0, 20]),
                "steps": rng.randint(5, 20)}
    if kind == "job":
        return {"kind": kind, "n": rng.randint(48, 160), "steps": rng.randint(100, 300)}
    if kind == "duct":
        return {"kind": kind, "nx": rng.randint(64, 256), "ny": rng.randint(48, 128), "nz": rng.randint(48, 128),
                "coll": rng.choice([BGK, TRT, MRT]), "steps": rng.randint(5, 20)}
    if kind == "tgv":
        return {"kind": kind, "edge": _log(rng, 32, 256), "q": rng.choice([19, 27]), "coll": rng.choice([TRT, MRT]),
                "storage": rng.choice(["f32", "f32", "f16c"]), "steps": rng.randint(5, 20)}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(8, 60), "layout": rng.randint(2, 1 << 20), "steps": rng.randint(40, 100)}
    if kind == "thermal":
        nx = rng.randint(64, 512)
        return {"kind": kind, "nx": nx, "ny": nx // 2, "steps": rng.randint(20, 100)}
    if kind == "dropin":
        return {"kind": kind, "nx": rng.randint(24, 200), "ny": rng.randint(24, 160), "nz": rng.randint(24, 160)}
    return {"kind": kind, "nx": rng.randint(32, 300), "ny": rng.randint(32, 160), "nz": rng.randint(32, 160),
            "storage": rng.choice(["f32", "f16"])}


# ------------------------------------------------------------------ inputs
def _waves(shape, seed, mean, amp):
    """(rho, u_x, u_y, u_z) of `shape` (nz, ny, nx): mean flow plus four long waves per component."""
    rs = np.random.RandomState(seed % (1 << 32))
    nz, ny, nx = shape
    ax = [2.0 * math.pi * (torch.arange(n, dtype=F64, device=DEV) + 0.5) / n for n in (nx, ny, nz)]
    dims = 3 if nz > 1 else 2
    out = []
    for c in range(4):
        f = torch.zeros(shape, dtype=F64, device=DEV)
        if c <= dims:
            for _ in range(4):
                k = rs.randint(1, 4, 3)
                p = rs.uniform(0.0, 2.0 * math.pi, 3)
                w = torch.cos(k[0] * ax[0] + p[0])[None, None, :] * torch.cos(k[1] * ax[1] + p[1])[None, :, None]
                if dims == 3:
                    w = w * torch.cos(k[2] * ax[2] + p[2])[:, None, None]
                f += (0.5 * amp if dims == 2 else amp) * w
        base = (1.0, mean, 0.0, 0.0)[c]
        out.append((base + (0.2 * f if c == 0 and dims == 2 else 0.1 * f if c == 0 else f)).float().reshape(-1).contiguous())
    return out


def _sphere_of(case):
    """Centre and radius in the proportions of the 256 x 128 x 128 channel."""
    nx, ny, nz = (case["n"],) * 3 if case["kind"] == "job" else (case["nx"], case["ny"], case["nz"])
    r = 3.0 * min(nx, ny, nz) / 32.0
    return (nx / 4.0, ny / 2.0, nz / 2.0), r


def _sphere_mask(shape, centre, r):
    nz, ny, nx = shape
    f = np.float32
    d = [(np.arange(n, dtype=f) - f(c)) ** 2 for n, c in ((nx, centre[0]), (ny, centre[1]), (nz, centre[2]))]
    return ((d[0][None, None, :] + d[1][None, :, None]) + d[2][:, None, None]) <= f(r) * f(r)


def _ellipses(case):
    """The sweep's domains: (nx, ny, chord, tau, solid mask); sizes and shapes from the case's layout number."""
    rs = np.random.RandomState(case["layout"])
    got = []
    f = np.float32
    for _ in range(case["members"]):
        nx = int(rs.randint(64, 513))
        ny = nx // 2
        a = ny / 16.0 + rs.rand() * (ny / 6.0 - ny / 16.0)
        b = max(ny / 16.0, a / 3.0) + rs.rand() * (a - max(ny / 16.0, a / 3.0))
        ang = math.radians(20.0 * rs.rand())
        tau = 0.5 + 3.0 * 0.05 * 2.0 * a / (50.0 + 250.0 * rs.rand())
        X, Y = np.meshgrid(np.arange(nx, dtype=f) - f(nx / 5.0), np.arange(ny, dtype=f) - f(ny / 2.0))
        u, v = X * f(math.cos(ang)) + Y * f(math.sin(ang)), Y * f(math.cos(ang)) - X * f(math.sin(ang))
        solid = (u / f(a)) ** 2 + (v / f(b)) ** 2 <= 1.0
        solid[0, :] = solid[-1, :] = True
        got.append((nx, ny, 2.0 * a, tau, solid))
    return got


def _types2d(solid, faces):
    t = np.zeros(solid.shape, np.uint8)
    if faces:
        t[:, 0], t[:, -1] = INFLOW, OUTFLOW
    t[solid] = SOLID
    return t


def _cylinder(case):
    """Layout of the cylinder scenario: solid rows at y = 0 and y = ny - 1 and a disk of diameter ny / 8."""
    nx, ny = case["nx"], case["ny"]
    d, cx, cy = ny / 8.0, nx / 5.0, ny / 2.0
    f = np.float32
    X, Y = np.meshgrid(np.arange(nx, dtype=f) - f(cx), np.arange(ny, dtype=f) - f(cy))
    solid = X * X + Y * Y <= f(d / 2.0) ** 2
    solid[0, :] = solid[-1, :] = True
    return solid, (cx, cy, 0.0, 1.5 * d)


def _temperature(case, seed):
    nx, ny = case["nx"], case["ny"]
    rs = np.random.RandomState((seed + 5) % (1 << 32))
    T = 1.0 - (np.arange(ny, dtype=np.float64)[:, None] + 0.5) / ny + np.zeros((ny, nx))
    x, y = np.arange(nx)[None, :] * (2 * math.pi / nx), np.arange(ny)[:, None] * (math.pi / ny)
    for _ in range(4):
        T += 0.05 * np.cos(rs.randint(1, 5) * x + rs.rand() * 6.28) * np.sin(rs.randint(1, 4) * y)
    return T.astype(np.float32)


def _thermal_of(case):
    """Rayleigh number 1e5, Prandtl number 0.71, free-fall velocity 0.05."""
    ny = case["ny"]
    gbeta = 0.05 ** 2 / ny
    nu = math.sqrt(gbeta * ny ** 3 / 1e5 * 0.71)
    return 0.5 + 3.0 * nu, 0.5 + 3.0 * nu / 0.71, gbeta


TAU_SPHERE, CS, U_IN = 0.52, 0.17, 0.05


# ------------------------------------------------------------------ the program before the call
class _View:
    """A device buffer of the library as an array (state buffers of a resident grid)."""

    def __init__(self, ptr, shape, typestr, strides):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 3,
                                         "strides": strides}


def _state_view(g):
    """The current populations [q][node] of a resident grid, in its storage type, without a copy."""
    e, ts = (4, "<f4") if g.storage == "f32" else (2, "<f2" if g.storage == "f16" else "<i2")
    n = g.total_nodes()
    v = torch.as_tensor(_View(wb.lib.wake_grid_state_buffer(g.handle, 0), (g.Q, n), ts, ((n + 63) // 64 * 64 * e, e)),
                        device=DEV)
    return v if g.storage in ("f32", "f16") else v.view(torch.bfloat16)


def _macro_buffers(n, dims):
    return {k: torch.empty(n, dtype=torch.float32, device=DEV)
            for k in (("rho", "ux", "uy", "uz", "speed") if dims == 3 else ("rho", "ux", "uy", "speed"))}


def _sphere_grid(case, storage, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    (cx, cy, cz), r = _sphere_of(case)
    g = wb.LatticeGrid3D(nx, ny, nz, TAU_SPHERE, storage=storage)
    g.initialize_fields(*_synced(_waves((nz, ny, nx), seed, U_IN, 0.02)))
    g.set_periodic_axes(True, True)
    g.set_inflow_west(U_IN)
    g.set_outflow_east(1.0)
    g.set_solid_sphere(cx, cy, cz, r)
    g.build_curved_sphere_links(cx, cy, cz, r)
    g.enable_forces(cx, cy, cz, 2.0 * r, case.get("steps", 1))
    return g


def _synced(t):
    torch.cuda.synchronize()
    return t


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k in ("channel2d", "cylinder2d"):
        nx, ny = case["nx"], case["ny"]
        if k == "channel2d":
            solid = np.zeros((ny, nx), bool)
            solid[0, :] = solid[-1, :] = True
            g = wb.LatticeGrid2D(nx, ny, 0.8)
        else:
            solid, mem = _cylinder(case)
            g = wb.LatticeGrid2D(nx, ny, 0.56)
        g.initialize_fields(*_synced(_waves((1, ny, nx), seed, U_IN, 0.02))[:3])
        if k == "cylinder2d":
            g.set_inflow_west(U_IN)
            g.set_outflow_east(1.0)
            g.enable_forces(*mem, case["steps"])
        g.set_cell_types(_types2d(solid, k == "cylinder2d"))
        s.update(g=g, out=_macro_buffers(nx * ny, 2))
    elif k == "sphere":
        g = _sphere_grid(case, case["storage"], seed)
        g.use_graph(case["graph"])
        g.prepare_steps(TRT, use_les=True, smag_const=CS)
        s.update(g=g)
        if case["storage"] in ("f32", "f16c"):
            s["out"] = _macro_buffers(g.total_nodes(), 3)
    elif k == "job":
        n = case["n"]
        f = _waves((n, n, n), seed, U_IN, 0.02)
        s.update(fields=[a.cpu().pin_memory().numpy() for a in f], out=[torch.empty(n ** 3).pin_memory() for _ in range(5)])
    elif k == "duct":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        (cx, cy, cz), r = _sphere_of(case)
        g = wb.LatticeGrid3D(nx, ny, nz, 0.6)
        g.initialize_fields(*_synced(_waves((nz, ny, nx), seed, U_IN, 0.02)))
        g.set_solid_sphere(cx, cy, cz, r)
        g.build_curved_sphere_links(cx, cy, cz, r)
        g.enable_forces(cx, cy, cz, 2.0 * r, case["steps"])
        s.update(g=g, out=_macro_buffers(nx * ny * nz, 3))
    elif k == "tgv":
        e = case["edge"]
        cls = wb.LatticeGrid3D if case["q"] == 19 else wb.LatticeGrid3DQ27
        g = cls(e, e, e, 0.51, storage=case["storage"])
        g.initialize_fields(*_synced(_waves((e, e, e), seed, 0.0, 0.03)))
        g.set_periodic_axes(True, True)
        s.update(g=g, out=_macro_buffers(e ** 3, 3))
    elif k == "batch":
        b = Batch(q=9)
        for i, (nx, ny, chord, tau, solid) in enumerate(_ellipses(case)):
            g = wb.LatticeGrid2D(nx, ny, tau)
            g.initialize_fields(*_synced(_waves((1, ny, nx), seed + i, U_IN, 0.01))[:3])
            g.set_inflow_west(U_IN)
            g.set_outflow_east(1.0)
            g.set_cell_types(_types2d(solid, True))
            g.enable_forces(nx / 5.0, ny / 2.0, 0.0, 1.5 * chord, case["steps"])
            b.add(g, TRT, use_les=True, smag_const=CS)
        b.use_graph(20)
        s.update(b=b)
    elif k == "thermal":
        tau, tau_t, gbeta = _thermal_of(case)
        g = wb.LatticeGrid2D(case["nx"], case["ny"], tau)
        g.initialize_fields(*_synced(_waves((1, case["ny"], case["nx"]), seed, 0.0, 0.02))[:3])
        g.enable_thermal(tau_t, 0.5, gbeta, 1.0, 0.0)
        g.initialize_temperature(_temperature(case, seed))
        s.update(g=g, out=_macro_buffers(case["nx"] * case["ny"], 2))
    elif k == "dropin":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        c, r = _sphere_of(case)
        w = _waves((nz, ny, nx), seed, U_IN, 0.02)
        f = _feq(19, [a.double().view(nz, ny, nx) for a in w]).float().view(19, -1).contiguous()
        t = torch.from_numpy(_sphere_mask((nz, ny, nx), c, r).astype(np.uint8)).to(DEV)
        s.update(f=f, g=torch.empty_like(f), t=t, out=_macro_buffers(nx * ny * nz, 3),
                 F=torch.zeros(3, dtype=torch.float32, device=DEV), c=c, r=r)
        torch.cuda.synchronize()
    else:  # snapshot
        g = _sphere_grid(case, case["storage"], seed)
        g.step(TRT, use_les=True, smag_const=CS, n=2)
        s.update(g=g, out=[torch.empty(g.total_nodes(), dtype=torch.float32, device=DEV) for _ in range(4)])
        g.synchronize()
    return s


# ------------------------------------------------------------------ the call
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "channel2d":
        s["g"].step(case["coll"], gx=1e-5, n=case["steps"])
        s["g"].macroscopic_into(**s["out"])
        return s["out"]
    if k in ("cylinder2d", "duct"):
        s["g"].step(case["coll"], n=case["steps"])
        s["g"].macroscopic_into(**s["out"])
        return dict(s["out"], forces=s["g"].force_history().astype(np.float32), state=_state_view(s["g"]))
    if k == "sphere":
        g = s["g"]
        g.step(TRT, use_les=True, smag_const=CS, n=case["steps"])
        if "out" not in s:
            return {"state": _state_view(g)}
        g.macroscopic_into(**s["out"])
        got = dict(s["out"], forces=g.force_history().astype(np.float32))
        return got if case["storage"] == "f16c" else dict(got, state=_state_view(g))
    if k == "job":
        n = case["n"]
        (cx, cy, cz), r = _sphere_of(case)
        g = wb.LatticeGrid3D(n, n, n, TAU_SPHERE)
        g.initialize_fields(*s["fields"])
        g.set_periodic_axes(True, True)
        g.set_inflow_west(U_IN)
        g.set_outflow_east(1.0)
        g.set_solid_sphere(cx, cy, cz, r)
        g.build_curved_sphere_links(cx, cy, cz, r)
        g.enable_forces(cx, cy, cz, 2.0 * r, case["steps"])
        g.step(TRT, use_les=True, smag_const=CS, n=case["steps"])
        g.macroscopic_into(*s["out"])
        forces = g.force_history().astype(np.float32)
        g.close()
        return {"macro": s["out"], "forces": forces}
    if k == "tgv":
        s["g"].step(case["coll"], n=case["steps"])
        s["g"].macroscopic_into(**s["out"])
        return s["out"]
    if k == "batch":
        s["b"].step(case["steps"])
        forces = np.stack([g.force_history() for g in s["b"].members]).astype(np.float32)
        return {"state": [_state_view(g) for g in s["b"].members], "forces": forces}
    if k == "thermal":
        s["g"].step(TRT, use_les=True, smag_const=CS, n=case["steps"])
        s["g"].macroscopic_into(**s["out"])
        return dict(s["out"], T=s["g"].temperature_data())
    if k == "dropin":
        nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["nx"] * case["ny"] * case["nz"]
        p = wb.addr
        f, g, t, o, F, (cx, cy, cz) = p(s["f"]), p(s["g"]), p(s["t"]), [p(a) for a in s["out"].values()], p(s["F"]), s["c"]
        wb.lib.d3q19_collide_trt(f, g, t, *o[:4], 0.6, 3.0, 0.0, 0.0, 0.0, n)
        wb.lib.d3q19_stream_with_boundaries(g, f, t, nx, ny, nz, 0.0, 0.0, 0.0)
        wb.lib.d3q19_compute_macroscopic_moments(f, *o[:4], n)
        wb.lib.d3q19_compute_velocity_magnitude(*o[1:5], n)
        wb.lib.d3q19_compute_momentum_exchange_forces(f, t, nx, ny, nz, cx, cy, cz, 2.0 * s["r"], F, F + 4, F + 8)
        return dict(s["out"], f=s["f"], forces=s["F"])
    return wb.FieldAnalytics.compute_3d_features(s["g"], *s["out"])


# ------------------------------------------------------------------ what a pass cannot do without
_FLOPS = {(9, BGK): 130, (9, TRT): 130, (9, MRT): 150, (19, BGK): 300, (19, TRT): 250, (19, MRT): 450, (27, TRT): 350,
          (27, MRT): 500}


def work(case):
    k = case["kind"]
    q, e, coll = 9, 4, case.get("coll", TRT)
    steps, n, out = case.get("steps", 1), case.get("nx", 1) * case.get("ny", 1) * case.get("nz", 1), 16
    if k in ("sphere", "duct", "snapshot", "dropin", "job"):
        q, out = 19, 20
        n = case["n"] ** 3 if k == "job" else n
    if k == "tgv":
        q, n, out = case["q"], case["edge"] ** 3, 20
    if case.get("storage", "f32") != "f32":
        e = 2
    if k == "batch":  # sizes of the mean domain: nx uniform in 64 .. 512, ny = nx / 2
        n = case["members"] * 50000
    per = 2 * q * e + 1
    if k == "dropin":  # collide and stream apart, as the host program has them
        return {"bytes": n * (4 * q * 4 + 2 * q * 4 + 60), "flops": n * 450}
    if k == "snapshot":
        return {"bytes": n * (q * e + 16), "flops": n * 120}
    if k == "thermal":
        return {"bytes": n * (steps * (per + 40) + q * e + out + 8), "flops": n * steps * 180}
    read = 0 if k == "batch" or (k == "sphere" and case["storage"] in ("f16", "bf16")) else q * e + out
    return {"bytes": n * (steps * per + read + (16 if k == "job" else 0)), "flops": n * steps * _FLOPS[q, coll]}


# ------------------------------------------------------------------ the scheme in 64 bits
C9 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
C19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0), (1, -1, 0),
       (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)]
C27 = C19 + [(x, y, z) for z in (1, -1) for y in (1, -1) for x in (1, -1)]
CS_OF = {9: C9, 19: C19, 27: C27}
W_OF = {9: {0: 4 / 9, 1: 1 / 9, 2: 1 / 36}, 19: {0: 1 / 3, 1: 1 / 18, 2: 1 / 36},
        27: {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}}


def _lat(q):
    c = CS_OF[q]
    return c, [W_OF[q][sum(abs(v) for v in a)] for a in c], [c.index(tuple(-v for v in a)) for a in c]


def _dot(a, v):
    """a . v for a lattice direction a; None where a is at rest."""
    r = None
    for s, x in zip(a, v):
        if s:
            r = s * x if r is None else r + s * x
    return r


def _feq(q, m):
    c, w, _ = _lat(q)
    rho, u = m[0], m[1:4]
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    f = torch.empty((q,) + tuple(rho.shape), dtype=F64, device=rho.device)
    for i in range(q):
        cu = _dot(c[i], u)
        f[i] = w[i] * rho * ((1.0 - 1.5 * u2) if cu is None else (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * u2))
    return f


def _moments(q, f, g=(0.0, 0.0, 0.0)):
    c, _, _ = _lat(q)
    rho = f.sum(0)
    u = []
    for a in range(3):
        j = torch.zeros_like(rho)
        for i in range(q):
            if c[i][a]:
                j += c[i][a] * f[i]
        u.append(j / rho + 0.5 * g[a])
    return [rho] + u


def _basis19(k, a):
    x, y, z = a
    c2 = x * x + y * y + z * z
    return [1, 19 * c2 - 30, (21 * c2 * c2 - 53 * c2 + 24) / 2, x, (5 * c2 - 9) * x, y, (5 * c2 - 9) * y, z,
            (5 * c2 - 9) * z, 3 * x * x - c2, (3 * c2 - 5) * (3 * x * x - c2), y * y - z * z,
            (3 * c2 - 5) * (y * y - z * z), x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y,
            (y * y - x * x) * z][k]


def _mrt19(f, m, tau):
    M = torch.tensor([[_basis19(k, a) for a in C19] for k in range(19)], dtype=F64, device=f.device)
    inv = (M / (M * M).sum(1, keepdim=True)).T
    inv = torch.round(inv * 1e7) / 1e7  # the reference's seven-decimal table
    rho, ux, uy, uz = m
    u2 = ux * ux + uy * uy + uz * uz
    z = torch.zeros_like(rho)
    e9, e11 = rho * (2 * ux * ux - uy * uy - uz * uz), rho * (uy * uy - uz * uz)
    eq = [rho, rho * (-11 + 19 * u2), rho * (3 - 5.5 * u2), None, -2 / 3 * rho * ux, None, -2 / 3 * rho * uy, None,
          -2 / 3 * rho * uz, e9, -0.5 * e9, e11, -0.5 * e11, rho * ux * uy, rho * uy * uz, rho * ux * uz, z, z, z]
    s = [1, 1 / 1.19, 1.4, 0, 1.2, 0, 1.2, 0, 1.2, 1 / tau, 1.4, 1 / tau, 1.4, 1 / tau, 1 / tau, 1 / tau, 1.98, 1.98, 1.98]
    v = torch.einsum("kq,qn->kn", M, f)
    for k in range(19):
        if eq[k] is not None:
            v[k] -= s[k] * (v[k] - eq[k])
    return torch.einsum("qk,kn->qn", inv, v)


def _mrt27(f, m, tau):
    """Raw-moment relaxation: shear at 1 / tau, trace and all higher moments at 1."""
    pw = [(a, b, c) for c in range(3) for b in range(3) for a in range(3)]
    M = torch.tensor([[float(x ** a * y ** b * z ** c) for (x, y, z) in C27] for (a, b, c) in pw], dtype=F64)
    S = torch.zeros(27, 27, dtype=F64)
    for k, p in enumerate(pw):
        S[k, k] = 0.0 if sum(p) <= 1 else (1.0 if sum(p) > 2 else 1.0 / tau)
    d = [pw.index((2, 0, 0)), pw.index((0, 2, 0)), pw.index((0, 0, 2))]
    for i in d:
        for j in d:
            S[i, j] = (1.0 - 1.0 / tau) / 3.0 + (1.0 / tau if i == j else 0.0)
    K = torch.linalg.solve(M, S @ M).to(f.device)
    return f - torch.einsum("qk,kn->qn", K, f - _feq(27, m))


def _mrt9(f, m, tau, g):
    rho, ux, uy = m[:3]
    T = torch.tensor([[1] * 9, [-4, -1, -1, -1, -1, 2, 2, 2, 2], [4, -2, -2, -2, -2, 1, 1, 1, 1], [0, 1, 0, -1, 0, 1, -1, -1, 1],
                      [0, -2, 0, 2, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1], [0, 0, -2, 0, 2, 1, 1, -1, -1],
                      [0, 1, -1, 1, -1, 0, 0, 0, 0], [0, 0, 0, 0, 0, 1, -1, 1, -1]], dtype=F64, device=f.device)
    v = torch.einsum("kq,qn->kn", T, f)
    u2 = ux * ux + uy * uy
    Fx, Fy = rho * g[0], rho * g[1]
    uF = ux * Fx + uy * Fy
    p = 1 - 0.5 / tau
    eq = [rho, rho * (-2 + 3 * u2), rho * (1 - 3 * u2), None, -rho * ux, None, -rho * uy, rho * (ux * ux - uy * uy), rho * ux * uy]
    s = [0, 1 / 1.63, 1.4, 0, 1.6, 0, 1.6, 1 / tau, 1 / tau]
    add = [0, 6 * p * uF, -6 * p * uF, Fx, -p * Fx, Fy, -p * Fy, 2 * p * (ux * Fx - uy * Fy), p * (ux * Fy + uy * Fx)]
    for k in range(9):
        v[k] = v[k] - (0 if eq[k] is None else s[k] * (v[k] - eq[k])) + add[k]
    return torch.einsum("qk,kn->qn", torch.linalg.inv(T), v)


def _collide(q, f, coll, tau, cs, g=(0.0, 0.0, 0.0), tau_a=None):
    """Post-collision populations of f [q, n]; g may hold tensors (a force per node)."""
    c, w, opp = _lat(q)
    m = _moments(q, f, g)
    if coll == MRT:
        return _mrt9(f, m, tau, g) if q == 9 else (_mrt19(f, m, tau) if q == 19 else _mrt27(f, m, tau))
    e = _feq(q, m)
    ts = tau
    if cs:
        P = {}
        for i in range(1, q):
            for a in range(3):
                for b in range(a, 3):
                    if c[i][a] * c[i][b]:
                        P[a, b] = P.get((a, b), 0.0) + c[i][a] * c[i][b] * (f[i] - e[i])
        pi = sum((1.0 if a == b else 2.0) * v * v for (a, b), v in P.items())
        ts = 0.5 * (tau + torch.sqrt(tau * tau + 18.0 * math.sqrt(2.0) * cs * cs * torch.sqrt(2.0 * pi) / m[0]))
    if coll == BGK:
        os = oa = 1.0 / ts
    else:
        os = 1.0 / ts
        oa = 1.0 / tau_a if tau_a else 1.0 / (0.5 + 0.25 / (ts - 0.5))
    forced = any(isinstance(x, torch.Tensor) or x for x in g)
    r = torch.empty_like(f)
    for i in range(q):
        o = opp[i]
        d, b = f[i] - e[i], f[o] - e[o]
        r[i] = f[i] - 0.5 * os * (d + b) - 0.5 * oa * (d - b)
        if forced:
            ug = m[1] * g[0] + m[2] * g[1] + m[3] * g[2]
            cu, cg = _dot(c[i], m[1:]), _dot(c[i], g)
            r[i] += (1 - 0.5 * os) * w[i] * m[0] * (-3.0 * ug + (0.0 if cu is None else 9.0 * cu * cg))
            if cu is not None:
                r[i] += (1 - 0.5 * oa) * w[i] * m[0] * 3.0 * cg
    return r


class _Exact:
    """One lattice in 64 bits: g^k = Collide(f^k) between steps, like the resident grid."""

    def __init__(self, q, m, solid, coll, tau, cs=0.0, g=(0.0, 0.0, 0.0), periodic=False, faces=False, sphere=None,
                 mem=None, tau_a=None):
        self.q, self.coll, self.tau, self.cs, self.g, self.tau_a = q, coll, tau, cs, g, tau_a
        self.c, self.w, self.opp = _lat(q)
        self.shape, self.per, self.faces, self.mem = tuple(m[0].shape), periodic, faces, mem
        nz, ny, nx = self.shape
        self.solid = solid
        self.wall, self.link = {}, []
        for i in range(1, q):
            cx, cy, cz = self.c[i]
            s = torch.roll(solid, (cz, cy, cx), (0, 1, 2))
            out = torch.zeros_like(solid)
            if not periodic:
                if cy:
                    out[:, 0 if cy > 0 else -1, :] = True
                if cz and q != 9:
                    out[0 if cz > 0 else -1] = True
            self.wall[i] = (s | out) if bool(s.any()) or not periodic else None
            if mem is not None:  # links x -> x + c_i into a solid node, y and z in range whatever the wrap
                n = torch.roll(solid, (-cz, -cy, -cx), (0, 1, 2)) & ~solid
                if cy:
                    n[:, -1 if cy > 0 else 0, :] = False
                if cz:
                    n[-1 if cz > 0 else 0] = False
                if faces:
                    n[:, :, 0] = n[:, :, -1] = False
                zz, yy, xx = torch.nonzero(n, as_tuple=True)
                r = [(v.float() + 0.5 * a) - np.float32(o) for v, a, o in zip((xx, yy, zz), self.c[i], mem)]
                r2 = r[0] * r[0] + r[1] * r[1]
                if q != 9:
                    r2 = r2 + r[2] * r[2]
                near = r2 <= float(np.float32(mem[3]) * np.float32(mem[3]))
                self.link.append((i, zz[near], yy[near], xx[near], r[0][near].double(), r[1][near].double()))
        self.bfl = _links(solid.cpu().numpy(), *sphere) if sphere is not None else None
        self.gpop = self.hit(_feq(q, m))
        self.forces = []

    def hit(self, f):
        """Collide in slices of nodes; solid nodes keep their populations."""
        q, n = self.q, f[0].numel()
        flat, out = f.view(q, n), torch.empty_like(f).view(q, n)
        gg = [x.view(-1) if isinstance(x, torch.Tensor) else x for x in self.g]
        for a in range(0, n, 1 << 22):
            b = min(n, a + (1 << 22))
            gs = tuple(x[a:b] if isinstance(x, torch.Tensor) else x for x in gg)
            out[:, a:b] = _collide(q, flat[:, a:b], self.coll, self.tau, self.cs, gs, self.tau_a)
        out = out.view(f.shape)
        return torch.where(self.solid[None], f, out) if bool(self.solid.any()) else out

    def pull(self):
        g, f = self.gpop, torch.empty_like(self.gpop)
        f[0] = g[0]
        for i in range(1, self.q):
            cx, cy, cz = self.c[i]
            s = torch.roll(g[i], (cz, cy, cx), (0, 1, 2))
            f[i] = s if self.wall[i] is None else torch.where(self.wall[i], g[self.opp[i]], s)
        if self.bfl is not None:
            for i, (z, y, x, d) in self.bfl.items():
                cx, cy, cz = self.c[i]
                nz, ny, nx = self.shape
                fi, fo = g[i, z, y, x], g[self.opp[i], z, y, x]
                yf, zf = y - cy, z - cz
                inside = (yf >= 0) & (yf < ny) & (zf >= 0) & (zf < nz)
                ff = torch.where(inside, g[i, zf.clamp(0, nz - 1), yf.clamp(0, ny - 1), (x - cx) % nx], fi)
                f[self.opp[i], z, y, x] = torch.where(d < 0.5, 2 * d * fi + (1 - 2 * d) * ff, fi / (2 * d) + (1 - 1 / (2 * d)) * fo)
        if self.faces:
            self.zou_he(f)
        return torch.where(self.solid[None], g, f) if bool(self.solid.any()) else f

    def zou_he(self, f):
        ui, ro = U_IN, 1.0
        if self.q == 9:
            a = f[:, :, 1:-1, 0]
            rho = (a[0] + a[2] + a[4] + 2 * (a[3] + a[6] + a[7])) / (1 - ui)
            t = 0.5 * (a[2] - a[4])
            f[1, :, 1:-1, 0] = a[3] + 2 / 3 * rho * ui
            f[5, :, 1:-1, 0] = a[7] - t + rho * ui / 6
            f[8, :, 1:-1, 0] = a[6] + t + rho * ui / 6
            a = f[:, :, 1:-1, -1]
            ux = -1 + (a[0] + a[2] + a[4] + 2 * (a[1] + a[5] + a[8])) / ro
            t = 0.5 * (a[2] - a[4])
            f[3, :, 1:-1, -1] = a[1] - 2 / 3 * ro * ux
            f[6, :, 1:-1, -1] = a[8] - t - ro * ux / 6
            f[7, :, 1:-1, -1] = a[5] + t - ro * ux / 6
            return
        a = f[:, :, :, 0].clone()
        s0 = a[[0, 3, 4, 5, 6, 15, 16, 17, 18]].sum(0)
        rho = (s0 + 2 * a[[2, 8, 10, 12, 14]].sum(0)) / (1 - ui)
        ny = 0.5 * (a[3] + a[15] + a[17] - a[4] - a[16] - a[18])
        nz = 0.5 * (a[5] + a[15] + a[16] - a[6] - a[17] - a[18])
        f[1, :, :, 0] = a[2] + rho * ui / 3
        for i, o, t in ((7, 10, -ny), (9, 8, ny), (11, 14, -nz), (13, 12, nz)):
            f[i, :, :, 0] = a[o] + rho * ui / 6 + t
        a = f[:, :, :, -1].clone()
        s0 = a[[0, 3, 4, 5, 6, 15, 16, 17, 18]].sum(0)
        ux = -1 + (s0 + 2 * a[[1, 7, 9, 11, 13]].sum(0)) / ro
        ny = 0.5 * (a[3] + a[15] + a[17] - a[4] - a[16] - a[18])
        nz = 0.5 * (a[5] + a[15] + a[16] - a[6] - a[17] - a[18])
        f[2, :, :, -1] = a[1] - ro * ux / 3
        for i, o, t in ((10, 7, ny), (8, 9, -ny), (14, 11, nz), (12, 13, -nz)):
            f[i, :, :, -1] = a[o] - ro * ux / 6 + t

    def measure(self, f):
        F = [0.0, 0.0, 0.0]
        for i, z, y, x, rx, ry in self.link:
            v = 2.0 * f[i, z, y, x]
            c = self.c[i]
            F[0] += float(v.sum()) * c[0]
            F[1] += float(v.sum()) * c[1]
            F[2] += float((rx * v * c[1] - ry * v * c[0]).sum()) if self.q == 9 else float(v.sum()) * c[2]
        self.forces.append(F)

    def step(self, n):
        for _ in range(n):
            self.f = self.pull()
            if self.mem is not None:
                self.measure(self.f)
            self.gpop = self.hit(self.f)

    def macro(self):
        m = [v.reshape(-1) for v in _moments(self.q, self.f, self.g)]
        speed = torch.sqrt(m[1] ** 2 + m[2] ** 2 + m[3] ** 2)
        if self.q == 9:
            return {"rho": m[0], "ux": m[1], "uy": m[2], "speed": speed}
        return {"rho": m[0], "ux": m[1], "uy": m[2], "uz": m[3], "speed": speed}


def _links(solid, centre, r):
    """Curved links by direction: fluid nodes with a solid neighbour (x periodic, y and z in range) and the wall
    distance on the link, in the float32 arithmetic that defines it."""
    nz, ny, nx = solid.shape
    f = np.float32
    out = {}
    for i in range(1, 19):
        c = C19[i]
        n = np.roll(solid, (-c[2], -c[1], -c[0]), (0, 1, 2)) & ~solid
        if c[1]:
            n[:, -1 if c[1] > 0 else 0, :] = False
        if c[2]:
            n[-1 if c[2] > 0 else 0] = False
        z, y, x = np.nonzero(n)
        if not len(z):
            continue
        p = [v.astype(f) - f(o) for v, o in zip((x, y, z), centre)]
        a = f(sum(v * v for v in c))
        b = f(2.0) * ((p[0] * f(c[0]) + p[1] * f(c[1])) + p[2] * f(c[2]))
        cc = ((p[0] * p[0] + p[1] * p[1]) + p[2] * p[2]) - f(r) * f(r)
        disc = b * b - f(4.0) * a * cc
        with np.errstate(invalid="ignore"):
            t1, t2 = (-b - np.sqrt(disc)) / (f(2.0) * a), (-b + np.sqrt(disc)) / (f(2.0) * a)
            d = np.where((t1 >= 0) & (t1 <= 1), t1, np.where((t2 >= 0) & (t2 <= 1), t2, f(0.5)))
        d = np.clip(np.where(disc >= 0, d, f(0.5)), f(0.01), f(0.99))
        out[i] = tuple(torch.from_numpy(v.copy()).to(DEV) for v in (z, y, x, d.astype(np.float64)))
    return out


def _exact_sphere(case, seed, steps):
    n3 = (case["n"],) * 3 if case["kind"] == "job" else (case["nz"], case["ny"], case["nx"])
    c, r = _sphere_of(case)
    m = [a.double().view(n3) for a in _waves(n3, seed, U_IN, 0.02)]
    solid = torch.from_numpy(_sphere_mask(n3, c, r)).to(DEV)
    x = _Exact(19, m, solid, TRT, TAU_SPHERE, CS, periodic=True, faces=True, sphere=(c, r), mem=(*c, 2.0 * r))
    x.step(steps)
    return x


def _forces(x):
    return np.array(x.forces, dtype=np.float64)


def _h_of(x):
    w = torch.tensor(x.w, dtype=F64, device=DEV).view(-1, 1)
    return x.gpop.view(x.q, -1) / w - 1.0


def exact(case, seed):
    k = case["kind"]
    with torch.no_grad():
        if k in ("channel2d", "cylinder2d"):
            shape = (1, case["ny"], case["nx"])
            m = [a.double().view(shape) for a in _waves(shape, seed, U_IN, 0.02)]
            if k == "channel2d":
                solid = np.zeros(shape[1:], bool)
                solid[0, :] = solid[-1, :] = True
                x = _Exact(9, m, torch.from_numpy(solid)[None].to(DEV), case["coll"], 0.8, g=(float(np.float32(1e-5)), 0.0, 0.0))
                x.step(case["steps"])
                return x.macro()
            solid, mem = _cylinder(case)
            x = _Exact(9, m, torch.from_numpy(solid)[None].to(DEV), case["coll"], 0.56, faces=True, mem=mem)
            x.step(case["steps"])
            return dict(x.macro(), forces=_forces(x), state=x.gpop.view(9, -1))
        if k == "sphere":
            x = _exact_sphere(case, seed, case["steps"])
            if case["storage"] in ("f16", "bf16"):
                return {"state": _h_of(x)}
            got = dict(x.macro(), forces=_forces(x))
            return got if case["storage"] == "f16c" else dict(got, state=x.gpop.view(19, -1))
        if k == "job":
            x = _exact_sphere(case, seed, case["steps"])
            return {"macro": list(x.macro().values()), "forces": _forces(x)}
        if k == "duct":
            shape = (case["nz"], case["ny"], case["nx"])
            c, r = _sphere_of(case)
            m = [a.double().view(shape) for a in _waves(shape, seed, U_IN, 0.02)]
            x = _Exact(19, m, torch.from_numpy(_sphere_mask(shape, c, r)).to(DEV), case["coll"], 0.6, sphere=(c, r),
                       mem=(*c, 2.0 * r))
            x.step(case["steps"])
            return dict(x.macro(), forces=_forces(x), state=x.gpop.view(19, -1))
        if k == "tgv":
            shape = (case["edge"],) * 3
            m = [a.double().view(shape) for a in _waves(shape, seed, 0.0, 0.03)]
            x = _Exact(case["q"], m, torch.zeros(shape, dtype=torch.bool, device=DEV), case["coll"], 0.51, periodic=True)
            x.step(case["steps"])
            return x.macro()
        if k == "batch":
            state, forces = [], []
            for i, (nx, ny, chord, tau, solid) in enumerate(_ellipses(case)):
                m = [a.double().view(1, ny, nx) for a in _waves((1, ny, nx), seed + i, U_IN, 0.01)]
                if i >= 4:  # a few domains stand for all of them
                    state.append(None)
                    continue
                x = _Exact(9, m, torch.from_numpy(solid)[None].to(DEV), TRT, tau, CS, faces=True,
                           mem=(nx / 5.0, ny / 2.0, 0.0, 1.5 * chord))
                x.step(case["steps"])
                state.append(x.gpop.view(9, -1))
            return {"state": state, "forces": None}
        if k == "thermal":
            return _exact_thermal(case, seed)
        if k == "dropin":
            shape = (case["nz"], case["ny"], case["nx"])
            c, r = _sphere_of(case)
            f = _feq(19, [a.double().view(shape) for a in _waves(shape, seed, U_IN, 0.02)]).float().double()
            x = _Exact(19, [a.double().view(shape) for a in _waves(shape, seed, U_IN, 0.02)],
                       torch.from_numpy(_sphere_mask(shape, c, r)).to(DEV), TRT, 0.6, mem=(*c, 2.0 * r), tau_a=3.0)
            x.gpop = x.hit(f)
            x.f = x.pull()
            x.measure(x.f)
            return dict(x.macro(), f=x.f.view(19, -1), forces=np.array(x.forces[0]))
        x = _exact_sphere(case, seed, 2)
        u = [x.macro()[a].view(x.shape) for a in ("ux", "uy", "uz")]
        d = [[0.5 * (torch.roll(v, -1, 2 - a) - torch.roll(v, 1, 2 - a)) for a in range(3)] for v in u]  # d[i][j] = du_i/dx_j
        s2 = sum((0.5 * (d[i][j] + d[j][i])) ** 2 for i in range(3) for j in range(3))
        o2 = sum((0.5 * (d[i][j] - d[j][i])) ** 2 for i in range(3) for j in range(3))
        w = (d[2][1] - d[1][2], d[0][2] - d[2][0], d[1][0] - d[0][1], 0.5 * (o2 - s2))
        return tuple(v.reshape(-1) for v in w)


def _exact_thermal(case, seed):
    tau, tau_t, gbeta = _thermal_of(case)
    shape = (1, case["ny"], case["nx"])
    m = [a.double().view(shape) for a in _waves(shape, seed, 0.0, 0.02)]
    cd, wt = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1)], [1 / 3] + [1 / 6] * 4
    T0 = torch.from_numpy(_temperature(case, seed)).to(DEV).double().view(shape)
    t = torch.stack([w * T0 for w in wt])
    solid = torch.zeros(shape, dtype=torch.bool, device=DEV)
    f = _feq(9, m)
    x = _Exact(9, m, solid, TRT, tau, CS)
    for n in range(case["steps"] + 1):
        if n:
            f = x.pull()
            s = torch.empty_like(t)
            for i, (cx, cy) in enumerate(cd):
                s[i] = torch.roll(t[i], (cy, cx), (1, 2))
                if cy:
                    o, row, tw = (4, 0, 1.0) if cy > 0 else (2, -1, 0.0)
                    s[i, :, row] = -t[o, :, row] + 2 * wt[i] * tw
            t = s
        T = t.sum(0)
        x.g = (0.0, gbeta * (T - 0.5), 0.0)
        x.f = f
        mm = _moments(9, f, x.g)
        x.gpop = x.hit(f)
        for i, (cx, cy) in enumerate(cd):
            t[i] = t[i] - (t[i] - wt[i] * T * (1 + 3 * (cx * mm[1] + cy * mm[2]))) / tau_t
    return dict(x.macro(), T=T.reshape(-1))
