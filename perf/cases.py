"""The work a user of this framework has it do, as cases to be timed.

A case is a dict of plain values; its "op" says which public entry points it goes through:

  sim        a scene whose particles stay on the device (bnn_flip_device_particles): the
             program writes particles, takes four sub-steps (bnn_flip_step, the call of the
             headline benchmark) and reads the particles back in its own order
  boundary   the same inside a turning box container, moved before every sub-step
             (bnn_flip_set_boundaries)
  batch      scenes served on one GPU: admitted (bnn_batch_add_scene), advanced together
             (bnn_batch_step), read back and released
  neighbors  neighbour lists of a device point set (bnn_neighbors)
  cell_sort, cell_sort_noalloc, z_sort
             the stand-alone sorts of a device point set
  aniso      anisotropic kernels of a device point set (bnn_anisotropic_kernels)
  pcg        a 7-point system in host memory (bnn_pcg_solve_7pt)

Sizes are those of the tests, of the benchmark and of its serving workload (32 to 256 cells
per axis, 8 particles per cell, blocks of 0.2 to 0.6 of the domain per axis), odd and unequal
axes among them.  Particles start with a smooth random velocity field plus noise, so that the
pressure solve has a real divergence to remove.
"""
import ctypes as C
import math

import numpy as np
import torch

from banana_b200 import capi, scenes

SUBSTEPS = 4        # sub-steps of one pass of a sim / boundary case
FRAME = float(np.float32(1.0 / 30.0))
KIND = {"flip": 0, "apic": 1, "aflip": 2}


def listed():
    return [
        # a small scene, stepped interactively: launches and waits count
        {"name": "flip-64", "op": "sim", "nx": 64, "ny": 64, "nz": 64, "bx": 0.4, "by": 0.6, "bz": 0.4,
         "solver": "flip", "pcg": "fp32", "tol": 1e-6},
        # APIC on a ragged grid, the ordinary off-line scene
        {"name": "apic-121x77x95", "op": "sim", "nx": 121, "ny": 77, "nz": 95, "bx": 0.45, "by": 0.5, "bz": 0.35,
         "solver": "apic", "pcg": "fp32", "tol": 1e-6},
        # AFLIP with the refined pressure solve
        {"name": "aflip-96-refined", "op": "sim", "nx": 96, "ny": 96, "nz": 96, "bx": 0.4, "by": 0.6, "bz": 0.4,
         "solver": "aflip", "pcg": "refined", "tol": 1e-6},
        # FLIP with the FP64 pressure solve, unequal axes
        {"name": "flip-160x192x128-fp64", "op": "sim", "nx": 160, "ny": 192, "nz": 128, "bx": 0.4, "by": 0.6,
         "bz": 0.4, "solver": "flip", "pcg": "fp64", "tol": 1e-6},
        # the headline scene
        {"name": "flip-256", "op": "sim", "nx": 256, "ny": 256, "nz": 256, "bx": 0.4, "by": 0.6, "bz": 0.4,
         "solver": "flip", "pcg": "fp32", "tol": 1e-6},
        # a tank that turns: weighted pressure system, boundary grids rebuilt every sub-step
        {"name": "boundary-80", "op": "boundary", "nx": 80, "ny": 80, "nz": 80, "bx": 0.4, "by": 0.6, "bz": 0.4,
         "solver": "flip", "pcg": "fp32", "tol": 1e-6},
        # a serving batch: two dozen requests of the batch workload's sizes
        {"name": "batch-24", "op": "batch", "scenes": 24, "steps": 30, "specs": 11},
        # neighbour lists of a small and of the benchmark's point set
        {"name": "neighbors-20k", "op": "neighbors", "n": 20011, "r": 0.05, "blobs": 4},
        {"name": "neighbors-4m", "op": "neighbors", "n": 4000000, "r": 0.01, "blobs": 16},
        # binning of a particle set onto a 128-cell grid
        {"name": "cell-sort-1m", "op": "cell_sort", "n": 999983, "g": 128, "blobs": 16},
        # surface reconstruction input of a medium scene
        {"name": "aniso-200k", "op": "aniso", "n": 200003, "bx": 0.4, "by": 0.6, "bz": 0.4},
        # a pressure system handed over from host code
        {"name": "pcg-152k", "op": "pcg", "nx": 51, "ny": 77, "nz": 51, "mode": "fp32", "tol": 1e-6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["sim", "sim", "sim", "boundary", "batch", "neighbors", "neighbors", "cell_sort",
                     "cell_sort_noalloc", "z_sort", "aniso", "pcg"])
    if op in ("sim", "boundary"):
        solver = rng.choice(["flip", "flip", "apic", "aflip"])
        pcg = rng.choice(["fp32", "fp32", "refined", "fp64"])
        top = 128 if op == "boundary" else 256 if (solver, pcg) == ("flip", "fp32") else 160
        n = [_log_int(rng, 32, top) for _ in range(3)]
        b = [round(rng.uniform(0.2, 0.6), 3) for _ in range(3)]
        # at most the share of the domain that the largest listed scene fills
        while b[0] * b[1] * b[2] > 0.09:
            b = [round(max(0.2, 0.95 * x), 3) for x in b]
        return {"op": op, "nx": n[0], "ny": n[1], "nz": n[2], "bx": b[0], "by": b[1], "bz": b[2], "solver": solver,
                "pcg": pcg, "tol": 1e-6}
    if op == "batch":
        return {"op": op, "scenes": rng.randint(3, 24), "steps": rng.randint(5, 30), "specs": rng.randint(1, 10 ** 6)}
    if op == "neighbors":
        n = _log_int(rng, 1000, 2000000)
        # the radius that gives a uniform half of the points 5 to 60 neighbours each
        r = (rng.uniform(5.0, 60.0) / (0.5 * n * 4.19)) ** (1.0 / 3.0)
        blobs = rng.randint(4, 64)
        # a denser half makes the lists long: keep them below the largest listed case's
        r = min(r, (80.0 * 3.4e-4 * blobs / (0.5 * n * 4.19)) ** (1.0 / 3.0) * 4.0, 0.1)
        return {"op": op, "n": n, "r": round(r, 5), "blobs": blobs}
    if op == "cell_sort":
        return {"op": op, "n": _log_int(rng, 1000, 4000000), "g": _log_int(rng, 16, 256), "blobs": rng.randint(2, 32)}
    if op == "cell_sort_noalloc":
        return {"op": op, "n": _log_int(rng, 1000, 1048576), "g": _log_int(rng, 16, 128), "blobs": rng.randint(2, 32)}
    if op == "z_sort":
        return {"op": op, "n": _log_int(rng, 1000, 4000000), "r": round(rng.uniform(0.005, 0.05), 5),
                "blobs": rng.randint(2, 32)}
    if op == "aniso":
        return {"op": op, "n": _log_int(rng, 1000, 1000000), "bx": round(rng.uniform(0.2, 0.6), 3),
                "by": round(rng.uniform(0.2, 0.6), 3), "bz": round(rng.uniform(0.2, 0.6), 3)}
    return {"op": "pcg", "nx": _log_int(rng, 16, 90), "ny": _log_int(rng, 16, 90), "nz": _log_int(rng, 16, 90),
            "mode": rng.choice(["fp32", "fp32", "refined", "fp64"]), "tol": 1e-6}


# ---- inputs -----------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _cell_size(case):
    return float(np.float32(1.0 / max(case["nx"], case["ny"], case["nz"])))


def _block(res, frac, dx, g, ppc=8):
    """`ppc` particles uniform in every cell of the block at the origin, cell by cell (n x 3),
    and their velocities: three random waves per component and 5% noise."""
    cells = [max(1, int(math.floor(f * r + 1e-9))) for f, r in zip(frac, res)]
    k, j, i = torch.meshgrid(*(torch.arange(c, device="cuda") for c in cells[::-1]), indexing="ij")
    cell = torch.stack([i, j, k], -1).reshape(-1, 1, 3).float()
    pos = ((cell + 0.998 * _rand(g, cell.shape[0], ppc, 3) + 0.001) * dx).reshape(-1, 3).contiguous()
    wave = (_rand(g, 3, 3, 3) * 2 - 1) * 12.0
    amp = 0.25 * _randn(g, 3, 3)
    phase = 6.28 * _rand(g, 3, 3)
    vel = 0.02 * _randn(g, *pos.shape)
    for d in range(3):
        for q in range(3):
            vel[:, d] += amp[d, q] * torch.sin(pos @ wave[d, q] + phase[d, q])
    return pos, vel.contiguous()


def _params(case):
    dx = _cell_size(case)
    ext = tuple(float(np.float32(case[a] * dx)) for a in ("nx", "ny", "nz"))
    return scenes.dam_break_params(64, cell_size=dx, box_max=ext, solver_kind=KIND[case["solver"]],
                                   pcg_mode=capi.PCG_MODE[case["pcg"]], cg_relative_tolerance=case["tol"],
                                   refine_tolerance=case["tol"], refine_inner_tolerance=1e-3)


def _scene(case, seed):
    return _block((case["nx"], case["ny"], case["nz"]), (case["bx"], case["by"], case["bz"]), _cell_size(case),
                  _gen(seed))


class _DeviceArray:
    """A device pointer of the library as an array that torch can view."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _device_particles(s):
    """The scene's particle arrays where they are now: (6, n) values and (n) ids."""
    p6 = C.POINTER(C.c_float)()
    ids = C.POINTER(C.c_uint32)()
    capi.check(s["solver"].L.bnn_flip_device_particles(s["solver"].h, C.byref(p6), C.byref(ids)),
               "bnn_flip_device_particles")
    n, stride = s["n"], (s["n"] + 63) // 64 * 64
    a = torch.as_tensor(_DeviceArray(C.cast(p6, C.c_void_p).value, (6, stride), "<f4"), device="cuda")
    b = torch.as_tensor(_DeviceArray(C.cast(ids, C.c_void_p).value, (n,), "<i4"), device="cuda")
    return a[:, :n], b


def _points(case, seed):
    """Half uniform in the unit cube, half in Gaussian blobs of deviation 0.03 (the
    benchmark's point set), clamped to the cube."""
    g = _gen(seed)
    n = case["n"]
    half = n // 2
    centre = 0.1 + 0.8 * _rand(g, case["blobs"], 3)
    which = torch.arange(n - half, device="cuda") % case["blobs"]
    pts = torch.cat([_rand(g, half, 3), centre[which] + 0.03 * _randn(g, n - half, 3)])
    return pts.clamp_(0.0, 0.999999).contiguous()


def _aniso_points(case, seed):
    """About n particles of a fluid block, 8 per cell, and their radius (half a cell)."""
    b = (case["bx"], case["by"], case["bz"])
    res = (case["n"] / 8.0 / (b[0] * b[1] * b[2])) ** (1.0 / 3.0)
    dx = 1.0 / res
    g = _gen(seed)
    per = [max(1, round(f * res)) for f in b]
    full = per[0] * per[1] * per[2]
    cell = torch.arange(case["n"], device="cuda") % full
    idx = torch.stack([cell % per[0], cell // per[0] % per[1], cell // (per[0] * per[1])], -1)
    pts = (idx + _rand(g, case["n"], 3)) * dx
    return pts.float().contiguous(), float(np.float32(0.5 * dx))


def _system(case, seed):
    """A pressure system as the step assembles it: the cells below a wavy surface of a
    box, in cell order, with the ghost-fluid terms of the free surface on the diagonal."""
    g = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dt = 0.004
    x = torch.linspace(0, 1, nx, device="cuda")
    z = torch.linspace(0, 1, nz, device="cuda")
    h = ny * (0.8 + 0.1 * torch.sin(5 * x[None, :]) * torch.cos(4 * z[:, None])
              + 0.04 * torch.sin(17 * x[None, :] + 13 * z[:, None]))
    y = torch.arange(ny, device="cuda")
    act = y[None, :, None] < h[:, None, :]              # (nz, ny, nx)
    row = (torch.cumsum(act.reshape(-1).long(), 0) - 1).reshape(act.shape)
    row = torch.where(act, row, torch.full_like(row, -1))
    pad = torch.nn.functional.pad(row, (1, 1, 1, 1, 1, 1), value=-1)
    c = pad[1:-1, 1:-1, 1:-1]
    nb = torch.stack([pad[:-2, 1:-1, 1:-1], pad[1:-1, :-2, 1:-1], pad[1:-1, 1:-1, :-2], pad[1:-1, 1:-1, 2:],
                      pad[1:-1, 2:, 1:-1], pad[2:, 1:-1, 1:-1]], -1)[c >= 0]
    theta = 0.01 + 0.99 * _rand(g, nb.shape[0], 6)
    one = torch.ones_like(theta)
    diag = torch.where(nb >= 0, one, one / theta).sum(1) * dt
    rhs = _randn(g, nb.shape[0]) * 0.1
    return (diag.float().cpu().numpy(), nb.int().cpu().numpy(), -dt, rhs.float().cpu().numpy())


def _batch_scenes(case, seed):
    g = _gen(seed)
    out = []
    for spec in scenes.batch_scene_specs(case["scenes"], seed=case["specs"]):
        cfg = scenes.dam_break_params(64, box_max=tuple(r / 64.0 for r in spec["res"]), pcg_mode=2,
                                      refine_tolerance=1e-6, refine_inner_tolerance=1e-3)
        pos, vel = _block(spec["res"], spec["block_frac"], 1.0 / 64.0, g)
        out.append((cfg, pos.cpu().numpy(), vel.cpu().numpy()))
    return out


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "case": case}
    if op in ("sim", "boundary"):
        pos, vel = _scene(case, seed)
        s["solver"] = capi.FlipSolver(_params(case))
        s["solver"].set_particles(pos.cpu().numpy(), vel.cpu().numpy())
        s["n"] = len(pos)
        s["p6"] = torch.cat([pos, vel], 1).t().contiguous()
        s["ids"] = torch.arange(len(pos), device="cuda", dtype=torch.int32)
        s["stream"] = torch.cuda.ExternalStream(s["solver"].stream_ptr())
    elif op == "batch":
        s["scenes"] = _batch_scenes(case, seed)
        s["batch"] = capi.FlipBatch()
    elif op == "pcg":
        s["system"] = _system(case, seed)
    elif op == "aniso":
        s["pos"], radius = _aniso_points(case, seed)
        s["prm"] = capi.aniso_params(radius)
        s["cen"] = torch.empty(case["n"], 3, device="cuda")
        s["mat"] = torch.empty(case["n"], 9, device="cuda")
    else:
        s["pos"] = _points(case, seed)
        n = case["n"]
        new = lambda k, t=torch.int32: torch.empty(k, device="cuda", dtype=t)  # noqa: E731
        if op == "neighbors":
            # room for twice the expected entries; what a pass does not write stays 0
            s["off"] = new(n + 1, torch.int64)
            s["idx"] = torch.zeros(int(2 * _entries(case)) + 64 * n, device="cuda", dtype=torch.int32)
        elif op == "z_sort":
            s["z"], s["perm"] = new(n, torch.int64), new(n)
        else:
            s["cid"], s["order"], s["start"] = new(n), new(n), new(case["g"] ** 3 + 1)
    torch.cuda.synchronize()
    return s


# ---- one pass ---------------------------------------------------------------------------


def _container(k):
    return capi.boundary_object("box", (-0.55, -0.55, -0.55), (0.55, 0.55, 0.55), translation=(0.5, 0.5, 0.5),
                                axis_angle=(0.0, 0.0, 1.0, math.radians(2.0 * k)), dynamic=True)


def _run_sim(s):
    with torch.cuda.stream(s["stream"]):
        p6, ids = _device_particles(s)
        p6.copy_(s["p6"])
        ids.copy_(s["ids"])
        for k in range(SUBSTEPS):
            if s["op"] == "boundary":
                s["solver"].set_boundaries([_container(k)])
            s["solver"].step()
        p6, ids = _device_particles(s)
        out = torch.empty_like(s["p6"])
        out.index_copy_(1, ids.long(), p6)
    return out[:3], out[3:]


def _run_batch(s):
    b = s["batch"]
    sids = [b.add_scene(cfg, pos, vel) for cfg, pos, vel in s["scenes"]]
    for _ in range(s["case"]["steps"]):
        b.step()
    out = []
    for sid in sids:
        out += b.get_scene(sid)
        b.remove_scene(sid)
    return out


def run(s):
    op, case = s["op"], s["case"]
    if op in ("sim", "boundary"):
        return _run_sim(s)
    if op == "batch":
        return _run_batch(s)
    if op == "pcg":
        diag, nbr, off, rhs = s["system"]
        x, _ = capi.pcg_solve_7pt(diag, nbr, off, rhs, case["tol"], 5000, case["mode"])
        return x
    stream = torch.cuda.current_stream().cuda_stream
    n = case["n"]
    if op == "aniso":
        capi.anisotropic_kernels_dev(s["pos"].data_ptr(), n, s["prm"], s["cen"].data_ptr(), s["mat"].data_ptr(), stream)
        return s["cen"], s["mat"]
    lib = capi.load()
    if op == "neighbors":
        total = C.c_uint64()
        capi.check(lib.bnn_neighbors(s["pos"].data_ptr(), n, case["r"], s["off"].data_ptr(), s["idx"].data_ptr(),
                                     s["idx"].numel(), C.byref(total), stream), "bnn_neighbors")
        return s["off"], s["idx"], int(total.value)
    if op == "z_sort":
        capi.check(lib.bnn_z_sort(s["pos"].data_ptr(), n, case["r"], s["z"].data_ptr(), s["perm"].data_ptr(), stream),
                   "bnn_z_sort")
        return s["z"], s["perm"]
    bmin = (C.c_float * 3)(0.0, 0.0, 0.0)
    nc = (C.c_int32 * 3)(case["g"], case["g"], case["g"])
    oor = C.c_uint32()
    call = lib.bnn_cell_sort if op == "cell_sort" else lib.bnn_cell_sort_noalloc
    capi.check(call(s["pos"].data_ptr(), n, bmin, 1.0 / case["g"], nc, s["cid"].data_ptr(), s["order"].data_ptr(),
                    s["start"].data_ptr(), C.byref(oor), stream), "bnn_" + op)
    return s["cid"], s["order"], s["start"], int(oor.value)


# ---- what one pass cannot do without ----------------------------------------------------


def _step_bytes(res, frac, ppc=8, vec=4):
    """Bytes of one sub-step: particles read and written by the sort (72 each), read by the
    particle-to-grid transfer and the fluid distance (36), read and written by the
    grid-to-particle transfer (48); face arrays through the transfer, two extrapolations and
    the projection (46 a face in all); 24 a cell; and for each pressure row 13 vector
    elements an iteration, about 1.2 iterations per cell of the longest axis."""
    cells = 1
    for r in res:
        cells *= r + 4
    rows = 1
    for r, f in zip(res, frac):
        rows *= max(1, int(f * r + 1e-9))
    return 156 * rows * ppc + 46 * 3 * cells + 24 * cells + 28 * rows + 13 * vec * rows * 1.2 * max(res)


def _entries(case):
    """Expected entries of a neighbour search: pairs inside the uniform half and inside the
    blobs (mean density of a Gaussian)."""
    n = case["n"]
    dens = 0.5 * n + 0.25 * n / (case["blobs"] * (4 * math.pi * 0.03 ** 2) ** 1.5)
    return n * min(float(n), dens * 4.19 * case["r"] ** 3)


def work(case):
    op = case["op"]
    if op in ("sim", "boundary"):
        res = (case["nx"], case["ny"], case["nz"])
        vec = 8 if case["pcg"] == "fp64" else 4
        b = SUBSTEPS * _step_bytes(res, (case["bx"], case["by"], case["bz"]), vec=vec)
        return {"bytes": b, "flops": 0.5 * b}  # about two operations for each 4-byte element
    if op == "batch":
        b = sum(_step_bytes(q["res"], q["block_frac"]) for q in scenes.batch_scene_specs(case["scenes"], case["specs"]))
        return {"bytes": case["steps"] * b, "flops": case["steps"] * 0.5 * b}
    n = case.get("n", 0)
    if op == "neighbors":
        entries = _entries(case)
        return {"bytes": 12 * n + 8 * (n + 1) + 4 * entries, "flops": 8 * 6.4 * entries}
    if op in ("cell_sort", "cell_sort_noalloc"):
        return {"bytes": 12 * n + 8 * n + 4 * case["g"] ** 3, "flops": 6 * n}
    if op == "z_sort":
        return {"bytes": 12 * n + 12 * n, "flops": 6 * n}
    if op == "aniso":
        # 8 particles a cell in a sphere of 4 cells: about 2140 neighbours, twice
        return {"bytes": 12 * n + 48 * n, "flops": n * min(n, 2140) * 46}
    rows = 0.8 * case["nx"] * case["ny"] * case["nz"]
    vec = 8 if case["mode"] == "fp64" else 4
    it = 2.0 * max(case["nx"], case["ny"], case["nz"])
    return {"bytes": rows * (32 + 8 + 13 * vec * it), "flops": rows * 30 * it}


# ---- the same results in 64 bits --------------------------------------------------------


def _bary(x, size):
    s = torch.floor(x)
    i = s.long()
    f = x - s
    f = torch.where(i < 0, torch.zeros_like(f), torch.where(i > size - 2, torch.ones_like(f), f))
    return i.clamp(0, size - 2), f


class _Exact:
    """The sub-step on the padded grid in 64 bits; arrays are (z, y, x)."""

    def __init__(self, case, pos, vel):
        f32 = np.float32
        dx32 = f32(_cell_size(case))
        ext = [f32(case[a] * _cell_size(case)) for a in ("nx", "ny", "nz")]
        pad = dx32 * f32(2)
        self.G = [int(np.ceil((e + pad - (f32(0) - pad)) / dx32)) for e in ext]
        self.dx, self.bmin = float(dx32), -float(pad)
        self.hi = torch.tensor([float(e) for e in ext], device="cuda", dtype=torch.float64)
        self.kind = case["solver"]
        self.x, self.v = pos.double(), vel.double()
        self.shape = [[self.G[a] + (a == d) for a in (2, 1, 0)] for d in range(3)]
        z = lambda d: torch.zeros(self.shape[d], device="cuda", dtype=torch.float64)  # noqa: E731
        self.u = [z(d) for d in range(3)]
        self.c = torch.zeros(len(pos), 3, 3, device="cuda", dtype=torch.float64)
        self.time = FRAME

    def stencil(self, x, d):
        """Flat indexes and per-axis (index, fraction) of the 8 faces around x."""
        g = (x - self.bmin) / self.dx
        ax = [_bary(g[:, a] - (0.0 if a == d else 0.5), self.G[a] + (a == d)) for a in range(3)]
        sz, sy, sx = self.shape[d]
        for q in range(8):
            o = (q & 1, q >> 1 & 1, q >> 2)
            idx = ((ax[2][0] + o[2]) * sy + ax[1][0] + o[1]) * sx + ax[0][0] + o[0]
            w = [ax[a][1] if o[a] else 1.0 - ax[a][1] for a in range(3)]
            yield o, idx, w, [ax[a][0] + o[a] for a in range(3)]

    def sample(self, arr, x, d):
        return sum(w[0] * w[1] * w[2] * arr.reshape(-1)[idx] for _, idx, w, _ in self.stencil(x, d))

    def gradient(self, arr, x, d):
        out = torch.zeros_like(x)
        for o, idx, w, _ in self.stencil(x, d):
            val = arr.reshape(-1)[idx] / self.dx
            out[:, 0] += (1 if o[0] else -1) * w[1] * w[2] * val
            out[:, 1] += (1 if o[1] else -1) * w[0] * w[2] * val
            out[:, 2] += (1 if o[2] else -1) * w[0] * w[1] * val
        return out

    def velocity(self, x):
        return torch.stack([self.sample(self.u[d], x, d) for d in range(3)], 1)

    def box(self, x):
        near = torch.minimum(x, self.hi - x).amin(1)
        far = (x - torch.minimum(x.clamp(min=0.0), self.hi)).norm(dim=1)
        return torch.where(near >= 0, near, -far)

    def constrain(self, x):
        phi = self.box(x)
        at = torch.nonzero(phi < 0).flatten()
        if len(at):
            e, y = 1e-4, x[at]
            grad = torch.zeros_like(y)
            for q in range(8):
                o = torch.tensor([1.0 if q >> a & 1 else -1.0 for a in range(3)], device="cuda", dtype=torch.float64)
                grad += o * self.box(y + e * o)[:, None]
            length = grad.norm(dim=1, keepdim=True)
            x[at] = torch.where(length > 0, y - phi[at, None] * grad / length.clamp(min=1e-300), y)
        return x

    def extrapolate(self, arr, valid):
        for _ in range(4):
            total, count = torch.zeros_like(arr), torch.zeros_like(arr)
            va = valid.double()
            for d in range(3):
                for s in (1, -1):
                    total += torch.roll(arr * va, s, d)
                    count += torch.roll(va, s, d)
            inner = torch.zeros_like(valid)
            inner[1:-1, 1:-1, 1:-1] = True
            new = ~valid & inner & (count > 0)
            arr = torch.where(new, total / count.clamp(min=1.0), arr)
            valid = valid | new
        return arr

    def step(self, mode_tol):
        if self.time >= FRAME:
            self.time = 0.0
        top = max(float(a.abs().max()) for a in self.u)
        dt = min(max(self.dx / top, 1e-6), FRAME) if top > 1.2e-38 else FRAME
        left = FRAME - self.time
        dt = left if self.time + dt >= FRAME else 0.5 * left if self.time + 1.5 * dt >= FRAME else dt
        x = self.x
        mid = x + 0.5 * dt * self.velocity(x)
        x = self.x = self.constrain(x + dt * self.velocity(mid))
        G = self.G
        old = []
        for d in range(3):
            num = torch.zeros(self.shape[d], device="cuda", dtype=torch.float64).reshape(-1)
            den = torch.zeros_like(num)
            for _, idx, w, ijk in self.stencil(x, d):
                ww = w[0] * w[1] * w[2]
                val = self.v[:, d]
                if self.kind != "flip":
                    face = torch.stack([ijk[a] + (0.0 if a == d else 0.5) for a in range(3)], 1) * self.dx + self.bmin
                    val = val + (self.c[:, d] * (face - x)).sum(1)
                num.index_add_(0, idx, ww * val)
                den.index_add_(0, idx, ww)
            valid = (den > 1.2e-38).reshape(self.shape[d])
            a = torch.where(valid, (num / den.clamp(min=1e-300)).reshape(self.shape[d]), num.reshape(self.shape[d]))
            self.u[d] = self.extrapolate(a, valid) if self.kind != "apic" else a
            old.append(self.u[d].clone())
        self.u[1] = self.u[1] - 9.81 * dt
        # fluid distance: the nearest particle within the 27 cells around a cell
        phi = torch.full((G[2] * G[1] * G[0],), 3.0 * self.dx, device="cuda", dtype=torch.float64)
        cell = [((x[:, a] - self.bmin) / self.dx).long().clamp(0, G[a] - 1) for a in range(3)]
        radius = self.dx * 1.01 * math.sqrt(3.0) / 2.0
        for q in range(27):
            at = [cell[a] + (q // 3 ** a) % 3 - 1 for a in range(3)]
            ok = (at[0] >= 0) & (at[0] < G[0]) & (at[1] >= 0) & (at[1] < G[1]) & (at[2] >= 0) & (at[2] < G[2])
            c = torch.stack([at[a].double() + 0.5 for a in range(3)], 1) * self.dx + self.bmin
            dist = (c - x).norm(dim=1) - radius
            idx = (at[2] * G[1] + at[1]) * G[0] + at[0]
            phi.scatter_reduce_(0, idx[ok], dist[ok], "amin")
        phi = phi.reshape(G[2], G[1], G[0])
        fluid = phi < 0
        rows = torch.nonzero(fluid.reshape(-1)).flatten()
        number = torch.full((phi.numel(),), -1, device="cuda", dtype=torch.long)
        number[rows] = torch.arange(len(rows), device="cuda")
        i, j, k = rows % G[0], rows // G[0] % G[1], rows // (G[0] * G[1])
        rhs = (self.u[0][k, j, i] - self.u[0][k, j, i + 1] + self.u[1][k, j, i] - self.u[1][k, j + 1, i]
               + self.u[2][k, j, i] - self.u[2][k + 1, j, i])
        flat, diag, nbr = phi.reshape(-1), torch.zeros_like(rhs), []
        theta = lambda a, b: torch.where(  # noqa: E731
            (a < 0) & (b < 0), torch.ones_like(a),
            torch.where(a < 0, a / (a - b), torch.where(b < 0, b / (b - a), torch.zeros_like(a)))).clamp(min=0.01)
        for off in (-G[0] * G[1], -G[0], -1, 1, G[0], G[0] * G[1]):
            other = flat[rows + off]
            diag += torch.where(other < 0, torch.full_like(diag, dt), dt / theta(flat[rows], other))
            nbr.append(torch.where(other < 0, number[rows + off], torch.full_like(rows, -1)))
        p = _cg(diag, torch.stack(nbr, 1), -dt, rhs, mode_tol)
        press = torch.zeros_like(flat)
        press[rows] = p
        press = press.reshape(phi.shape)
        for d in range(3):
            a = 2 - d
            n = G[d]
            lo, hi = phi.narrow(a, 0, n - 1), phi.narrow(a, 1, n - 1)
            keep = (lo < 0) | (hi < 0)
            inner = self.u[d].narrow(a, 1, n - 1)
            new = torch.where(keep, inner - dt * (press.narrow(a, 1, n - 1) - press.narrow(a, 0, n - 1)) / theta(lo, hi),
                              torch.zeros_like(inner))
            u, valid = torch.zeros_like(self.u[d]), torch.zeros(self.shape[d], device="cuda", dtype=torch.bool)
            u.narrow(a, 1, n - 1).copy_(new)
            valid.narrow(a, 1, n - 1).copy_(keep)
            self.u[d] = self.extrapolate(u, valid)
        got = self.velocity(x)
        if self.kind == "apic":
            self.v = got
            self.c = torch.stack([self.gradient(self.u[d], x, d) for d in range(3)], 1)
        else:
            ratio = float(np.float32(0.97))
            diff = [self.u[d] - old[d] for d in range(3)]
            change = torch.stack([self.sample(diff[d], x, d) for d in range(3)], 1)
            self.v = (1.0 - ratio) * got + ratio * (self.v + change)
            if self.kind == "aflip":
                grad = torch.stack([self.gradient(self.u[d], x, d) for d in range(3)], 1)
                dgrad = torch.stack([self.gradient(diff[d], x, d) for d in range(3)], 1)
                self.c = (1.0 - ratio) * grad + ratio * (self.c + dgrad)
        self.time += dt


def _cg(diag, nbr, off, rhs, tol):
    """Jacobi CG in 64 bits on the compact rows, to a residual far below the framework's."""
    zero = torch.zeros(1, device=rhs.device, dtype=rhs.dtype)
    at = torch.where(nbr >= 0, nbr, torch.full_like(nbr, len(rhs)))

    def mul(s):
        t = torch.cat([s, zero])
        return diag * s + off * t[at].sum(1)

    x, r = torch.zeros_like(rhs), rhs.clone()
    z = r / diag
    s, rho = z.clone(), torch.dot(z, r)
    stop = float(r.abs().max()) * tol
    for it in range(20000):
        q = mul(s)
        alpha = rho / torch.dot(s, q)
        x += alpha * s
        r -= alpha * q
        if it % 32 == 31 and float(r.abs().max()) <= stop:
            break
        z = r / diag
        new = torch.dot(z, r)
        s = z + new / rho * s
        rho = new
    return x


def _exact_aniso(case, seed):
    pts, radius = _aniso_points(case, seed)
    p = pts.double()
    n = len(p)
    r = 8.0 * float(np.float32(radius))
    cen = torch.empty(n, 3, device="cuda", dtype=torch.float64)
    mat = torch.empty(n, 9, device="cuda", dtype=torch.float64)
    for b in range(0, n, 512):
        a = p[b:b + 512]
        d2 = ((a[:, None] - p[None]) ** 2).sum(-1)
        hit = d2 < r * r
        hit[torch.arange(len(a)), torch.arange(b, b + len(a))] = False
        w = torch.where(hit, 1.0 - (d2.sqrt() / r) ** 3, torch.zeros_like(d2))
        m = (a + w @ p) / (1.0 + w.sum(1, keepdim=True))
        cen[b:b + 512] = 0.5 * a + 0.5 * m
        e2 = ((m[:, None] - p[None]) ** 2).sum(-1)
        w = torch.where(hit & (e2 < r * r), 1.0 - (e2.sqrt() / r) ** 3, torch.zeros_like(d2))
        tot, first = w.sum(1), w @ p
        second = (w @ (p[:, :, None] * p[:, None, :]).reshape(n, 9)).reshape(-1, 3, 3)
        cov = (second - m[:, :, None] * first[:, None, :] - first[:, :, None] * m[:, None, :]
               + tot[:, None, None] * m[:, :, None] * m[:, None, :]) / (1.0 + tot)[:, None, None]
        lam, vec = torch.linalg.eigh(cov)
        lam = torch.maximum(lam, lam[:, 2:] / 8.0)
        lam = lam / lam.prod(1, keepdim=True).abs().clamp(min=1e-300) ** (1.0 / 3.0)
        out = (vec * lam[:, None, :]) @ vec.transpose(1, 2)
        spray = 0.75 * torch.eye(3, device="cuda", dtype=torch.float64).expand_as(out)
        out = torch.where((hit.sum(1) >= 25)[:, None, None], out, spray)
        mat[b:b + 512] = out.reshape(-1, 9)
    return cen, mat


def exact(case, seed):
    op = case["op"]
    if op == "pcg":
        diag, nbr, off, rhs = (torch.as_tensor(a, device="cuda") if isinstance(a, np.ndarray) else a
                               for a in _system(case, seed))
        off = float(np.float32(off))
        return _cg(diag.double(), nbr.long(), off, rhs.double(), 1e-12)
    if op == "aniso":
        return _exact_aniso(case, seed) if case["n"] <= 250000 else None
    if op == "sim":
        pos, vel = _scene(case, seed)
        e = _Exact(case, pos, vel)
        for _ in range(SUBSTEPS):
            e.step(1e-9)
        return e.x.t().contiguous(), e.v.t().contiguous()
    # sorts and lists are whole numbers; the turning container and the batch have no short
    # restatement that takes under 20 seconds
    return None
