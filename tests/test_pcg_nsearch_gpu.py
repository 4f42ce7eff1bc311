"""Standalone PCG, cell sort, z-sort and neighbour search through the C ABI, against the
oracle (restatements of PCGSolver.cpp, Grid.cpp and NeighborSearch.cpp)."""
import ctypes as C

import numpy as np
import pytest
import torch

from banana_b200 import scenes

pytestmark = pytest.mark.gpu


def _system(oracle_mod, n=32, steps=3):
    cfg = scenes.dam_break_params(n)
    pos, vel = scenes.dam_break(n)
    o = oracle_mod.Oracle(cfg)
    o.set_particles(pos, vel)
    for _ in range(steps):
        o.step()
    rs, ci, va, rhs = o.system()
    nrow = len(rhs)
    diag = np.zeros(nrow, np.float32)
    nbr = -np.ones((nrow, 6), np.int32)
    off = None
    for r in range(nrow):
        cols = ci[rs[r]:rs[r + 1]]
        vals = va[rs[r]:rs[r + 1]]
        lo = [c for c in cols if c < r]
        hi = [c for c in cols if c > r]
        for c, v in zip(cols, vals):
            if c == r:
                diag[r] = v
            else:
                off = v
        nbr[r, 3 - len(lo):3] = lo
        nbr[r, 3:3 + len(hi)] = hi
    return (rs, ci, va, rhs), diag, nbr, off


SINGLE = 0x10  # BNN_PCG_SINGLE_REDUCTION: both inner products in one reduction


@pytest.mark.parametrize("form", [0, SINGLE], ids=["two_reductions", "single_reduction"])
@pytest.mark.parametrize("mode,omode", [("fp32", 0), ("fp64", 1), ("refined", 2)])
def test_pcg_7pt_matches_oracle(bnn, oracle_mod, mode, omode, form):
    (rs, ci, va, rhs), diag, nbr, off = _system(oracle_mod)
    tol = 1e-8 if mode == "refined" else 1e-6
    m = bnn.capi.PCG_MODE[mode] | form
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, tol, 5000, mode=m, inner_tol=1e-3)
    xo, so = oracle_mod.pcg(rs, ci, va, rhs, tol, 5000, omode | form, inner_tol=1e-3)
    assert st["success"] == 1 and so["success"]
    assert st["iterations"] == so["iterations"]
    if mode == "fp32":
        assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))
    else:
        assert np.array_equal(x, xo)


def test_refined_reaches_1e8_fp64_checked(bnn, oracle_mod):
    """Refined FP32 PCG: max|b - A x| (FP64) < 1e-8 max|b|"""
    (rs, ci, va, rhs), diag, nbr, off = _system(oracle_mod, n=32, steps=4)
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, 1e-8, 5000, mode="refined", inner_tol=1e-3)
    n = len(rhs)
    ax = np.zeros(n)
    for r in range(n):
        for j in range(rs[r], rs[r + 1]):
            ax[r] += float(va[j]) * x[ci[j]]
    res = np.abs(rhs.astype(np.float64) - ax).max()
    assert res < 1e-8 * np.abs(rhs).max()


def _box_system(nx=40, ny=36, nz=30, holes=0.08, seed=5):
    """A 7-point system on a box of cells with random holes (air cells), rows in cell
    order and neighbours in their direction slots (-z,-y,-x,+x,+y,+z): the layout of a
    grid, which the solver packs into 16-byte row records.  Returns the slot layout, the
    same system with each row's neighbours listed compactly (the general layout), and the
    CSR form for the oracle."""
    rng = np.random.default_rng(seed)
    act = rng.random((nz, ny, nx)) > holes
    row = -np.ones((nz, ny, nx), np.int64)
    row[act] = np.arange(int(act.sum()))
    n = int(act.sum())
    dt = np.float32(1.0 / 30)
    nbr = -np.ones((n, 6), np.int32)
    k, j, i = np.nonzero(act)
    r = row[k, j, i]
    for slot, (dk, dj, di) in enumerate([(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (0, 1, 0), (1, 0, 0)]):
        kk, jj, ii = k + dk, j + dj, i + di
        ok = (kk >= 0) & (kk < nz) & (jj >= 0) & (jj < ny) & (ii >= 0) & (ii < nx)
        nb = np.full(n, -1, np.int64)
        nb[ok] = row[kk[ok], jj[ok], ii[ok]]
        nbr[r, slot] = nb
    cnt = (nbr >= 0).sum(1)
    diag = (cnt * dt + (6 - cnt) * dt / np.float32(0.5)).astype(np.float32)
    rhs = (rng.standard_normal(n) * 1e-3).astype(np.float32)
    compact = -np.ones_like(nbr)
    rs, ci, va = [0], [], []
    for q in range(n):
        lo = [c for c in nbr[q, :3] if c >= 0]
        hi = [c for c in nbr[q, 3:] if c >= 0]
        compact[q, 3 - len(lo):3] = lo
        compact[q, 3:3 + len(hi)] = hi
        for c in lo:
            ci.append(c); va.append(-dt)
        ci.append(q); va.append(diag[q])
        for c in hi:
            ci.append(c); va.append(-dt)
        rs.append(len(ci))
    return nbr, compact, diag, -dt, rhs, (np.array(rs), np.array(ci), np.array(va, np.float32))


@pytest.mark.parametrize("form", [0, SINGLE], ids=["two_reductions", "single_reduction"])
@pytest.mark.parametrize("mode,omode", [("fp32", 0), ("fp64", 1), ("refined", 2)])
def test_pcg_7pt_grid_rows_packed_matches_oracle(bnn, oracle_mod, mode, omode, form):
    """Grid-ordered rows take the packed-record solve (x neighbours by warp shuffle); the
    compact layout of the same system takes the general one.  Both equal the oracle, in
    either step order."""
    nbr, compact, diag, off, rhs, (rs, ci, va) = _box_system()
    tol = 1e-8 if mode == "refined" else 1e-6
    xo, so = oracle_mod.pcg(rs, ci, va, rhs, tol, 5000, omode | form, inner_tol=1e-3)
    assert so["success"]
    for layout in (nbr, compact):
        x, st = bnn.pcg_solve_7pt(diag, layout, off, rhs, tol, 5000, mode=bnn.capi.PCG_MODE[mode] | form,
                                  inner_tol=1e-3)
        assert st["success"] == 1
        assert st["iterations"] == so["iterations"]
        if mode == "fp32":
            assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))
        else:
            assert np.array_equal(x, xo)


def _slot_system(nbr, seed):
    """Diagonal (every missing neighbour counted as a face to air, so the matrix is
    strictly diagonally dominant), right-hand side and CSR (columns in slot order, the
    solver's summation order) of a system given as slot neighbours."""
    rng = np.random.default_rng(seed)
    n = len(nbr)
    dt = np.float32(1.0 / 30)
    cnt = (nbr >= 0).sum(1)
    diag = (cnt * dt + (6 - cnt) * dt / np.float32(0.5)).astype(np.float32)
    rhs = (rng.standard_normal(n) * 1e-3).astype(np.float32)
    rs, ci, va = [0], [], []
    for q in range(n):
        for c in nbr[q, :3]:
            if c >= 0:
                ci.append(c); va.append(-dt)
        ci.append(q); va.append(diag[q])
        for c in nbr[q, 3:]:
            if c >= 0:
                ci.append(c); va.append(-dt)
        rs.append(len(ci))
    return diag, -dt, rhs, (np.array(rs), np.array(ci), np.array(va, np.float32))


def _grid_slots(act):
    """Slot neighbours (-z,-y,-x,+x,+y,+z) of the active cells of a (z, y, x) mask, rows
    in cell order."""
    nz, ny, nx = act.shape
    row = -np.ones(act.shape, np.int64)
    row[act] = np.arange(int(act.sum()))
    k, j, i = np.nonzero(act)
    r = row[k, j, i]
    nbr = -np.ones((int(act.sum()), 6), np.int32)
    for slot, (dk, dj, di) in enumerate([(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (0, 1, 0), (1, 0, 0)]):
        kk, jj, ii = k + dk, j + dj, i + di
        ok = (kk >= 0) & (kk < nz) & (jj >= 0) & (jj < ny) & (ii >= 0) & (ii < nx)
        nb = np.full(len(r), -1, np.int64)
        nb[ok] = row[kk[ok], jj[ok], ii[ok]]
        nbr[r, slot] = nb
    return nbr


def _layout_system(kind):
    """Grid-row systems of unusual shape for the packed-record solve: 'box' (a box of
    cells with holes), 'wide_rows' (z layers of 120 then 2000 cells along x: y neighbours
    up to ~2000 rows away) and 'unordered_z' (x chains whose z partners are shuffled in
    blocks of 16 rows: valid grid rows whose -z / +z neighbours are not in row order)."""
    rng = np.random.default_rng(21)
    if kind == "box":
        nbr = _grid_slots(rng.random((30, 36, 40)) > 0.08)
    elif kind == "wide_rows":
        act = rng.random((6, 6, 2000)) > 0.08
        act[:3, :, 120:] = False
        nbr = _grid_slots(act)
    else:
        half = 6 * 2048
        n = 2 * half
        nbr = -np.ones((n, 6), np.int32)
        r = np.arange(n)
        chain = (r % 64) != 0  # x chains of 64 rows
        nbr[chain, 2] = r[chain] - 1
        nxt = np.roll(chain, -1) & (r < n - 1)
        nbr[nxt, 3] = r[nxt] + 1
        perm = np.arange(half).reshape(-1, 16)
        for b in perm:
            rng.shuffle(b)
        perm = perm.ravel()
        nbr[np.arange(half), 5] = half + perm
        nbr[half + perm, 0] = np.arange(half)
    return (nbr,) + _slot_system(nbr, 22)


@pytest.mark.parametrize("kind", ["box", "wide_rows", "unordered_z"])
@pytest.mark.parametrize("mode,omode", [("fp32", 0), ("fp64", 1), ("refined", 2)])
def test_pcg_grid_row_layouts_match_oracle(bnn, oracle_mod, kind, mode, omode):
    """Grid rows whose y neighbours lie far away, or whose z partners are out of row order,
    still take the packed-record solve (its x neighbours by warp shuffle, the others by row
    distance) and equal the oracle bit for bit."""
    nbr, diag, off, rhs, (rs, ci, va) = _layout_system(kind)
    tol = 1e-8 if mode == "refined" else 1e-6
    xo, so = oracle_mod.pcg(rs, ci, va, rhs, tol, 5000, omode, inner_tol=1e-3)
    assert so["success"]
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, tol, 5000, mode=bnn.capi.PCG_MODE[mode], inner_tol=1e-3)
    assert st["success"] == 1 and st["iterations"] == so["iterations"]
    if mode == "fp32":
        assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))
    else:
        assert np.array_equal(x, xo)


def _first_cells(nx, ny, n, seed):
    """The first n cells, in cell order, of a grid of nx by ny cells a plane: neighbour
    table (-z, -y, -x, +x, +y, +z), diagonal with 1/theta terms, right-hand side."""
    r = np.arange(n, dtype=np.int64)
    x, y = r % nx, r // nx % ny
    cand = [r - nx * ny, r - nx, r - 1, r + 1, r + nx, r + nx * ny]
    ok = [r >= nx * ny, y > 0, x > 0, x < nx - 1, y < ny - 1, np.ones(n, bool)]
    nbr = np.stack([np.where(o & (c >= 0) & (c < n), c, -1) for c, o in zip(cand, ok)], 1).astype(np.int32)
    rng = np.random.default_rng(seed)
    theta = (0.05 + 0.95 * rng.random((n, 6))).astype(np.float32)
    one = np.float32(1.0)
    diag = (np.where(nbr >= 0, one, one / theta).sum(1) * np.float32(0.004)).astype(np.float32)
    return nbr, diag, rng.standard_normal(n).astype(np.float32)


def _csr_of(nbr, diag, off):
    """The same rows for the oracle: entries in column order, the diagonal in its place."""
    n = len(diag)
    cols = np.concatenate([nbr[:, :3], np.arange(n, dtype=np.int32)[:, None], nbr[:, 3:]], 1)
    vals = np.full(cols.shape, off, np.float32)
    vals[:, 3] = diag
    keep = cols >= 0
    start = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.uint32)
    return start, cols[keep].astype(np.uint32), vals[keep]


# Edges of the chunk-resident solve on 148 SMs: of a 2048-row chunk; of the 16 chunks of one
# cluster; of one, two, three and six chunks per SM (FP32) and of one, two and four (FP64); of the
# rows its 8-byte records hold (512 cells along x, 2^18 - 1 a plane), past which the other kernels
# take over.
_SM = 148 * 2048


@pytest.mark.parametrize("nx,ny,n", [
    (1, 1, 1), (7, 5, 2047), (7, 5, 2048), (7, 5, 2049), (512, 3, 4 * 2048 + 1), (513, 3, 4 * 2048 + 1),
    (31, 29, 15 * 2048 + 1), (31, 29, 16 * 2048), (31, 29, 16 * 2048 + 1),
    (31, 29, 32 * 2048), (31, 29, 33 * 2048 + 5), (64, 80, _SM), (64, 80, _SM + 1), (101, 90, 2 * _SM), (101, 90, 2 * _SM + 1),
    (102, 154, 3 * _SM + 1), (102, 154, 4 * _SM), (102, 154, 4 * _SM + 1), (260, 260, 6 * _SM), (260, 260, 6 * _SM + 1),
    (512, 511, 600_000), (512, 512, 600_000)])
@pytest.mark.parametrize("mode,omode", [("fp32", 0), ("fp64", 1)])
def test_pcg_chunk_edges_match_oracle(bnn, oracle_mod, nx, ny, n, mode, omode):
    nbr, diag, rhs = _first_cells(nx, ny, n, seed=nx + n)
    off = -float(np.float32(0.004))
    # a handful of iterations: what differs would differ in the first ones already
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, 1e-6, 5, mode=mode)
    xo, so = oracle_mod.pcg(*_csr_of(nbr, diag, off), rhs, 1e-6, 5, omode)
    assert st["iterations"] == so["iterations"]
    if mode == "fp32":
        assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))
    else:
        assert np.array_equal(x, xo)


@pytest.mark.parametrize("chunks", [155, 195, 345])
@pytest.mark.parametrize("mode,omode", [("fp32", 0), ("fp64", 1)])
def test_pcg_groups_without_a_chunk_match_oracle(bnn, oracle_mod, chunks, mode, omode):
    """Chunk counts that leave groups of the last blocks without work (two or three groups a block on
    148 SMs): they take every wait's result all the same, over many exchanges."""
    n = chunks * 2048 - 3
    nbr, diag, rhs = _first_cells(64, 80, n, seed=chunks)
    off = -float(np.float32(0.004))
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, 1e-6, 60, mode=mode)
    xo, so = oracle_mod.pcg(*_csr_of(nbr, diag, off), rhs, 1e-6, 60, omode)
    assert st["iterations"] == so["iterations"] == 60
    if mode == "fp32":
        assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))
    else:
        assert np.array_equal(x, xo)


@pytest.mark.parametrize("mode", ["fp32", "fp64", "refined"])
def test_pcg_unbounded_offdiagonal_without_neighbours(bnn, mode):
    """Rows without neighbours never meet the off-diagonal value, finite or not"""
    n = 3000
    nbr = np.full((n, 6), -1, np.int32)
    diag = np.full(n, 0.5, np.float32)
    rhs = np.random.default_rng(2).standard_normal(n).astype(np.float32)
    x, st = bnn.pcg_solve_7pt(diag, nbr, -np.inf, rhs, 1e-6, 10, mode=mode)
    assert st["success"] == 1 and np.array_equal(x, (2 * rhs).astype(np.float64))


def test_barrier_wait_gives_up_and_device_stays_usable(bnn, oracle_mod):
    """A block waiting at a barrier that nothing completes (sized for two blocks, one
    launched) gives up after its limit and reports a timeout; the device then solves a
    system as before."""
    from banana_b200 import capi
    status, ms = bnn.pcg_barrier_probe(0.05)
    assert status == capi.STATUS_CODE["TIMEOUT"]
    assert 50.0 <= ms < 5000.0, ms
    nbr, _, diag, off, rhs, (rs, ci, va) = _box_system(12, 10, 8)
    xo, so = oracle_mod.pcg(rs, ci, va, rhs, 1e-6, 5000, 0)
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, 1e-6, 5000)
    assert st["success"] == 1 and st["iterations"] == so["iterations"]
    assert np.array_equal(x.astype(np.float32), xo.astype(np.float32))


@pytest.mark.parametrize("chunks", [3, 17, 60, 200, 420])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_pcg_residual_that_is_not_a_number(bnn, chunks, bad):
    """A right-hand side with an infinity or a NaN makes every later sum and maximum NaN: on every kernel
    the waits still see each exchange (the call returns instead of timing out), and FP64 takes the
    iterations and the outcome of FP32; the refined solve returns too"""
    n = chunks * 2048 - 11
    nbr, diag, rhs = _first_cells(64, 80, n, seed=chunks)
    rhs[n // 2] = bad
    out = {}
    for mode in ("fp32", "fp64", "refined"):
        x, st = bnn.pcg_solve_7pt(diag, nbr, -float(np.float32(0.004)), rhs, 1e-6, 7, mode=mode)
        out[mode] = (st["iterations"], st["success"], int(np.isnan(x).sum()))
    assert out["fp32"] == out["fp64"]
    assert out["fp32"][2] == (n if bad == np.inf else 0)


@pytest.mark.parametrize("limit", [0.02, 0.2])
def test_packet_waits_give_up_and_device_stays_usable(bnn, oracle_mod, limit):
    """The probe's status also covers the waits of the chunk-resident solves, block-wide and per group:
    each gives up on a packet that nobody publishes, says so in its own flag and returns, a group that
    has its packets passes beside it; a solve on their kernel then works"""
    from banana_b200 import capi
    status, ms = bnn.pcg_barrier_probe(limit)
    assert status == capi.STATUS_CODE["TIMEOUT"] and ms >= 1000 * limit
    nbr, diag, rhs = _first_cells(64, 80, 40 * 2048 + 7, seed=8)
    off = -float(np.float32(0.004))
    x, st = bnn.pcg_solve_7pt(diag, nbr, off, rhs, 1e-6, 20)
    xo, so = oracle_mod.pcg(*_csr_of(nbr, diag, off), rhs, 1e-6, 20, 0)
    assert st["iterations"] == so["iterations"] and np.array_equal(x.astype(np.float32), xo.astype(np.float32))


def test_pcg_7pt_rejects_bad_neighbour_index(bnn):
    nbr, _, diag, off, rhs, _ = _box_system(8, 8, 8)
    bad = nbr.copy()
    bad[5, 4] = len(rhs)  # one past the last row
    with pytest.raises(bnn.BnnError):
        bnn.pcg_solve_7pt(diag, bad, off, rhs, 1e-6, 100)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_cell_sort_bitexact(bnn, oracle_mod):
    pts = scenes.point_cloud(200_000, seed=7)
    bmin = np.zeros(3, np.float32)
    nc = np.array([100, 100, 100], np.int32)
    cid, srt, start, oor = oracle_mod.cell_sort(pts, bmin, np.float32(0.01), nc)
    L = bnn.load()
    p = _dev(pts)
    n = len(pts)
    gc = torch.zeros(n, dtype=torch.int32, device="cuda")
    gs = torch.zeros(n, dtype=torch.int32, device="cuda")
    gst = torch.zeros(int(nc.prod()) + 1, dtype=torch.int32, device="cuda")
    o = C.c_uint32()
    rc = L.bnn_cell_sort(C.c_void_p(p.data_ptr()), n, bmin.ctypes.data_as(C.POINTER(C.c_float)), 0.01,
                         nc.ctypes.data_as(C.POINTER(C.c_int32)), C.c_void_p(gc.data_ptr()), C.c_void_p(gs.data_ptr()),
                         C.c_void_p(gst.data_ptr()), C.byref(o), None)
    torch.cuda.synchronize()
    assert rc == 0
    assert o.value == oor
    assert np.array_equal(gc.cpu().numpy().view(np.uint32), cid)
    assert np.array_equal(gs.cpu().numpy().view(np.uint32), srt)
    assert np.array_equal(gst.cpu().numpy().view(np.uint32), start)


@pytest.mark.parametrize("nc,cell", [((3, 5, 7), 0.34), ((17, 33, 41), 1 / 16.5), ((129, 130, 131), 1 / 128)],
                         ids=["105_cells", "23001_cells", "2196870_cells"])
def test_cell_sort_grid_sizes_bitexact(bnn, oracle_mod, nc, cell):
    """Cell starts (the exclusive prefix sum of the cell counts, total last) on grids of one
    scan tile, of a few tiles with a ragged end, and of many tiles"""
    pts = scenes.point_cloud(150_000, seed=11)
    bmin = np.zeros(3, np.float32)
    nc = np.array(nc, np.int32)
    cid, srt, start, oor = oracle_mod.cell_sort(pts, bmin, np.float32(cell), nc)
    L = bnn.load()
    p = _dev(pts)
    n = len(pts)
    gc = torch.zeros(n, dtype=torch.int32, device="cuda")
    gs = torch.zeros(n, dtype=torch.int32, device="cuda")
    gst = torch.full((int(nc.prod()) + 1,), -1, dtype=torch.int32, device="cuda")
    o = C.c_uint32()
    rc = L.bnn_cell_sort(C.c_void_p(p.data_ptr()), n, bmin.ctypes.data_as(C.POINTER(C.c_float)), float(np.float32(cell)),
                         nc.ctypes.data_as(C.POINTER(C.c_int32)), C.c_void_p(gc.data_ptr()), C.c_void_p(gs.data_ptr()),
                         C.c_void_p(gst.data_ptr()), C.byref(o), None)
    torch.cuda.synchronize()
    assert rc == 0
    assert o.value == oor
    assert np.array_equal(gc.cpu().numpy().view(np.uint32), cid)
    assert np.array_equal(gs.cpu().numpy().view(np.uint32), srt)
    assert np.array_equal(gst.cpu().numpy().view(np.uint32), start)


@pytest.mark.parametrize("n", [1, 31, 2_047, 2_048, 2_049, 6_145, 300_001])
@pytest.mark.parametrize("nc", [(1, 1, 1), (16, 16, 1), (257, 1, 1), (40, 41, 40), (300, 300, 200)])
def test_cell_sort_tiles_and_digits(bnn, n, nc):
    """Around the sort's 2048-item tiles and 8-bit digits (0 to 4 passes), points outside the
    grid and a crowded cell among them; the allocation-free call gives the same."""
    rng = np.random.default_rng(n)
    ncf = np.array(nc, np.float32)
    p = (rng.random((n, 3)) * 1.02 * ncf - 0.01 * ncf).astype(np.float32)
    p[n // 2:] = p[n // 2]  # half of the points in one cell
    c = np.clip(p.astype(np.int32), 0, np.array(nc) - 1)
    out = ((p.astype(np.int32) < 0) | (p.astype(np.int32) >= np.array(nc))).any(1).sum()
    cid = (c[:, 2].astype(np.int64) * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    cells = nc[0] * nc[1] * nc[2]
    pos = _dev(p)
    calls = [bnn.load().bnn_cell_sort] + ([bnn.load().bnn_cell_sort_noalloc] if cells <= 1 << 21 else [])
    for call in calls:
        ids, order, start = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (n, n, cells + 1))
        oor = C.c_uint32()
        bnn.capi.check(call(pos.data_ptr(), n, (C.c_float * 3)(), 1.0, (C.c_int32 * 3)(*nc), ids.data_ptr(), order.data_ptr(),
                            start.data_ptr(), C.byref(oor), None), "bnn_cell_sort")
        assert oor.value == out
        assert np.array_equal(ids.cpu().numpy(), cid)
        assert np.array_equal(order.cpu().numpy(), np.argsort(cid, kind="stable"))
        assert np.array_equal(start.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(cid, minlength=cells))]))


def test_z_sort_bitexact(bnn, oracle_mod):
    pts = scenes.point_cloud(100_000, seed=3)
    z, perm = oracle_mod.z_sort(pts, np.float32(0.01))
    L = bnn.load()
    p = _dev(pts)
    n = len(pts)
    gz = torch.zeros(n, dtype=torch.int64, device="cuda")
    gp = torch.zeros(n, dtype=torch.int32, device="cuda")
    rc = L.bnn_z_sort(C.c_void_p(p.data_ptr()), n, 0.01, C.c_void_p(gz.data_ptr()), C.c_void_p(gp.data_ptr()), None)
    assert rc == 0
    assert np.array_equal(gz.cpu().numpy().view(np.uint64), z)
    assert np.array_equal(gp.cpu().numpy().view(np.uint32), perm)


def _lists(off, idx, n):
    return [np.sort(idx[off[i]:off[i + 1]]) for i in range(n)]


@pytest.mark.parametrize("n,seed", [(30_000, 7), (60_000, 1)])
def test_neighbors_set_equal(bnn, oracle_mod, n, seed):
    pts = scenes.point_cloud(n, seed=seed)
    r = np.float32(0.01)
    off_o, idx_o = oracle_mod.neighbors(pts, r)
    L = bnn.load()
    p = _dev(pts)
    goff = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    cap = int(off_o[-1]) + 16
    gidx = torch.zeros(max(cap, 1), dtype=torch.int32, device="cuda")
    tot = C.c_uint64()
    rc = L.bnn_neighbors(C.c_void_p(p.data_ptr()), n, r, C.c_void_p(goff.data_ptr()), C.c_void_p(gidx.data_ptr()),
                         cap, C.byref(tot), None)
    assert rc == 0
    assert tot.value == off_o[-1]
    go = goff.cpu().numpy().view(np.uint64)
    gi = gidx.cpu().numpy().view(np.uint32)[: tot.value]
    assert np.array_equal(go, off_o)
    # set equality per point (the reference's list order depends on its thread schedule)
    owner = np.repeat(np.arange(n), np.diff(go).astype(np.int64))
    a = np.lexsort((gi, owner))
    assert np.array_equal(gi[a], idx_o)


@pytest.mark.parametrize("n,seed,r", [(1, 3, 0.1), (2, 3, 2.0), (31, 3, 0.4), (33, 3, 0.4), (2_049, 3, 0.2), (149_999, 5, 0.012),
                                      (150_001, 5, 0.012)])
def test_neighbors_order_and_edges(bnn, n, seed, r):
    """Lists in their order (27 cells z, y, x major, a cell's points by index), around the sizes
    where a warp's points end and where the points per warp change, with coincident points and a
    cell of one point beside crowded ones; the reference is the same test in numpy float32."""
    rng = np.random.default_rng(seed)
    p = rng.random((n, 3)).astype(np.float32)
    p[: n // 3] = np.float32(0.5) + np.float32(0.02) * rng.standard_normal((n // 3, 3)).astype(np.float32)
    if n > 40:
        p[5:9] = p[4]
    pos = _dev(p)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    idx = torch.zeros(max(1, min(n * n, 60_000_000)), dtype=torch.int32, device="cuda")
    tot = C.c_uint64()
    bnn.capi.check(bnn.load().bnn_neighbors(pos.data_ptr(), n, r, off.data_ptr(), idx.data_ptr(), idx.numel(),
                                            C.byref(tot), None), "bnn_neighbors")
    off = off.cpu().numpy()
    assert off[0] == 0 and off[-1] == tot.value
    idx = idx[: tot.value].cpu().numpy()
    rf = np.float32(r)
    inv = np.float32(1.0 / float(rf))
    t = p - np.float32(1.2345)
    key = np.where(t >= 0, (inv * t).astype(np.int32), (inv * t).astype(np.int32) - 1)
    d = key.max(0) - key.min(0) + 3
    cell = key - key.min(0) + 1
    lin = (cell[:, 2].astype(np.int64) * d[1] + cell[:, 1]) * d[0] + cell[:, 0]
    order = np.argsort(lin, kind="stable")
    slin = lin[order]
    for i in np.unique(np.concatenate([np.arange(min(n, 40)), rng.integers(0, n, 300)])):
        cand = [order[np.searchsorted(slin, lin[i] + dz * d[0] * d[1] + dy * d[0] - 1):
                      np.searchsorted(slin, lin[i] + dz * d[0] * d[1] + dy * d[0] + 1, "right")]
                for dz in (-1, 0, 1) for dy in (-1, 0, 1)]
        cand = np.concatenate(cand)
        cand = cand[cand != i]
        e = p[i] - p[cand]
        l2 = (e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2]
        assert np.array_equal(idx[off[i]:off[i + 1]], cand[l2 < rf * rf]), i


def test_neighbors_capacity_error(bnn):
    pts = scenes.point_cloud(5_000, seed=2)
    L = bnn.load()
    p = _dev(pts)
    goff = torch.zeros(len(pts) + 1, dtype=torch.int64, device="cuda")
    gidx = torch.zeros(4, dtype=torch.int32, device="cuda")
    tot = C.c_uint64()
    rc = L.bnn_neighbors(C.c_void_p(p.data_ptr()), len(pts), 0.05, C.c_void_p(goff.data_ptr()),
                         C.c_void_p(gidx.data_ptr()), 4, C.byref(tot), None)
    assert rc == 8 and tot.value > 4


@pytest.mark.parametrize("n,r", [(150_000, 0.008), (150_003, 0.03), (400_000, 0.0165), (400_001, 0.021)])
def test_neighbors_sparse_and_mixed_sets_equal(bnn, oracle_mod, n, r):
    """Warps whose points lie in many cells walk them a thread per point: sets of less than a point a
    cell, of about four and eight cells a warp, each with crowded cells beside sparse ones"""
    rng = np.random.default_rng(n)
    p = rng.random((n, 3)).astype(np.float32)
    p[: n // 50] = np.float32(0.3) + np.float32(0.01) * rng.standard_normal((n // 50, 3)).astype(np.float32)
    pos = _dev(p)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    idx = torch.zeros(120_000_000, dtype=torch.int32, device="cuda")
    tot = C.c_uint64()
    bnn.capi.check(bnn.load().bnn_neighbors(pos.data_ptr(), n, r, off.data_ptr(), idx.data_ptr(), idx.numel(),
                                            C.byref(tot), None), "bnn_neighbors")
    want_off, want = oracle_mod.neighbors(p, np.float32(r))
    off = off.cpu().numpy()
    assert np.array_equal(off, want_off.astype(np.int64)) and off[-1] == tot.value
    idx = idx[: tot.value].cpu().numpy()
    rows = np.repeat(np.arange(n), np.diff(off))
    a, b = np.lexsort((idx, rows)), np.lexsort((want, rows))
    assert np.array_equal(idx[a], want[b])


def test_pcg_kinds_in_flight_together(bnn):
    """Solves of every kind from several threads at once (one cluster, chunks on one and two groups an
    SM, a general row order, one reduction an iteration): each gives what it gives alone"""
    import threading

    jobs = []
    for nx, ny, n, mode in [(31, 29, 9 * 2048, "fp32"), (64, 80, 60 * 2048 + 3, "fp64"), (64, 80, 160 * 2048, "fp32"),
                            (513, 40, 300_000, "fp32"), (101, 90, 250 * 2048 + 1, "refined")]:
        nbr, diag, rhs = _first_cells(nx, ny, n, seed=n)
        jobs.append((diag, nbr, rhs, mode))
    d, nb, b, _ = jobs[1]
    perm = np.random.default_rng(4).permutation(len(d))
    inv = np.empty(len(d), np.int64)
    inv[perm] = np.arange(len(d))
    jobs.append((d[perm], np.where(nb[perm] >= 0, inv[nb[perm]], -1).astype(np.int32), b[perm], "fp32"))

    def solve(j, form):
        mode = bnn.capi.PCG_MODE[j[3]] | form
        return bnn.pcg_solve_7pt(j[0], j[1], -float(np.float32(0.004)), j[2], 1e-5, 40, mode=mode)[0]

    forms = [(j, 0) for j in jobs] + [(jobs[0], SINGLE), (jobs[2], SINGLE)]
    alone = [solve(*f) for f in forms]
    got = [[] for _ in forms]

    def run(i):
        for _ in range(6):
            got[i].append(solve(*forms[i]))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(forms))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, a in enumerate(alone):
        assert len(got[i]) == 6 and all(np.array_equal(a, x) for x in got[i]), i
