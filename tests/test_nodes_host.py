"""The node form's plan (mk_nodes_plan, host only) replayed in FP64 NumPy with
the kernels' index arithmetic: leaf, merge and pixel steps over the plan's own
tables, every array access in range, against the direct sum.

Tolerance: the plan interpolates with e = 4 (phi/2)^n / n! <= 3e-8 per axis
and step; two axes and Lebesgue constants L below 2.8 give e (1 + L) (1 + L^2)
< 1.1e-6 of the sum of |E| at worst for two steps, e (1 + L) (1 + L^2 + L^4)
< 8.0e-6 for three; the dropped third-order phase is below 1e-6 rad."""
import ctypes

import numpy as np
import pytest

from mosaic_gb300 import _lib

K = 2 * np.pi / 1.2398e-10
MERGE = np.dtype([(n, "i4") for n in ("ratio_y", "ratio_z", "strip", "strips", "rowg", "chunks")] +
                 [(n, "i8") for n in ("w_off", "item_off")])
FRAME = np.dtype([("p0", "f8", 3), ("ey", "f8", 3), ("ez", "f8", 3), ("b", "f8", 3), ("ny", "i4"), ("nz", "i4")] +
                 [(n, "i4", 3) for n in ("ly", "lz", "py", "pz")] + [("bpy", "i4"), ("bpz", "i4"), ("mg", MERGE, 2)] +
                 [("off", "i8", 3)] + [(n, "i8") for n in ("pix_off", "pblk_off", "part_off", "w_off")])
SRC = np.dtype([("dh", "f4", 3), ("species", "i4"), ("dl", "f4", 3), ("count", "i4"), ("o", "f8", 3),
                ("first", "i8")])


def _cheb(n):
    return np.cos((2 * np.arange(n) + 1) * np.pi / (2 * n))


def _half(n):
    return 0.5 * (n - 1) + 0.25


def _lagrange(x, n):
    xs = _cheb(n)
    return np.array([np.prod([(x - xs[i]) / (xs[j] - xs[i]) for i in range(n) if i != j]) for j in range(n)])


def _grid(ny, nz, dist, pitch, tt):
    R = np.array([[np.cos(tt), 0, -np.sin(tt)], [0, 1, 0], [np.sin(tt), 0, np.cos(tt)]])
    y, z = (np.arange(ny) - (ny - 1) / 2) * pitch, (np.arange(nz) - (nz - 1) / 2) * pitch
    Z, Y = np.meshgrid(z, y, indexing="ij")
    return (R @ np.stack([np.full(Y.size, dist), Y.ravel(), Z.ravel()])).T


def _fit(P, ny, nz):
    p0 = P[0]
    ey = (P[ny - 1] - p0) / (ny - 1) if ny > 1 else np.zeros(3)
    ez = (P[(nz - 1) * ny] - p0) / (nz - 1) if nz > 1 else np.zeros(3)
    return np.concatenate([p0, ey, ez, [0.0, np.linalg.norm(P, axis=1).min(), 0.0]])


def _tiles(rng, tile_boxes, T, side):
    """Tiles of T atoms in boxes of the given side around given centres."""
    org, atoms = [], []
    for c in tile_boxes:
        a = c + (rng.random((T, 3)) - 0.5) * side
        o = 0.5 * (a.min(0) + a.max(0))
        org.append([*o, np.linalg.norm(a - o, axis=1).max()])
        atoms.append(a)
    return np.array(org), np.array(atoms)


def _plan(org, counts, T, shapes, fits, bd, direct=1.0, group=-1):
    L = _lib.load()
    nf, nt = len(shapes), len(org)
    nb = L.mk_nodes_plan_bytes(nf, nt)
    buf = np.zeros(nb, np.uint8)
    plan = _lib.MkNodePlan()
    counts = np.asarray(counts, np.int64)
    shapes = np.ascontiguousarray(shapes, np.int64)
    fits = np.ascontiguousarray(fits)
    bd = np.ascontiguousarray(bd)
    rc = L.mk_nodes_plan(nt, T, len(counts), counts.ctypes.data, org.ctypes.data, nf, shapes.ctypes.data,
                         fits.ctypes.data, bd.ctypes.data, K, 1e-6, direct, group, ctypes.byref(plan),
                         buf.ctypes.data, nb)
    return rc, plan, buf


def _phase(P, b, o_ref, d):
    """Cycles of a source at o_ref + d relative to o_ref, as the kernels expand it."""
    kap = K / (2 * np.pi)
    R = np.linalg.norm(P, axis=1)
    u = P / R[:, None]
    uo = u @ o_ref
    w = b - u + (o_ref - uo[:, None] * u) / R[:, None]
    ud = u @ d
    return kap * (w @ d) + 0.5 * kap / (R * (1 - uo / R)) * (d @ d - ud ** 2)


def _run(plan, buf, org, atoms, shapes, P, n_pix):
    fr = np.frombuffer(buf, FRAME, plan.n_frames, 0)
    ints = lambda n, off: np.frombuffer(buf, np.int32, n, off)
    src = np.frombuffer(buf, SRC, plan.n_src, plan.off_src)
    msrc = np.frombuffer(buf, SRC, plan.n_msrc, plan.off_msrc)
    morg = np.frombuffer(buf, np.float64, 4 * plan.n_msrc, plan.off_morg).reshape(-1, 4)
    mem, mid = ints(plan.n_members, plan.off_members), ints(plan.n_mid, plan.off_mid)
    n = (plan.n0, plan.nm, plan.n1)
    out = np.zeros(n_pix, complex)
    hit = np.zeros(n_pix, int)

    def nodes(F, p, lv):
        pz, pyi = divmod(p, F["py"][lv])
        ly, lz = F["ly"][lv], F["lz"][lv]
        y = pyi * ly + 0.5 * (ly - 1) + _half(ly) * _cheb(n[lv])
        z = pz * lz + 0.5 * (lz - 1) + _half(lz) * _cheb(n[lv])
        Z, Y = np.meshgrid(z, y, indexing="ij")
        return F["p0"] + Y.ravel()[:, None] * F["ey"] + Z.ravel()[:, None] * F["ez"]

    def leaf(F, t, lv):         # a tile's field on every patch of a level
        o = org[t, :3]
        one = lambda Pn: np.array([np.exp(2j * np.pi * _phase(Pn, F["b"], o, a - o)) for a in atoms[t]]).sum(0)
        return np.array([one(nodes(F, p, lv)) for p in range(F["py"][lv] * F["pz"][lv])]).reshape(-1, n[lv], n[lv])

    def blocks(M, F, lo, hi):   # the merge's blocks cover every node of the finer level once
        rows = {6: 3, 8: 4, 10: 5, 12: 3, 16: 4}[n[hi]]
        got = np.zeros((F["pz"][hi], F["py"][hi], n[hi], n[hi]), int)
        for e in range(F["pz"][hi] * F["py"][lo] * M["strips"] * M["chunks"]):
            e, chunk = divmod(e, M["chunks"])
            e, strip = divmod(e, M["strips"])
            pz, cy = divmod(e, F["py"][lo])
            s0 = strip * M["strip"]
            patches = min(M["strip"], M["ratio_y"] - s0, F["py"][hi] - cy * M["ratio_y"] - s0)
            row0 = chunk * M["rowg"] * rows
            nrow = min(M["rowg"] * rows, n[hi] - row0)
            assert M["rowg"] * rows <= 16 and M["strip"] * n[hi] * M["rowg"] <= 128 and nrow % rows == 0
            for th in range(128 if patches > 0 else 0):
                rg, oc = divmod(th, M["strip"] * n[hi])
                if oc < patches * n[hi] and rg * rows < nrow and rg < M["rowg"]:
                    r = row0 + rg * rows
                    got[pz, cy * M["ratio_y"] + s0 + oc // n[hi], r:r + rows, oc % n[hi]] += 1
        assert (got == 1).all()

    def merge(M, F, lo, hi, sources, V, where):
        """sources' runs of V's rows, at `where`, onto the finer level."""
        blocks(M, F, lo, hi)
        full = np.zeros((len(sources), F["py"][hi] * F["pz"][hi], n[hi], n[hi]), complex)
        for p in range(F["py"][hi] * F["pz"][hi]):
            pz, py = divmod(p, F["py"][hi])
            Pn = nodes(F, p, hi)
            cy, cz = py // M["ratio_y"], pz // M["ratio_z"]
            assert cy < F["py"][lo] and cz < F["pz"][lo]
            pos = lambda sub, l1, l0: (sub * l1 + 0.5 * (l1 - 1) + _half(l1) * _cheb(n[hi]) - 0.5 * (l0 - 1)) / _half(l0)
            Wy = np.array([_lagrange(x, n[lo]) for x in pos(py - cy * M["ratio_y"], F["ly"][hi], F["ly"][lo])])
            Wz = np.array([_lagrange(x, n[lo]) for x in pos(pz - cz * M["ratio_z"], F["lz"][hi], F["lz"][lo])])
            for s, S in enumerate(sources):
                for i in range(S["first"], S["first"] + S["count"]):
                    v = Wz @ V[i, cz * F["py"][lo] + cy] @ Wy.T
                    ph = _phase(Pn, F["b"], S["o"], where[i] - S["o"])
                    full[s, p] += v * np.exp(2j * np.pi * ph).reshape(n[hi], n[hi])
        return full

    for F in fr:
        V1 = np.zeros((0, F["py"][2] * F["pz"][2], n[2], n[2]), complex)
        if n[0]:
            V = np.array([leaf(F, t, 0) for t in mem])
            lo, where = 0, org[mem, :3]
            if n[1]:
                V = merge(F["mg"][0], F, 0, 1, msrc, V, where)
                for row, t in zip(ints(plan.n_msingle, plan.off_mrow), ints(plan.n_msingle, plan.off_msingle)):
                    assert msrc[row]["count"] == 0
                    V[row] = leaf(F, t, 1)
                assert sum(msrc["count"]) == len(mem) and (msrc["count"] == 0).sum() == plan.n_msingle
                lo, where = 1, morg[:, :3]
            V1 = merge(F["mg"][1], F, lo, 2, src[:plan.n_groups], V, where)
        if plan.n_mid:
            V1 = np.concatenate([V1, np.array([leaf(F, t, 2) for t in mid])])
        n1, ly, lz = n[2], F["ly"][2], F["lz"][2]
        for p in range(F["py"][2] * F["pz"][2]):
            pz, py = divmod(p, F["py"][2])
            cols = np.arange(py * ly, min((py + 1) * ly, F["ny"]))
            rows = np.arange(pz * lz, min((pz + 1) * lz, F["nz"]))
            assert F["bpy"] * 32 >= len(cols) and F["bpz"] * 16 >= len(rows)
            Wy = np.array([_lagrange((c - py * ly - 0.5 * (ly - 1)) / _half(ly), n1) for c in cols])
            Wz = np.array([_lagrange((r - pz * lz - 0.5 * (lz - 1)) / _half(lz), n1) for r in rows])
            g = (F["pix_off"] + rows[:, None] * F["ny"] + cols[None, :]).ravel()
            for s in range(plan.n_src):
                S = src[s]
                o = S["dh"].astype(float) + S["dl"]
                v = (Wz @ V1[s, p] @ Wy.T).ravel()
                out[g] += v * np.exp(2j * np.pi * _phase(P[g], F["b"], np.zeros(3), o))
            hit[g] += 1
    assert (hit == 1).all()
    return out


@pytest.mark.parametrize("shapes, tiles, side, group", [
    ([(40, 33)], 6, 2e-9, 0),                    # no groups, ragged
    ([(200, 70)], 64, 2e-9, 8),                   # groups, several fine patches
    ([(64, 48), (100, 16)], 64, 2e-9, 8),         # frames of two shapes
    ([(1, 50), (50, 1)], 6, 2e-9, 0),            # single column, single row
])
def test_plan_reproduces_the_direct_sum(shapes, tiles, side, group):
    rng = np.random.default_rng(5)
    T = 4
    g = int(np.ceil(tiles ** (1 / 3)))
    cells = np.array([(x, y, z) for x in range(g) for y in range(g) for z in range(g)])[:tiles]
    if group:                   # octants first, as a space-filling curve visits them
        cells = cells[np.lexsort((cells[:, 2], cells[:, 1], cells[:, 0], *(cells // 2).T[::-1]))]
    org, atoms = _tiles(rng, (cells - g / 2) * 3e-9, T, side)
    P = [_grid(ny, nz, 0.3, 55e-6, 0.4) for ny, nz in shapes]
    offs = np.concatenate([[0], np.cumsum([len(p) for p in P])])
    sh = np.array([(o, ny, nz) for o, (ny, nz) in zip(offs, shapes)])
    fits = np.array([_fit(p, ny, nz) for p, (ny, nz) in zip(P, shapes)])
    bd = np.array([[1.0, 0, 0]] * len(shapes))
    half = tiles // 2 * T       # two species
    rc, plan, buf = _plan(org, [half, tiles * T - half], T, sh, fits, bd, group=group)
    assert rc == _lib.MK_OK, _lib.load().mk_last_error()
    assert plan.n_wide == 0 and (plan.n_groups > 0) == (group > 0)
    allP = np.concatenate(P)
    got = _run(plan, buf, org, atoms, shapes, allP, len(allP))
    a = atoms.reshape(-1, 3)
    R = np.linalg.norm(allP, axis=1)
    num = (a * a).sum(1)[None] - 2 * allP @ a.T
    d = num / (np.sqrt(R[:, None] ** 2 + num) + R[:, None])
    ref = np.exp(1j * K * (a[:, 0][None] + d)).sum(1)
    assert np.abs(got - ref).max() <= 2.1e-6 * len(a)


def test_plan_with_a_middle_level():
    """Tiles in runs on middle nodes and runs in groups; a few tiles too wide
    for the coarse nodes on the middle ones by themselves."""
    rng = np.random.default_rng(7)
    T, g, (ny, nz) = 3, 6, (400, 300)
    cells = np.array([(x, y, z) for x in range(g) for y in range(g) for z in range(g)])
    # octants first, as a space-filling curve visits them
    cells = cells[np.lexsort((*(cells % 2).T[::-1], *(cells // 2 % 2).T[::-1], *(cells // 4).T[::-1]))]
    org, atoms = _tiles(rng, (cells - g / 2) * 2.8e-9, 8, 2.6e-9)
    atoms = atoms[:, :T].copy()
    for t in (5, 100, 101, 215):            # spread out about their centres
        atoms[t] = org[t, :3] + 2.0 * (atoms[t] - org[t, :3])
        org[t, 3] *= 2.0
    P = _grid(ny, nz, 0.3, 55e-6, 0.4)
    n = len(org)
    rc, plan, buf = _plan(org, [40 * T, (n - 40) * T], T, [(0, ny, nz)], [_fit(P, ny, nz)], [[1.0, 0, 0]])
    assert rc == _lib.MK_OK and plan.nm > 0 and plan.n_msingle > 0
    got = _run(plan, buf, org, atoms, [(ny, nz)], P, len(P))
    a = atoms.reshape(-1, 3)
    R = np.linalg.norm(P, axis=1)
    ref = np.zeros(len(P), complex)
    for x in a:
        num = x @ x - 2 * P @ x
        ref += np.exp(1j * K * (x[0] + num / (np.sqrt(R ** 2 + num) + R)))
    assert np.abs(got - ref).max() <= 9.0e-6 * len(a)


def test_plan_declines():
    """Pixels off their plane, off their grid or at the origin, tiles without
    a finite extent, tiles at a distance where the factor changes across the
    sample: the split kernel's, or the FP64 sum's, to take."""
    rng = np.random.default_rng(1)
    org, _ = _tiles(rng, np.zeros((4, 3)), 4, 2e-9)
    sh, bd = np.array([(0, 40, 40)]), np.array([[1.0, 0, 0]])
    good = _fit(_grid(40, 40, 1.0, 55e-6, 0.4), 40, 40)[None]
    assert _plan(org, [16], 4, sh, good, bd)[0] == _lib.MK_OK
    for i, v in ((9, 1e-3), (9, np.inf), (9, np.nan), (10, 0.0), (11, 0.3), (11, np.nan)):
        bad = good.copy()
        bad[0, i] = v
        assert _plan(org, [16], 4, sh, bad, bd)[0] == _lib.MK_EDECLINE, (i, v)
    for v in (np.nan, np.inf, 1.0):
        bad = org.copy()
        bad[2, 3] = v
        assert _plan(bad, [16], 4, sh, good, bd)[0] == _lib.MK_EDECLINE, v
    far = org.copy()
    far[:, 0] += 1e-6
    assert _plan(far, [16], 4, sh, good, bd)[0] == _lib.MK_EDECLINE
    assert _plan(org, [16], 4, sh, good, bd, direct=1e-30)[0] == _lib.MK_EDECLINE
