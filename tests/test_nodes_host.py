"""The node form's plan (mk_nodes_plan, host only) replayed in FP64 NumPy with
the kernels' index arithmetic: leaf, merge and pixel steps over the plan's own
tables, every array access in range, against the direct sum.

Tolerance: the plan interpolates with 4 (phi/2)^n / n! <= 3e-8 per axis and
step; two axes, at most two steps and Lebesgue constants below 2.8 give
3e-8 * (1 + 2.8) * (1 + 2.8^2) < 1.1e-6 of the sum of |E| at worst; the
dropped third-order phase is below 1e-6 rad."""
import ctypes

import numpy as np
import pytest

from mosaic_gb300 import _lib

K = 2 * np.pi / 1.2398e-10
FRAME = np.dtype([("p0", "f8", 3), ("ey", "f8", 3), ("ez", "f8", 3), ("b", "f8", 3)] +
                 [(n, "i4") for n in ("ny", "nz", "l1y", "l1z", "p1y", "p1z", "ratio_y", "ratio_z",
                                      "p0y", "p0z", "bpy", "bpz", "strip", "strips", "rowg", "chunks")] +
                 [(n, "i8") for n in ("pix_off", "node0_off", "patch1_off", "pblk_off", "part_off", "w_off", "item_off")])
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
    src = np.frombuffer(buf, SRC, plan.n_src, plan.off_src)
    mem = np.frombuffer(buf, np.int32, plan.n_members, plan.off_members)
    mid = np.frombuffer(buf, np.int32, plan.n_mid, plan.off_mid)
    n0, n1 = plan.n0, plan.n1
    out = np.zeros(n_pix, complex)
    hit = np.zeros(n_pix, int)

    def nodes(F, p, py, ly, lz, n):
        pz, pyi = divmod(p, py)
        y = pyi * ly + 0.5 * (ly - 1) + _half(ly) * _cheb(n)
        z = pz * lz + 0.5 * (lz - 1) + _half(lz) * _cheb(n)
        Z, Y = np.meshgrid(z, y, indexing="ij")
        return F["p0"] + Y.ravel()[:, None] * F["ey"] + Z.ravel()[:, None] * F["ez"]

    def leaf(t, Pn, b):
        o = org[t, :3]
        return np.array([np.exp(2j * np.pi * _phase(Pn, b, o, a - o)) for a in atoms[t]]).sum(0)

    for F in fr:
        if n0:                  # the merge's blocks cover every fine node once
            rows = {6: 3, 8: 4, 10: 5, 12: 3}[n1]
            got = np.zeros((F["p1z"], F["p1y"], n1, n1), int)
            for e in range(F["p1z"] * F["p0y"] * F["strips"] * F["chunks"]):
                e, chunk = divmod(e, F["chunks"])
                e, strip = divmod(e, F["strips"])
                pz, cy = divmod(e, F["p0y"])
                s0 = strip * F["strip"]
                patches = min(F["strip"], F["ratio_y"] - s0, F["p1y"] - cy * F["ratio_y"] - s0)
                row0 = chunk * F["rowg"] * rows
                nrow = min(F["rowg"] * rows, n1 - row0)
                assert F["rowg"] * rows <= 16 and F["strip"] * n1 * F["rowg"] <= 128 and nrow % rows == 0
                for th in range(128 if patches > 0 else 0):
                    rg, oc = divmod(th, F["strip"] * n1)
                    if oc < patches * n1 and rg * rows < nrow and rg < F["rowg"]:
                        r = row0 + rg * rows
                        got[pz, cy * F["ratio_y"] + s0 + oc // n1, r:r + rows, oc % n1] += 1
            assert (got == 1).all()
        l0y, l0z = F["l1y"] * F["ratio_y"], F["l1z"] * F["ratio_z"]
        V0 = {}
        for p in range(F["p0y"] * F["p0z"] if n0 else 0):
            Pn = nodes(F, p, F["p0y"], l0y, l0z, n0)
            for i, t in enumerate(mem):
                V0[i, p] = leaf(t, Pn, F["b"]).reshape(n0, n0)
        for p in range(F["p1y"] * F["p1z"]):
            pz, py = divmod(p, F["p1y"])
            Pn = nodes(F, p, F["p1y"], F["l1y"], F["l1z"], n1)
            V1 = np.zeros((plan.n_src, n1, n1), complex)
            for s in range(plan.n_groups):
                S = src[s]
                cy, cz = py // F["ratio_y"], pz // F["ratio_z"]
                sy, sz = py - cy * F["ratio_y"], pz - cz * F["ratio_z"]
                assert cy < F["p0y"] and cz < F["p0z"]
                pos = lambda sub, l1, l0: (sub * l1 + 0.5 * (l1 - 1) + _half(l1) * _cheb(n1) - 0.5 * (l0 - 1)) / _half(l0)
                Wy = np.array([_lagrange(x, n0) for x in pos(sy, F["l1y"], l0y)])
                Wz = np.array([_lagrange(x, n0) for x in pos(sz, F["l1z"], l0z)])
                for i in range(S["first"], S["first"] + S["count"]):
                    v = Wz @ V0[i, cz * F["p0y"] + cy] @ Wy.T
                    ph = _phase(Pn, F["b"], S["o"], org[mem[i], :3] - S["o"])
                    V1[s] += v * np.exp(2j * np.pi * ph).reshape(n1, n1)
            for j, t in enumerate(mid):
                V1[plan.n_groups + j] = leaf(t, Pn, F["b"]).reshape(n1, n1)
            cols = np.arange(py * F["l1y"], min((py + 1) * F["l1y"], F["ny"]))
            rows = np.arange(pz * F["l1z"], min((pz + 1) * F["l1z"], F["nz"]))
            assert F["bpy"] * 32 >= len(cols) and F["bpz"] * 16 >= len(rows)
            Wy = np.array([_lagrange((c - py * F["l1y"] - 0.5 * (F["l1y"] - 1)) / _half(F["l1y"]), n1) for c in cols])
            Wz = np.array([_lagrange((r - pz * F["l1z"] - 0.5 * (F["l1z"] - 1)) / _half(F["l1z"]), n1) for r in rows])
            g = (F["pix_off"] + rows[:, None] * F["ny"] + cols[None, :]).ravel()
            for s in range(plan.n_src):
                S = src[s]
                o = S["dh"].astype(float) + S["dl"]
                v = (Wz @ V1[s] @ Wy.T).ravel()
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
