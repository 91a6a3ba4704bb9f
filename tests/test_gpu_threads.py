"""Host threads that run one kernel with different amounts of shared memory at
the same time, each on its own stream: the sizes one sets must not stop
another's launch, and every result is the one the thread gets alone."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from mosaic_gb300 import _lib, engine, propagation, workloads
from mosaic_gb300.tables import ScatteringTables

pytestmark = pytest.mark.gpu


def _together(jobs, runs):
    """Every job alone, then all of them `runs` times side by side."""
    alone = [j() for j in jobs]
    torch.cuda.synchronize()
    wrong, gate = [], threading.Barrier(len(jobs))

    def work(j, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                for _ in range(runs):
                    got = j()
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(got, want):
                        wrong.append("another result")
        except Exception as e:              # a launch refused
            wrong.append(repr(e))
    ts = [threading.Thread(target=work, args=(j, a)) for j, a in zip(jobs, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong, (len(wrong), wrong[0])


def test_fp64_sums_of_one_and_sixteen_species(cuda):
    tab = ScatteringTables()
    wk = np.asarray(tab.f0["Cu"], np.float64).ravel()[:11].astype(np.float32)
    k = 5.0e10
    rng = np.random.default_rng(0)
    phys = engine.physics(k)
    xyz = np.stack([np.full(64, 1.0), np.arange(64) * 1e-5, np.zeros(64)])

    def job(ns):
        table = engine.SpeciesTable([f"s{i}" for i in range(ns)], np.repeat(wk[None], ns, 0),
                                    np.full(ns, 29.0, np.float32), np.zeros(ns, complex))
        sp = torch.tensor(np.arange(160) % ns, dtype=torch.int32, device=cuda)
        atoms = engine.Atoms(torch.tensor(rng.uniform(-5e-9, 5e-9, (160, 3)), device=cuda), sp,
                             torch.ones((160, 2), device=cuda), np.bincount(np.arange(160) % ns, minlength=ns), table)
        pix = engine.Pixels(xyz, 64, 1, phys, device=cuda)
        return lambda: engine.run_plain(atoms, pix, phys)
    _together([job(1), job(16), job(2), job(16)], 400)


def test_fp64_launches_are_not_refused(cuda):
    """The same two sizes as bare calls in a row, which meet between one's
    setting of its limit and its launch."""
    L = _lib.load()
    wk = np.asarray(ScatteringTables().f0["Cu"], np.float64).ravel()[:11].astype(np.float32)
    phys = engine.physics(5.0e10)
    pix = engine.Pixels(np.stack([np.full(8, 1.0), np.arange(8) * 1e-5, np.zeros(8)]), 8, 1, phys, device=cuda)
    bad = []

    def work(ns):
        table = engine.SpeciesTable([f"s{i}" for i in range(ns)], np.repeat(wk[None], ns, 0),
                                    np.full(ns, 29.0, np.float32), np.zeros(ns, complex))
        pos = torch.zeros((32, 3), dtype=torch.float64, device=cuda)
        sp = torch.tensor(np.arange(32) % ns, dtype=torch.int32, device=cuda)
        amp = torch.ones((32, 2), device=cuda)
        out = torch.zeros((8, 2), dtype=torch.float64, device=cuda)
        ws = torch.empty(L.mk_sum_workspace_size(8, 1), dtype=torch.uint8, device=cuda)
        s = torch.cuda.Stream()
        tab = table.abi()
        args = (32, pos.data_ptr(), sp.data_ptr(), amp.data_ptr(), ctypes.byref(tab), ctypes.byref(phys),
                ctypes.byref(pix.abi), 1, out.data_ptr(), 0, ws.data_ptr(), ws.numel(), s.cuda_stream)
        gate.wait()
        for i in range(20000):
            if L.mk_kin_plain_f64(*args) != 0:
                bad.append(L.mk_last_error())
            if i % 500 == 499:
                s.synchronize()
        s.synchronize()
    gate = threading.Barrier(4)
    ts = [threading.Thread(target=work, args=(ns,)) for ns in (1, 16, 1, 16)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, (len(bad), bad[0])


def test_propagations_of_two_sizes(cuda):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)

    def job(n):
        E = torch.randn((n, 64), generator=g, device=cuda).to(torch.complex64)
        return lambda: propagation.propagate(E, 1e-6, 1e-6, 1e-3, 1.24e-10)[0]
    _together([job(400), job(1800), job(400), job(1800)], 150)


def test_node_sums_of_two_tile_sizes(cuda):
    w = workloads.fcc_cu_32k(cells=14, npix=64)
    B = w.beam
    phys = B.physics(**w.sc_kwargs)
    atoms = B.stage_atoms(w.sample, w.stage, device=cuda)
    pix = engine.Pixels(np.asarray(w.detector.pixel_coordinates) / 1e10, 64, 64, phys, device=cuda)

    def job(T):
        tiles = engine.Tiles(atoms, B.k, T, device=cuda)
        plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0, group_tiles=0)
        assert plan is not None and plan.wide is None
        factor = pix.factor_table(atoms.table, phys)
        return lambda: engine.run_nodes(plan, tiles, pix, phys, atoms.table, factor=factor)
    _together([job(128), job(4096), job(256), job(4096)], 300)
