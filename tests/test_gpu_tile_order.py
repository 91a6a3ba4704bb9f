"""The tile order of samples whose bounding box is mostly empty: tiles stay as
compact as those of the same atoms in a box of their own.

The bound: the tiles of a cluster in a box of its own have a median radius r.
With the atoms of both clusters interleaved at random, a tile may differ in
where the curve is cut, so 1.3 r (in input order the tiles span the cluster:
2.5 r and more at these sizes)."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine
from mosaic_gb300.tables import ScatteringTables

pytestmark = pytest.mark.gpu


def _tiles(cuda, pos, T):
    table = engine.SpeciesTable.build(["Cu", "Ni", "Na"], ScatteringTables(), 10000.0)
    sp = (np.arange(len(pos)) % 3).astype(np.int32)
    atoms = engine.atoms_lab(pos.astype(np.float32), sp, np.eye(3), np.zeros(3), table, device=cuda)
    return engine.Tiles(atoms, 5e10, T, device=cuda)


@pytest.mark.parametrize("n, side, apart, T", [
    (30000, 100.0, 1.0e5, 128),         # two particles 10 um apart along the diagonal
    (60000, 150.0, 2.0e4, 512),
    (400000, 300.0, 1.0e5, 512),        # 32-bit keys
])
def test_two_particles_far_apart(cuda, n, side, apart, T):
    rng = np.random.default_rng(n)
    one = (rng.random((n, 3)) - 0.5) * side
    alone = np.median(engine.origins_host(_tiles(cuda, one, T))[:, 3])
    both = np.concatenate([one, one + apart / np.sqrt(3.0)])[rng.permutation(2 * n)]
    t = _tiles(cuda, both, T)
    r = engine.origins_host(t)[:, 3]
    assert t.n_tiles == sum(-(-int(c) // T) for c in t.counts)
    assert np.median(r) <= 1.3 * alone, (np.median(r), alone)


def test_an_atom_far_off(cuda):
    rng = np.random.default_rng(1)
    one = (rng.random((90000, 3)) - 0.5) * 200.0
    alone = np.median(engine.origins_host(_tiles(cuda, one, 512))[:, 3])
    one[17] = [5e5, 4e5, -3e5]
    assert np.median(engine.origins_host(_tiles(cuda, one, 512))[:, 3]) <= 1.3 * alone


def test_build_on_another_stream_and_read_back(cuda):
    rng = np.random.default_rng(2)
    pos = (rng.random((20000, 3)) * 100.0)
    a = _tiles(cuda, pos, 256)
    table = a.table
    sp = (np.arange(len(pos)) % 3).astype(np.int32)
    atoms = engine.atoms_lab(pos.astype(np.float32), sp, np.eye(3), np.zeros(3), table, device=cuda)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    b = engine.Tiles(atoms, 5e10, 256, device=cuda, stream=s)
    torch.cuda.synchronize()
    assert np.array_equal(engine.origins_host(a), engine.origins_host(b))
    assert np.array_equal(engine.origins_host(b), b.origin.cpu().numpy())
    assert torch.equal(a.pos, b.pos)


@pytest.mark.parametrize("apart, again", [(0.0, False), (3.0e3, False), (2.0e4, True)])
def test_built_again_only_where_it_pays(cuda, monkeypatch, apart, again):
    """A few dozen atoms a cell leave the tiles as they are; hundreds do not."""
    rng = np.random.default_rng(3)
    one = (rng.random((30000, 3)) - 0.5) * 70.0
    pos = np.concatenate([one, one + apart / np.sqrt(3.0)])[rng.permutation(60000)]
    L = engine._require_cuda()
    keys = []

    class Spy:
        def __getattr__(self, name):
            return getattr(L, name)

        def mk_tiles_build_keys(self, *a):
            keys.append(a[8])
            return L.mk_tiles_build_keys(*a)
    table = engine.SpeciesTable.build(["Cu"], ScatteringTables(), 10000.0)
    atoms = engine.atoms_lab(pos.astype(np.float32), np.zeros(60000, np.int32), np.eye(3), np.zeros(3), table,
                             device=cuda)
    monkeypatch.setattr(engine, "_require_cuda", lambda: Spy())
    engine.Tiles(atoms, 5e10, 512, device=cuda)
    assert keys == ([0, 1] if again else [0])
