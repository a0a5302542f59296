"""Re-walks of large trees.  From 64 MB of leaf records on (2^21 leaves) the octant walk's re-walks take the
lattice records: the walk's segments are the same floats, so the tallies and the counts of cell steps are those of
the lattice walk throughout, alone, with the jobs in walk order, and in a batch."""
import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime

from test_walks_gpu import CLOSE, EXT, phase, same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    inner = (8 ** 7 - 1) // 7                              # every node above level 7 is divided
    return runtime.tree_from_splits(A.GRID_OCTREE, EXT, np.repeat([1, 0], [inner, 8 ** 7]).astype(np.uint8))


@pytest.mark.parametrize("absorb", [False, True])
def test_large_trees_rewalk_on_the_lattice_records(grid, absorb, monkeypatch):
    assert grid.ncells * 32 >= 64 << 20
    m = models.oligo_disk(N=(2, 2, 2), npix=40, write_absorption=absorb)
    m.dustGrid = grid
    m.rho = np.random.default_rng(3).uniform(0.5, 2, (1, grid.ncells)) * 3e-24
    octant = [runtime.Context(m) for _ in range(2)]
    monkeypatch.setenv("SKG_TREE_RECORDS", "lattice")
    lattice = runtime.Context(m)
    assert octant[0].device_bytes - lattice.device_bytes == 256 * grid.ncells
    n = 30001
    want = phase(lattice, n)
    assert want[1]["scatterings"] > n // 2                 # (re-walks)
    same(phase(octant[0], n), want)
    b = runtime.Batch(max_slots=2)
    for graph in (False, True):
        for c in octant:
            c.reset_tallies()
        b.run(A.PHASE_STELLAR, [(c, [0], n, 0, n, 7) for c in octant], graph=graph)
        b.sync()
        for c in octant:
            assert np.allclose(c.read_instrument(0)[0], want[0][0], **CLOSE)
    b.close()
    n = 800001
    same(phase(octant[0], n), phase(lattice, n))           # (in walk order)
    for c in octant + [lattice]:
        c.close()
