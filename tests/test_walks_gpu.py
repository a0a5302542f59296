"""The traversal's forms against one another: packets draw from streams keyed by their index, so the same
phase gives the same tallies, up to the summation order of the FP64 atomics, however its jobs are ordered,
chunked, and walked.  And the tables that the phases hand on: the absorbed luminosities as they are read
back, the cells' temperatures and the cumulative luminosities that dust packets are launched from."""
import math

import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime
from skirt7_b200.scene import DEG, KPC, MPC, CartesianDustGrid, FrameInstrument, FullInstrument

from helpers import cell_center_density

pytestmark = pytest.mark.gpu
EXT = (-20 * KPC, -20 * KPC, -2 * KPC, 20 * KPC, 20 * KPC, 2 * KPC)
# sums of at most a few thousand positive FP64 terms per bin, in any order: 1e-12 is over a thousand roundings
CLOSE = dict(rtol=1e-11, atol=0)


def model(grid, absorb=True, fraction=1e-4):
    m = models.oligo_disk(N=(40, 40, 20), npix=40, write_absorption=absorb)
    if grid == "octree":
        m.dustGrid = runtime.build_tree(m, A.GRID_OCTREE, EXT, minLevel=2, maxLevel=8, maxMassFraction=fraction)
    elif grid == "kdtree":
        m.dustGrid = runtime.build_tree(m, A.GRID_BINTREE, EXT, minLevel=6, maxLevel=21, maxMassFraction=fraction)
    elif grid == "voronoi":
        rng = np.random.default_rng(5)
        lo, hi = np.array(EXT[:3]), np.array(EXT[3:])
        m.dustGrid = runtime.build_voronoi(lo + rng.random((17000, 3)) * (hi - lo), EXT)
    else:
        m.rho = cell_center_density(m)
    return m


def phase(ctx, n, seed=7, **kw):
    ctx.reset_tallies()
    ctx.run_phase(A.PHASE_STELLAR, np.arange(ctx.nlambda), n, seed=seed, **kw)
    ctx.sync()
    out = [x for i in range(len(ctx.model.instruments)) for x in ctx.read_instrument(i) if x is not None]
    if ctx.model.writeAbsorption:
        out.append(ctx.read_absorption()[0])
    c = ctx.counters()
    assert c["errors"] == 0
    return out, {k: c[k] for k in ("packets", "steps", "traversals", "scatterings", "peeloffs", "nbr_scanned")}


def same(a, b):
    assert a[1] == b[1]
    for x, y in zip(a[0], b[0]):
        assert np.allclose(x, y, **CLOSE), np.nanmax(np.abs(x - y) / np.maximum(np.abs(y), 1e-300))


@pytest.mark.parametrize("grid", ["cartesian", "octree", "kdtree", "voronoi"])
def test_small_phases_and_pools(grid, monkeypatch):
    """The tail pass alone (up to 2^13 packets, Cartesian 20000) against waves, and waves over pools whose
    sizes do not fill a warp, a chunk or a block."""
    ctx = runtime.Context(model(grid))
    for n in (1, 33, 600):
        tail = phase(ctx, n)
        monkeypatch.setenv("SKG_TAIL_DIV", "0")
        for pool in (0, 1, 31, 257):
            if n <= 33 or pool != 1:
                same(phase(ctx, n, pool=pool), tail)
        monkeypatch.delenv("SKG_TAIL_DIV")
    ctx.close()


@pytest.mark.parametrize("grid,absorb", [("octree", False), ("kdtree", True), ("voronoi", False), ("voronoi", True)])
def test_spatial_order(grid, absorb):
    """Jobs walked in spatial order (from 786432 records on, grids of 8 MB of records) and as appended."""
    ctx = runtime.Context(model(grid, absorb, fraction=3e-6))
    assert ctx.ncells * (512 if grid == "voronoi" else 32) >= 8 << 20
    n = 800001
    same(phase(ctx, n), phase(ctx, n, pool=300007))
    ctx.close()


@pytest.mark.parametrize("grid", ["octree", "kdtree"])
@pytest.mark.parametrize("absorb", [False, True])
def test_octant_records(grid, absorb, monkeypatch):
    """The walk on the octant records is the walk on the lattice records, also in a batch of both."""
    m = model(grid, absorb)
    m.instruments.append(FrameInstrument(10 * MPC, 0.0, 40, 40, 40 * KPC, 40 * KPC))       # along an axis
    octant = runtime.Context(m)
    monkeypatch.setenv("SKG_TREE_RECORDS", "lattice")
    lattice = runtime.Context(m)
    a = phase(lattice, 60001)
    same(phase(octant, 60001), a)
    b = runtime.Batch(max_slots=2)
    for c in (octant, lattice):
        c.reset_tallies()
    b.run(A.PHASE_STELLAR, [(c, [0], 60001, 0, 60001, 7) for c in (octant, lattice)])
    b.sync()
    for c in (octant, lattice):
        assert np.allclose(c.read_instrument(0)[0], a[0][0], **CLOSE)
    b.close()


@pytest.mark.parametrize("views", [1, 4, 5])
def test_voronoi_lists_per_direction(views):
    """With up to four observers the peel-offs scan the planes ahead of their direction, with more the full
    lists: the first observer's frame does not change."""
    m = model("voronoi", False)
    m.instruments = [FrameInstrument(10 * MPC, (88 - 22 * i) * DEG, 40, 40, 40 * KPC, 40 * KPC) for i in range(views)]
    ctx = runtime.Context(m)
    got = phase(ctx, 50000)
    m.instruments = [m.instruments[0]] + [FrameInstrument(10 * MPC, (3 + i) * DEG, 8, 8, 40 * KPC, 40 * KPC) for i in range(5)]
    full = runtime.Context(m)
    assert np.allclose(got[0][0], phase(full, 50000)[0][0], **CLOSE)


def test_detection_alone_and_in_a_batch():
    """SED bins summed per warp and block (one simulation) and added directly (a batch)."""
    m = model("cartesian")
    m.instruments.append(FullInstrument(scatteringLevels=2, distance=10 * MPC, inclination=30 * DEG, pixelsX=33, pixelsY=31,
                                        fieldOfViewX=40 * KPC, fieldOfViewY=40 * KPC))
    ctxs = [runtime.Context(m) for _ in range(2)]
    alone = phase(ctxs[0], 30001, seed=3)
    b = runtime.Batch(max_slots=2)
    for c in ctxs:
        c.reset_tallies()
    b.run(A.PHASE_STELLAR, [(c, [0], 30001, 0, 30001, 3) for c in ctxs])
    b.sync()
    for c in ctxs:
        out = [x for i in range(len(m.instruments)) for x in c.read_instrument(i) if x is not None]
        for x, y in zip(out, alone[0]):
            assert np.allclose(x, y, **CLOSE)
    b.close()


@pytest.mark.parametrize("nl", [1, 3, 33])
def test_absorption_layout(nl):
    """[cell][wavelength], for cell counts and wavelengths off the tiles of the transpose: a phase of one
    wavelength fills its column alone, with what the phase of all wavelengths puts there."""
    m = models.oligo_disk(N=(7, 5, 3), npix=8, wavelengths=[(0.4 + 0.01 * i) * 1e-6 for i in range(nl)])
    ctx = runtime.Context(m)
    full = phase(ctx, 3000)[0][-1]
    assert full.shape == (105, nl) and np.all(full.sum(0) > 0)
    for ell in {0, nl // 2, nl - 1}:
        ctx.reset_tallies()
        ctx.run_phase(A.PHASE_STELLAR, [ell], 3000, seed=7)
        one = ctx.read_absorption()[0]
        assert np.allclose(one[:, ell], full[:, ell], **CLOSE)
        assert np.count_nonzero(np.delete(one, ell, axis=1)) == 0
    ctx.close()


@pytest.mark.parametrize("nx", [1, 31, 2048, 4100])
def test_dust_sources(nx):
    """Temperatures from the absorbed luminosities (DustMix.cpp:674-697), restated in numpy, and dust packets
    launched from the cells in proportion to what they absorbed, for cell counts around the tiles of the
    cumulative sums: a row of thin cells seen from above shows each part's share of the emission."""
    m = models.pan_disk(nlambda=5, lmin=0.1e-6, lmax=1000e-6, tauV=1e-4, inclinations=(0,), npix=10, dust_emission=True,
                        write_absorption=True)
    m.dustGrid = CartesianDustGrid(EXT[0], EXT[3], EXT[1], EXT[4], EXT[2], EXT[5], nx, 1, 1)
    m.rho = np.random.default_rng(nx).uniform(0.5, 2, (1, nx)) * 1e-30
    m.dustEmissionBias = 0.0
    ctx = runtime.Context(m)
    ctx.run_phase(A.PHASE_STELLAR, np.arange(5), 200000, seed=2)
    T = ctx.calc_dust_emission()
    labs = ctx.read_absorption()[0]
    mix, lam, dl = m.dustComps[0].mix, m.wavelengthGrid.lambdav, m.wavelengthGrid.dlambdav
    kabs = mix.kappaext * (1 - mix.albedo)
    vol = (EXT[3] - EXT[0]) * (EXT[4] - EXT[1]) * (EXT[5] - EXT[2]) / nx
    pa = labs.sum(1) / (m.rho[0] * 4 * math.pi * vol)
    q = 500.0 ** (1 / 999)
    Tv = (1 - q ** np.arange(1001)) / (1 - q ** 1000) * 5000
    with np.errstate(over="ignore", divide="ignore"):
        table = np.concatenate([[0], [(kabs * models.planck(lam, t) * dl).sum() for t in Tv[1:]]])
    p = np.clip(np.searchsorted(table, pa, side="right") - 1, 0, 999)
    want = Tv[p] + (pa - table[p]) / (table[p + 1] - table[p]) * (Tv[p + 1] - Tv[p])
    assert np.allclose(T, want, rtol=1e-9, atol=0)
    # the share of each tenth of the row, per wavelength: n packets of equal weight, binomial
    cube0 = ctx.read_instrument(0)[0].copy()
    n = 100000
    ctx.run_phase(A.PHASE_DUST_EMISSION, np.arange(5), n, seed=4)
    cube = (ctx.read_instrument(0)[0] - cube0)[0]
    # (seen from above, the image's rows run along -x)
    shares = cube.sum(2)[:, ::-1] / np.maximum(cube.sum((1, 2)), 1e-300)[:, None]
    edges = np.linspace(0, 10, nx + 1)
    overlap = np.maximum(0, np.minimum(edges[1:, None], np.arange(1, 11)) - np.maximum(edges[:-1, None], np.arange(10)))
    for ell in range(5):
        with np.errstate(over="ignore"):
            w = kabs[ell] * models.planck(lam[ell], T[:, None]) * dl[ell]
            tot = (kabs * models.planck(lam, T[:, None]) * dl).sum(1)
        L = labs.sum(1) * w[:, 0] / tot
        # (cube0 is subtracted from sums that hold it: 1e-9 of the stellar flux is far below the noise)
        if L.sum() > 1e-6 * labs.sum():
            expect = ((L / L.sum())[:, None] * overlap / (edges[1] - edges[0])).sum(0)
            assert np.all(np.abs(shares[ell] - expect) < 6 * np.sqrt(expect / n) + 1e-4), ell
    ctx.close()
