"""Batches of the default capacity (64 slots): the walks of both precisions launch with any number of
slots in use, and give each simulation the tallies that it gets alone (packets draw from streams keyed by
their index; the sums differ by the order of the FP64 atomics)."""
import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime

from helpers import cell_center_density
from test_walks_gpu import CLOSE, model

pytestmark = pytest.mark.gpu


def alone(ctx, n, seed, precision):
    ctx.reset_tallies()
    ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=seed, precision=precision)
    ctx.sync()
    return ctx.read_instrument(0)[0].copy()


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("grid", ["cartesian", "octree", "kdtree", "voronoi"])
@pytest.mark.parametrize("n", [30001, 701])     # waves on every grid; the tail pass alone
def test_one_simulation_in_a_batch_of_default_capacity(grid, precision, n):
    ctx = runtime.Context(model(grid))
    want = alone(ctx, n, 3, precision)
    b = runtime.Batch()
    for graph in (False, True, True):
        ctx.reset_tallies()
        ctx.sync()
        b.run(A.PHASE_STELLAR, [(ctx, [0], n, 0, n, 3)], precision=precision, graph=graph)
        b.sync()
        assert np.allclose(ctx.read_instrument(0)[0], want, **CLOSE)
    assert b.counters()["errors"] == 0
    b.close()
    ctx.close()


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
def test_every_slot_in_use_and_fewer_on_the_same_graph(precision):
    ctxs = []
    for i in range(64):
        m = models.oligo_disk(N=(6 + i % 5, 7, 5), npix=12)
        m.rho = np.random.default_rng(i).uniform(0.5, 2, (1, (6 + i % 5) * 35)) * 1e-24
        ctxs.append(runtime.Context(m))
    n = 401
    want = [alone(c, n, 100 + i, precision) for i, c in enumerate(ctxs)]
    assert all(w.sum() > 0 for w in want)
    b = runtime.Batch()
    for graph, slots in ((False, 64), (True, 64), (True, 55), (True, 57), (False, 57)):
        for c in ctxs:
            c.reset_tallies()
            c.sync()
        b.run(A.PHASE_STELLAR, [(c, [0], n, 0, n, 100 + i) for i, c in enumerate(ctxs[:slots])], precision=precision,
              graph=graph)
        b.sync()
        for i, c in enumerate(ctxs):
            got = c.read_instrument(0)[0]
            assert np.allclose(got, want[i] if i < slots else 0, **CLOSE), (graph, slots, i)
    b.close()
    for c in ctxs:
        c.close()


def test_a_replay_goes_on_as_it_was_captured():
    """A captured phase with absorption on a pool of 2^16; a smaller direct phase without, on another walk; the
    graph again, for a simulation that takes more waves than were captured (thick dust)."""
    def ctx(tau, absorb):
        m = models.oligo_disk(N=(12, 11, 9), tauV=tau, npix=12, write_absorption=absorb)
        m.rho = cell_center_density(m)
        return runtime.Context(m)
    thin, thick, plain = ctx(0.01, True), ctx(200.0, True), ctx(1.0, False)
    n = 60000
    want = alone(thick, n, 5, A.PREC_FP32)
    absorbed = thick.read_absorption()[0]
    b = runtime.Batch(max_slots=2)
    b.run(A.PHASE_STELLAR, [(thin, [0], n, 0, n, 5)], graph=True)
    b.sync()
    captured = b.counters()["waves"]
    for _ in range(2):
        b.run(A.PHASE_STELLAR, [(plain, [0], 23000, 0, 23000, 5)], precision=A.PREC_FP64, pool=21000)
        b.sync()
        thick.reset_tallies()
        thick.sync()
        b.run(A.PHASE_STELLAR, [(thick, [0], n, 0, n, 5)], graph=True)
        b.sync()
        assert np.allclose(thick.read_instrument(0)[0], want, **CLOSE)
        assert np.allclose(thick.read_absorption()[0], absorbed, **CLOSE)
    assert captured > 1 and b.counters()["errors"] == 0
    b.close()


@pytest.mark.parametrize("tail", ["0", "16"])
def test_replays_that_take_more_waves_than_the_last(tail, monkeypatch):
    """A captured phase that ends within its waves, replayed as it is and then for thick dust: the host sees the
    replay's own counters, not those that the last one left, and adds waves."""
    monkeypatch.setenv("SKG_TAIL_DIV", tail)
    def ctx(tau):
        m = models.oligo_disk(N=(12, 11, 9), tauV=tau, npix=12, write_absorption=False)
        m.rho = cell_center_density(m)
        return runtime.Context(m)
    thin, thick = ctx(1e-4), ctx(10.0)
    n, pool = 60000, 6000
    want = alone(thick, n, 5, A.PREC_FP32), alone(thin, n, 5, A.PREC_FP32)
    b = runtime.Batch(max_slots=2)
    for i, c in enumerate((thin, thin, thick, thin, thin, thick)):
        c.reset_tallies()
        b.run(A.PHASE_STELLAR, [(c, [0], n, 0, n, 5)], graph=True, pool=pool)
        b.sync()
        assert np.allclose(c.read_instrument(0)[0], want[c is thin], **CLOSE), i
        waves = b.counters()["waves"]
        if i < 2:
            captured = waves
        elif i == 2:
            assert waves > captured or tail != "0"
    assert b.counters()["errors"] == 0 and b.counters()["packets"] == 6 * n
    b.close()
