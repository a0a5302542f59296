"""Simulations without dust, whose packets have no walk where no frame sees them: every packet is launched,
over any pool, with and without the tail pass."""
import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime
from skirt7_b200.scene import DEG, KPC, MPC, FrameInstrument

from test_walks_gpu import CLOSE, model

pytestmark = pytest.mark.gpu


def narrow(fov):
    m = models.oligo_disk(N=(6, 5, 4), npix=8)
    m.dustComps, m.rho = [], None
    m.instruments = [FrameInstrument(10 * MPC, 30 * DEG, 4, 4, fov, fov)]
    return runtime.Context(m)


@pytest.mark.parametrize("tail", [True, False])
@pytest.mark.parametrize("fov", [1e-3 * KPC, 8 * KPC])
def test_every_packet_is_launched(fov, tail, monkeypatch):
    n = 5003
    ctx = narrow(fov)
    ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=3)
    ctx.sync()
    want = ctx.read_instrument(0)[0].copy()
    if not tail:
        monkeypatch.setenv("SKG_TAIL_DIV", "0")
    for pool in (1000, 32):
        ctx.reset_tallies()
        ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=3, pool=pool)
        ctx.sync()
        c = ctx.counters()
        assert c["packets"] == n and c["errors"] == 0, pool
        assert np.allclose(ctx.read_instrument(0)[0], want, **CLOSE)
    ctx.close()


def test_in_a_batch_before_a_simulation_with_dust():
    blank, dusty = narrow(1e-3 * KPC), runtime.Context(model("cartesian", False))
    n = 4001
    dusty.run_phase(A.PHASE_STELLAR, [0], n, seed=4)
    dusty.sync()
    want = dusty.read_instrument(0)[0].copy()
    dusty.reset_tallies()
    dusty.sync()
    b = runtime.Batch(max_slots=2)
    b.run(A.PHASE_STELLAR, [(blank, [0], n, 0, n, 3), (dusty, [0], n, 0, n, 4)], pool=64)
    b.sync()
    c = b.counters()
    assert c["packets"] == 2 * n and c["errors"] == 0
    assert np.allclose(dusty.read_instrument(0)[0], want, **CLOSE)
    b.close()
