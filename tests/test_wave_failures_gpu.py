"""Failures reported by the waves: phases of more packets than the tail pass alone takes (20000 on Cartesian grids,
2^13 on others), to the end in waves and with the tail pass behind them, alone and in a batch.  As in the phases of
few packets, a finite density whose optical depth overflows gives SKG_ERR_NAN_TAU and a step budget of one cell
SKG_ERR_STEP_BUDGET; the context goes on."""
import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime

from helpers import cell_center_density
from test_walks_gpu import EXT

pytestmark = pytest.mark.gpu
N = 30000


def _model(grid, bad=False):
    m = models.oligo_disk(N=(20, 20, 10), npix=32)
    if grid == "octree":
        m.dustGrid = runtime.tree_from_splits(A.GRID_OCTREE, EXT, np.repeat([1, 0], [73, 512]).astype(np.uint8))
        m.rho = np.full((1, 512), 1e-25)
    else:
        m.rho = cell_center_density(m)
    if bad:
        m.rho[0, ::7] = 1e300
    return m


@pytest.fixture(params=["0", "16"])
def tail(request, monkeypatch):
    monkeypatch.setenv("SKG_TAIL_DIV", request.param)


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("grid", ["cartesian", "octree"])
def test_overflowing_optical_depth(grid, precision, tail):
    ctx = runtime.Context(_model(grid, True))
    ctx.run_phase(A.PHASE_STELLAR, [0], N, 0, N, seed=3, precision=precision)
    with pytest.raises(A.SkirtError) as e:
        ctx.sync(60000)
    assert e.value.code == A.SKG_ERR_NAN_TAU
    assert ctx.phase_times()[2] > 0 and ctx.counters()["errors"] > 0
    b = runtime.Batch(max_slots=2)
    b.run(A.PHASE_STELLAR, [(ctx, [0], N, 0, N, 3)], precision=precision)
    with pytest.raises(A.SkirtError) as e:
        b.sync(60000)
    assert e.value.code == A.SKG_ERR_NAN_TAU
    ok = runtime.Context(_model(grid))
    b.run(A.PHASE_STELLAR, [(ok, [0], N, 0, N, 3)], precision=precision)
    b.sync(60000)
    ok.run_phase(A.PHASE_STELLAR, [0], N, 0, N, seed=3, precision=precision)
    ok.sync(60000)
    assert ok.phase_times()[2] > 0 and ok.counters()["errors"] == 0 and ok.counters()["packets"] == N
    b.close()
    ctx.close()
    ok.close()


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("grid", ["cartesian", "octree"])
def test_step_budget(grid, precision, tail):
    ctx = runtime.Context(_model(grid))
    ctx.run_phase(A.PHASE_STELLAR, [0], N, 0, N, seed=4, max_steps=1, precision=precision)
    with pytest.raises(A.SkirtError) as e:
        ctx.sync(60000)
    assert e.value.code == A.SKG_ERR_STEP_BUDGET
    assert ctx.phase_times()[2] > 0 and ctx.counters()["errors"] > 0
    ctx.reset_tallies()
    ctx.run_phase(A.PHASE_STELLAR, [0], N, 0, N, seed=4, precision=precision)
    ctx.sync(60000)
    c = ctx.counters()
    assert c["errors"] == 0 and c["packets"] == N
    ctx.close()
