"""Phases on a caller's stream: reads, resets and the next phase go on behind their last launch."""
import numpy as np
import pytest

from skirt7_b200 import _abi as A
from skirt7_b200 import runtime

from test_walks_gpu import CLOSE, model

pytestmark = pytest.mark.gpu


def test_reads_and_phases_behind_a_callers_stream():
    import torch
    ctx = runtime.Context(model("octree"))
    n = 60001
    ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=2)
    assert sum(ctx.phase_times()[:2]) > 0               # (without a sync before it)
    want, labs = ctx.read_instrument(0)[0].copy(), ctx.read_absorption()[0]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for i in range(6):
        ctx.reset_tallies()
        ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=2, stream=streams[i % 2].cuda_stream)
        if i % 3 == 0:
            assert np.allclose(ctx.read_absorption()[0], labs, **CLOSE)
        elif i % 3 == 1:
            out = torch.zeros(want.size, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ctx.read_instrument_device(0, out.data_ptr(), stream=streams[(i + 1) % 2].cuda_stream)
            streams[(i + 1) % 2].synchronize()
            assert np.allclose(out.cpu().numpy().reshape(want.shape), want, **CLOSE)
        else:                                            # the same packets once more on the other stream
            ctx.run_phase(A.PHASE_STELLAR, [0], n, seed=2, stream=streams[(i + 1) % 2].cuda_stream)
            assert np.allclose(ctx.read_instrument(0)[0], 2 * want, **CLOSE)
    assert ctx.counters()["errors"] == 0
    ctx.close()
