"""The cumulative cell luminosities that dust packets are launched from (NR::cdf, NR.hpp:388-394), against numpy: from 0
to exactly 1, within [0, 1], for cell counts around the tiles and for luminosities down to denormal numbers."""
import ctypes as C

import numpy as np
import pytest

from skirt7_b200 import _abi as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 31, 32, 257, 2047, 2048, 2049, 5000, 600001])
def test_cumulative_luminosities(nc):
    import torch
    lib = A.load()
    tiles = lib._ZN3skg14emission_tilesEi
    tiles.restype, tiles.argtypes = C.c_size_t, [C.c_int]
    sources = lib._ZN3skg23launch_emission_sourcesEiiPKdPdS2_S2_P11CUstream_st
    sources.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 5
    rng = np.random.default_rng(nc)
    L = rng.uniform(0, 1, (5, nc)) ** 8 * 1e36
    L[1] *= rng.random(nc) < 0.1                            # most cells dark
    L[1, 0] = 1.0
    L[2, max(1, nc // 2):] = 0                              # the end of the row dark
    L[3] = np.floor(rng.uniform(1, 1000, nc)) * 5e-324      # denormal luminosities
    L[4] = 0
    x = torch.from_numpy(L).cuda()
    cdf = torch.full((5, nc + 1), -1.0, dtype=torch.float64, device="cuda")
    tot = torch.full((5,), -1.0, dtype=torch.float64, device="cuda")
    sums = torch.zeros(5 * tiles(nc), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert sources(5, nc, x.data_ptr(), cdf.data_ptr(), tot.data_ptr(), sums.data_ptr(), None) == 0
    torch.cuda.synchronize()
    cdf, tot = cdf.cpu().numpy(), tot.cpu().numpy()
    want = np.cumsum(L.astype(np.longdouble), axis=1)
    # sums of nc non-negative terms, in any order: nc roundings of 2^-53
    bound = (nc + 2) * 2.0 ** -53
    assert np.all(np.abs(tot - want[:, -1]) <= bound * want[:, -1])
    assert tot[4] == 0 and np.all(cdf[4] == 0)
    for c, w in zip(cdf[:4], want[:4]):
        assert c[0] == 0 and c[-1] == 1 and c.min() >= 0 and c.max() <= 1
        assert np.all(np.abs(c[1:] - w / w[-1]) <= 2 * bound * (w / w[-1]))
        assert np.all(np.diff(c) >= -2 * bound)
