"""GPU: the 16-bit step at the edges of its four-cell words (rows of one word,
rows of an odd number of words, planes that do not fill a block).

The periodic step commutes with tiling: a box repeated along x steps to the
repeated result, and since the words and the pairs of a row do not move under a
shift by a multiple of 4 cells, the codes must be equal bit for bit, stochastic
rounding included. So every row length is held to the same state in rows of
another length, and the face planes of a slab are covered by the slab tests."""
import numpy as np
import pytest
import torch

import _util as U

pytestmark = pytest.mark.gpu

FMTS = ("f16s", "bf16s", "e3m12s", "q15s")


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("lat,op", [("D2Q9", "MRT"), ("D2Q9", "RLBM"), ("D3Q19", "BGK"), ("D3Q19", "TRT"),
                                    ("D3Q19", "MRT"), ("D3Q19", "RLBM"), ("D3Q27", "TRT"), ("D3Q27", "MRT")])
@pytest.mark.parametrize("nx,copies", [(4, 5), (12, 3), (20, 4), (100, 2)])
def test_step_commutes_with_tiling(engine, dev, fmt, lat, op, nx, copies):
    ny, nz = (9, 1) if lat == "D2Q9" else (5, 3)
    q = U.Q_OF[lat]
    f = torch.from_numpy(U.random_state(lat, nx, ny, nz, np.float32, seed=nx)).to(dev)
    h0 = torch.empty((q, nz, ny, nx), dtype=torch.int16, device=dev)
    engine.check(engine.encode_shifted_async(lat, fmt, "float", f, h0, nx, ny, nz, 1.0))
    wide0 = h0.repeat(1, 1, 1, copies).contiguous()
    h1, wide1 = torch.full_like(h0, -1), torch.full_like(wide0, -1)
    engine.check(engine.step_shifted_async(lat, fmt, op, h0, h1, nx, ny, nz, 1 / 0.6, 1.0))
    engine.check(engine.step_shifted_async(lat, fmt, op, wide0, wide1, nx * copies, ny, nz, 1 / 0.6, 1.0))
    torch.cuda.synchronize()
    assert torch.equal(h1.repeat(1, 1, 1, copies), wide1)
