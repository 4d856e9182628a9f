"""GPU: the blocks-over-planes cell mapping at the edges of its tiles (planes
of fewer cells than a block, of exactly one, of one more, one-row planes),
against the CPU oracle: steps bit for bit, FP64 statistics and diagnostics to
1e-12 (sums of the same FP64 terms in another order)."""
import numpy as np
import pytest
import torch

import _util as U
import oracle as O

pytestmark = pytest.mark.gpu

PLANES = [(5, 7), (16, 8), (43, 3), (127, 1), (257, 1), (1, 200), (33, 31)]


@pytest.mark.parametrize("lat", ["D2Q9", "D3Q19", "D3Q27"])
@pytest.mark.parametrize("nx,ny", PLANES)
def test_step_and_diagnostics(engine, dev, lat, nx, ny):
    nz = 1 if lat == "D2Q9" else 3
    f0 = U.random_state(lat, nx, ny, nz, np.float32, seed=nx + ny)
    cur = torch.from_numpy(f0).to(dev)
    nxt = torch.empty_like(cur)
    nbytes = engine.diagnostics_partials_bytes(lat, nx, ny, nz)
    part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
    out = torch.empty(5, dtype=torch.float64, device=dev)
    engine.check(engine.step_diagnostics_async(lat, "float", "MRT", cur, nxt, nx, ny, nz, 1 / 0.6, part, nbytes, out))
    torch.cuda.synchronize()
    want = O.step(f0, lat, "MRT", nx, ny, nz, 1 / 0.6, steps=1)
    assert U.same_bits(nxt.cpu().numpy(), want)
    diag = O.fluid_diagnostics64(want, lat, nx, ny, nz)
    for g, w in zip(out.cpu().numpy()[:3], diag[:3]):
        assert abs(g - w) <= 1e-12 * max(abs(w), 1e-6)


@pytest.mark.parametrize("lat", ["D2Q9", "D3Q19"])
@pytest.mark.parametrize("nx,ny", PLANES)
def test_statistics(engine, dev, lat, nx, ny):
    nz, sl = (1, "D2Q5") if lat == "D2Q9" else (3, "D3Q7")
    a = U.random_scalar(sl, nx, ny, nz, np.float64, seed=nx)
    b = U.random_scalar(sl, nx, ny, nz, np.float64, seed=ny)
    nbytes = engine.stats_partials_bytes(lat, nx, ny, nz)
    part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
    out = torch.empty(8, dtype=torch.float64, device=dev)
    engine.check(engine.reactive_stats_async(sl, "double", torch.from_numpy(a).to(dev), torch.from_numpy(b).to(dev),
                                             nx, ny, nz, 0.03, part, nbytes, out))
    torch.cuda.synchronize()
    want = O.reactive_stats(a, b, sl, nx, ny, nz, 0.03, accumulate_f64=True)
    for g, w in zip(out.cpu().numpy(), want):
        assert abs(g - w) <= 1e-12 * max(abs(w), 1e-6)
