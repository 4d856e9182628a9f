"""GPU: the 16-bit fluid + A + B -> C step four cells per thread against one
cell per thread. Whole words per row in word-aligned buffers take the first,
buffers one code off the alignment the second; the same state must give the
same codes bit for bit, and the same statistics to 1e-12 (FP64 sums of the same
terms in another order)."""
import numpy as np
import pytest
import torch

import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["f16s", "bf16s", "e3m12s", "q15s"])
@pytest.mark.parametrize("fl", ["D2Q9", "D3Q19"])
@pytest.mark.parametrize("op,nx,ny", [("BGK", 4, 3), ("TRT", 100, 6), ("MRT", 12, 50), ("TRT", 516, 1)])
@pytest.mark.parametrize("stats", [False, True])
def test_words_match_single_cells(engine, dev, fmt, fl, op, nx, ny, stats):
    nz, sl = (1, "D2Q5") if fl == "D2Q9" else (3, "D3Q7")
    n = nx * ny * nz
    words, off = [], []
    for lat, t, ref in ((fl, U.random_state(fl, nx, ny, nz, np.float32, seed=8), 1.0),
                        (sl, U.random_scalar(sl, nx, ny, nz, np.float32, seed=9), 0.5),
                        (sl, U.random_scalar(sl, nx, ny, nz, np.float32, seed=10), 0.5)):
        h = torch.empty((t.shape[0], n), dtype=torch.int16, device=dev)
        engine.check(engine.encode_shifted_async(lat, fmt, "float", torch.from_numpy(t).to(dev), h, nx, ny, nz, ref))
        h_off = torch.empty(h.numel() + 1, dtype=torch.int16, device=dev)[1:].view(h.shape)
        h_off.copy_(h)
        words.append(h)
        off.append(h_off)
    nbytes = engine.stats_partials_bytes(fl, nx, ny, nz)
    rows = []
    for state in (words, off):
        nxt = [torch.empty(h.numel() + 1, dtype=torch.int16, device=dev)[(1 if state is off else 0):][:h.numel()]
               .view(h.shape) for h in state]
        part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
        out = torch.zeros(8, dtype=torch.float64, device=dev)
        engine.check(engine.fluid_reaction_ab_shifted_async(
            fl, fmt, op, state[0], nxt[0], state[1], nxt[1], state[2], nxt[2], nx, ny, nz, 1 / 0.6, 1 / 0.8, 0.3, 1.0,
            0.5, part if stats else None, nbytes if stats else 0))
        if stats:
            engine.check(engine.reactive_stats_finalize_async(fl, "float", nx, ny, nz, 0.3, part, nbytes, out))
        rows.append((nxt, out))
    torch.cuda.synchronize()
    for a, b in zip(rows[0][0], rows[1][0]):
        assert torch.equal(a, b)
    if stats:
        assert bool(torch.isfinite(rows[0][1]).all())
        scale = rows[1][1].abs().clamp_min(1e-2)
        assert float(((rows[0][1] - rows[1][1]).abs() / scale).max()) <= 1e-12
