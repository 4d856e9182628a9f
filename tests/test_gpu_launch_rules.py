"""GPU: the kernels on either side of the launch rules (tests/test_launch_rules.py),
at boxes that reach them.

* 16-bit coupled step, four cells per thread: the same state in buffers one code
  off the word alignment takes one cell per thread; the same codes bit for bit, the
  same statistics to 1e-12 (FP64 sums of the same terms in another order)."""
import numpy as np
import pytest
import torch

import _util as U
import oracle as O

pytestmark = pytest.mark.gpu


def _off(t):
    o = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    o.copy_(t)
    return o


WORDS = [("D3Q19", "f16s", "TRT", (100, 51, 50)), ("D3Q19", "f16s", "MRT", (64, 64, 32)), ("D3Q19", "bf16s", "BGK", (68, 60, 64)),
         ("D3Q19", "e3m12s", "TRT", (100, 99, 50)), ("D3Q19", "q15s", "MRT", (84, 84, 72)),
         ("D2Q9", "f16s", "BGK", (516, 225, 1)), ("D2Q9", "bf16s", "MRT", (508, 240, 1)),
         ("D2Q9", "e3m12s", "MRT", (916, 500, 1)), ("D2Q9", "q15s", "TRT", (700, 701, 1))]


@pytest.mark.parametrize("fl,fmt,op,dims", WORDS)
@pytest.mark.parametrize("stats", [False, True])
def test_coupled_words_match_single_cells(engine, dev, fl, fmt, op, dims, stats):
    nx, ny, nz = dims
    sl = O.SCALAR_OF[fl]
    words = []
    for lat, t, ref in ((fl, U.random_state(fl, *dims, np.float32, seed=61), 1.0),
                        (sl, U.random_scalar(sl, *dims, np.float32, seed=62), 0.5),
                        (sl, U.random_scalar(sl, *dims, np.float32, seed=63), 0.5)):
        h = torch.empty(t.shape, dtype=torch.int16, device=dev)
        engine.check(engine.encode_shifted_async(lat, fmt, "float", torch.from_numpy(t).to(dev), h, *dims, ref))
        words.append(h)
    nbytes = engine.stats_partials_bytes(fl, *dims)
    rows = []
    for state in (words, [_off(h) for h in words]):
        nxt = [torch.empty_like(h) if state is words else _off(h) for h in state]
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
        assert float(((rows[0][1] - rows[1][1]).abs() / rows[1][1].abs().clamp_min(1e-2)).max()) <= 1e-12
