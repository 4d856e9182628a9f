"""GPU: the kernels on either side of the launch rules (tests/test_launch_rules.py),
at boxes that reach them.

* 16-bit coupled step, four cells per thread: the same state in buffers one code
  off the word alignment takes one cell per thread; the same codes bit for bit, the
  same statistics to 1e-12 (FP64 sums of the same terms in another order).
* FP32 adjoint step, two cells per thread: against the one-cell kernel on buffers one
  element off the alignment. lambda to 1e-6. dJ/dtau slot by slot: a pair's block
  adds the terms of 256 cells to the slot of the first of the two one-cell blocks
  that it covers. A cell's term is a sum of products lambda_i times a relaxed difference
  of f_i, formed in FP32 with at most 2e-6 of s = sum |lambda_i| |f_i| between two
  orders of contraction (19 roundings of 2^-24 each on either side); over the cells of
  a slot the differences add like independent ones, so the bar is six times 2e-6 of the
  root of the sum of their s^2 (one missing cell, about 1e-2, is 50 times that).
* FP32 D3Q19 step and diagnostics in the range where the pairs run in 7 or 8 blocks
  per SM, of D3Q27, whose diagnostics keep one cell per thread, and of FP64 in small
  and in 96-thread blocks: against the CPU oracle, bit for bit (diagnostics 1e-12).
* Coupled step with statistics in small blocks and on the kernels with register
  budgets: against the step without, bit for bit, and the statistics of the fields it
  wrote, 1e-12."""
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


@pytest.mark.parametrize("lat,op,dims", [("D3Q19", "BGK", (66, 62, 60)), ("D3Q19", "TRT", (50, 48, 52)),
                                         ("D3Q19", "MRT", (82, 80, 76)), ("D2Q9", "TRT", (274, 273, 1)),
                                         ("D2Q9", "MRT", (602, 301, 1)), ("D2Q9", "BGK", (514, 230, 1))])
def test_adjoint_pairs_slot_by_slot(engine, dev, lat, op, dims):
    nx, ny, nz = dims
    f = torch.from_numpy(U.random_state(lat, *dims, np.float32, seed=64)).to(dev)
    lam = torch.randn(f.shape, generator=torch.Generator(device=dev).manual_seed(65), device=dev)
    count = engine.stats_partials_bytes(lat, *dims) // 40
    got = []
    for aligned in (True, False):
        cur, nxt, out = (f, lam, torch.empty_like(f)) if aligned else (_off(f), _off(lam), _off(f))
        tau = torch.zeros(count, dtype=torch.float64, device=dev)
        engine.check(engine.adjoint_step_async(lat, "float", op, cur, nxt, out, *dims, 0.7, tau))
        got.append((out.double(), tau))
    torch.cuda.synchronize()
    (a, pair), (b, one) = got
    assert float((a - b).norm() / b.norm()) <= 1e-6
    tiles = -(-nx * ny // 128)
    pad = tiles % 2
    one = torch.nn.functional.pad(one[:tiles * nz].view(nz, tiles), (0, pad)).view(nz, -1, 2)
    pair = torch.nn.functional.pad(pair[:tiles * nz].view(nz, tiles), (0, pad)).view(nz, -1, 2)
    assert float(pair[..., 1].abs().max()) == 0.0
    s = (lam.double().abs() * f.double().abs()).sum(0).view(nz, nx * ny)
    s2 = torch.nn.functional.pad(s * s, (0, 256 * one.shape[1] - nx * ny)).view(nz, -1, 256).sum(-1)
    assert bool(((pair[..., 0] - one.sum(-1)).abs() <= 6 * 2e-6 * s2.sqrt()).all())


STEPS = [("D3Q19", "float", "BGK", (64, 64, 32)), ("D3Q19", "float", "TRT", (52, 50, 54)),
         ("D3Q19", "float", "MRT", (48, 48, 56)), ("D3Q27", "float", "TRT", (74, 70, 72)),
         ("D3Q27", "double", "BGK", (16, 15, 17)), ("D3Q19", "double", "MRT", (7, 9, 11)),
         ("D3Q19", "double", "RLBM", (33, 2, 5)), ("D2Q9", "double", "BGK", (385, 383, 1)),
         ("D2Q9", "double", "BGK", (97, 4001, 1)), ("D2Q9", "double", "BGK", (544, 301, 1))]


@pytest.mark.parametrize("lat,real,op,dims", STEPS)
def test_steps(engine, dev, lat, real, op, dims):
    f0 = U.random_state(lat, *dims, np.float32 if real == "float" else np.float64, seed=66)
    cur = torch.from_numpy(f0).to(dev)
    nxt, again = torch.empty_like(cur), torch.empty_like(cur)
    nbytes = engine.diagnostics_partials_bytes(lat, *dims)
    part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
    out = torch.empty(5, dtype=torch.float64, device=dev)
    engine.check(engine.step_async(lat, real, op, cur, nxt, *dims, 1 / 0.6))
    engine.check(engine.step_diagnostics_async(lat, real, op, cur, again, *dims, 1 / 0.6, part, nbytes, out))
    torch.cuda.synchronize()
    want = O.step(f0, lat, op, *dims, 1 / 0.6, steps=1)
    assert U.same_bits(nxt.cpu().numpy(), want)
    assert U.same_bits(again.cpu().numpy(), want)
    for g, w in zip(out.cpu().numpy()[:3], O.fluid_diagnostics64(want, lat, *dims)[:3]):
        assert abs(g - w) <= 1e-12 * max(abs(w), 1e-6)


@pytest.mark.parametrize("fl,real,op,dims", [("D3Q19", "double", "BGK", (16, 16, 16)), ("D3Q27", "double", "TRT", (33, 5, 7)),
                                             ("D3Q19", "float", "TRT", (32, 32, 32)), ("D2Q9", "float", "MRT", (64, 63, 1)), ("D3Q27", "double", "TRT", (36, 35, 33)),
                                             ("D2Q9", "float", "TRT", (801, 799, 1))])
def test_statistics(engine, dev, fl, real, op, dims):
    """The fused statistics against those of the fields it wrote, in scratch of exactly
    the public size, and the field against the step without statistics."""
    dt, sl = np.float32 if real == "float" else np.float64, O.SCALAR_OF[fl]
    state = [torch.from_numpy(x).to(dev) for x in (U.random_state(fl, *dims, dt, seed=67), U.random_scalar(sl, *dims, dt, seed=68),
                                                   U.random_scalar(sl, *dims, dt, seed=69))]
    nbytes = engine.stats_partials_bytes(fl, *dims)
    runs = []
    for stats in (True, False):
        nxt = [torch.empty_like(t) for t in state]
        part = torch.full((nbytes // 8 + 1,), float("nan"), dtype=torch.float64, device=dev)
        part[-1] = 7.0
        engine.check(engine.fluid_reaction_ab_async(fl, real, op, state[0], nxt[0], state[1], nxt[1], state[2], nxt[2], *dims,
                                                    1 / 0.6, 1 / 0.8, 0.3, part if stats else None, nbytes if stats else 0))
        runs.append((nxt, part))
    out, ref = (torch.zeros(8, dtype=torch.float64, device=dev) for _ in range(2))
    engine.check(engine.reactive_stats_finalize_async(fl, real, *dims, 0.3, runs[0][1], nbytes, out))
    scratch = torch.empty(nbytes // 8, dtype=torch.float64, device=dev)
    engine.check(engine.reactive_stats_async(sl, real, runs[0][0][1], runs[0][0][2], *dims, 0.3, scratch, nbytes, ref))
    torch.cuda.synchronize()
    for a, b in zip(runs[0][0], runs[1][0]):
        assert U.same_bits(a.cpu().numpy(), b.cpu().numpy())
    assert float(runs[0][1][-1]) == 7.0
    assert float(((out - ref).abs() / ref.abs().clamp_min(1e-2)).max()) <= 1e-12
