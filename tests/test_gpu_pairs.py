"""GPU: the kernels with two FP32 cells per thread, and the loads that evict
their lines first, at sizes that reach them (pairs_eligible and
evict_first_loads in csrc; smaller boxes and odd rows take one cell per thread).

* Fluid steps: bit-identical to the CPU oracle.
* Coupled, scalar and reaction steps: the same state in buffers one element off
  the 8-byte alignment takes the one-cell kernels; every output, the FP64
  statistics included, must have the same bits.
* Fused diagnostics: 1e-12 of the oracle's FP64 sums (another order).
* Adjoint step: the one-cell result to 1e-6, its tau sum to 2e-6 of the sum of
  |lambda| |f| (FP32 sums of at most 19 terms per cell, which the two kernels may
  contract differently: 19 roundings of 2^-24 each).
* Reactive gradient: a box whose planes in one piece take pairs and in two slabs
  do not; the bars of test_gpu_slab_adjoint.py."""
import numpy as np
import pytest
import torch

import _util as U
import oracle as O
from test_gpu_adjoint_reactive import fields
from test_gpu_slab_adjoint import slabs, whole_box

pytestmark = pytest.mark.gpu

REALS = {"float": np.float32, "double": np.float64}
FLUID = [("D3Q19", "float", op, (66, 62, 60)) for op in ("BGK", "TRT", "MRT", "RLBM")]
FLUID += [("D2Q9", "float", op, (602, 598, 1)) for op in ("BGK", "TRT", "MRT", "RLBM")]
FLUID += [("D3Q27", "float", op, (70, 68, 66)) for op in ("BGK", "TRT")]
FLUID += [("D3Q27", "float", op, (90, 86, 84)) for op in ("MRT", "RLBM")]
# buffers just above the L2: evict-first loads, pairs, single cells, plane pointers, FP64
FLUID += [("D3Q19", "float", "TRT", (98, 96, 94)), ("D3Q19", "float", "BGK", (97, 95, 95)),
          ("D3Q19", "float", "MRT", (97, 95, 95)), ("D3Q27", "float", "MRT", (82, 84, 84)),
          ("D3Q19", "double", "BGK", (80, 80, 80)), ("D3Q19", "double", "MRT", (79, 80, 80)),
          ("D2Q9", "double", "TRT", (1024, 1000, 1))]


@pytest.mark.parametrize("lat,real,op,dims", FLUID)
def test_step_bitwise(engine, dev, lat, real, op, dims):
    f0 = U.random_state(lat, *dims, REALS[real], seed=11)
    cur = torch.from_numpy(f0).to(dev)
    nxt = torch.empty_like(cur)
    engine.check(engine.launch_step_gpu(lat, real, op, cur, nxt, *dims, 1 / 0.6))
    torch.cuda.synchronize()
    assert U.same_bits(nxt.cpu().numpy(), O.step(f0, lat, op, *dims, 1 / 0.6, steps=1))


@pytest.mark.parametrize("shift", [0, 1])
def test_packed_d3q27_mrt_mixed_cells(engine, dev, shift):
    """Cells inside and outside the bounds of the fast path in one pair: ordinary
    cells next to tiny (subnormal moments, dividends around 2^-123), huge, zero,
    negative-zero and non-finite ones, whose populations reach their neighbours
    as the step pulls."""
    dims = (90, 86, 84)
    n = dims[0] * dims[1] * dims[2]
    f0 = U.random_state("D3Q27", *dims, np.float64, seed=21, neq=2e-2)
    kind = (np.arange(n) + shift) % 97
    for k, scale in ((3, 2.0 ** -104), (11, 2.0 ** -110), (19, 2.0 ** -116), (27, 2.0 ** -122), (35, 2.0 ** -140),
                     (43, 2.0 ** 61), (51, 2.0 ** 100), (59, 0.0), (67, -0.0)):
        f0[:, kind == k] *= scale
    f0 = f0.astype(np.float32)
    f0[4, np.flatnonzero(kind == 75)[::50]] = np.inf
    f0[9, np.flatnonzero(kind == 83)[::50]] = np.nan
    cur = torch.from_numpy(f0).to(dev)
    nxt = torch.empty_like(cur)
    engine.check(engine.launch_step_gpu("D3Q27", "float", "MRT", cur, nxt, *dims, 1 / 0.6))
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        want = O.step(f0, "D3Q27", "MRT", *dims, 1 / 0.6, steps=1)
    assert U.same_bits(nxt.cpu().numpy(), want)


@pytest.mark.parametrize("lat,op,dims", [("D3Q19", "TRT", (66, 62, 60)), ("D2Q9", "MRT", (602, 598, 1)),
                                         ("D3Q27", "BGK", (70, 68, 66))])
def test_step_diagnostics(engine, dev, lat, op, dims):
    f0 = U.random_state(lat, *dims, np.float32, seed=12)
    cur = torch.from_numpy(f0).to(dev)
    nxt = torch.empty_like(cur)
    nbytes = engine.diagnostics_partials_bytes(lat, *dims)
    part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
    out = torch.empty(5, dtype=torch.float64, device=dev)
    engine.check(engine.step_diagnostics_async(lat, "float", op, cur, nxt, *dims, 1 / 0.6, part, nbytes, out))
    torch.cuda.synchronize()
    want = O.step(f0, lat, op, *dims, 1 / 0.6, steps=1)
    assert U.same_bits(nxt.cpu().numpy(), want)
    for g, w in zip(out.cpu().numpy()[:3], O.fluid_diagnostics64(want, lat, *dims)[:3]):
        assert abs(g - w) <= 1e-12 * max(abs(w), 1e-6)


def _off(t):
    """The same values one element off the allocation's alignment."""
    o = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    o.copy_(t)
    return o


def _like(t, aligned):
    return torch.empty_like(t) if aligned else torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)


def _state(lat, dims, dev):
    sl = O.SCALAR_OF[lat]
    return [torch.from_numpy(U.random_state(lat, *dims, np.float32, seed=13)).to(dev),
            torch.from_numpy(U.random_scalar(sl, *dims, np.float32, seed=14)).to(dev),
            torch.from_numpy(U.random_scalar(sl, *dims, np.float32, seed=15)).to(dev)]


@pytest.mark.parametrize("lat,op,dims", [("D2Q9", "MRT", (602, 598, 1)), ("D2Q9", "TRT", (1024, 1024, 1)),
                                         ("D3Q19", "TRT", (66, 62, 60)), ("D3Q19", "BGK", (70, 66, 58))])
@pytest.mark.parametrize("stats", [False, True])
def test_coupled_step(engine, dev, lat, op, dims, stats):
    state = _state(lat, dims, dev)
    nbytes = engine.stats_partials_bytes(lat, *dims)
    got = []
    for aligned in (True, False):
        cur = state if aligned else [_off(t) for t in state]
        nxt = [_like(t, aligned) for t in state]
        part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
        out = torch.zeros(8, dtype=torch.float64, device=dev)
        engine.check(engine.fluid_reaction_ab_async(lat, "float", op, cur[0], nxt[0], cur[1], nxt[1], cur[2], nxt[2],
                                                    *dims, 1 / 0.6, 1 / 0.8, 0.05, part if stats else None,
                                                    nbytes if stats else 0))
        if stats:
            engine.check(engine.reactive_stats_finalize_async(lat, "float", *dims, 0.05, part, nbytes, out))
        got.append([t.contiguous().view(torch.int32) for t in nxt] + [out])
    torch.cuda.synchronize()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lat,dims", [("D2Q9", (602, 598, 1)), ("D3Q19", (66, 62, 60))])
@pytest.mark.parametrize("species", [1, 2])
def test_scalar_and_reaction_steps(engine, dev, lat, dims, species):
    f, a, b = _state(lat, dims, dev)
    got = []
    for aligned in (True, False):
        cf, ca, cb = (f, a, b) if aligned else (_off(f), _off(a), _off(b))
        na, nb = _like(a, aligned), _like(b, aligned)
        if species == 1:
            engine.check(engine.scalar_step_async(lat, "float", ca, na, cf, *dims, 1 / 0.8, 2e-3))
            got.append([na])
        else:
            engine.check(engine.reaction_ab_async(lat, "float", ca, na, cb, nb, cf, *dims, 1 / 0.8, 0.05))
            got.append([na, nb])
    torch.cuda.synchronize()
    for p, q in zip(*got):
        assert torch.equal(p.view(torch.int32), q.contiguous().view(torch.int32))


@pytest.mark.parametrize("lat,op,dims", [("D3Q19", "BGK", (18, 7, 5)), ("D3Q19", "TRT", (66, 31, 9)),
                                         ("D3Q19", "MRT", (2, 5, 3)), ("D2Q9", "MRT", (130, 33, 1)),
                                         ("D2Q9", "TRT", (514, 2, 1))])
def test_adjoint_step(engine, dev, lat, op, dims):
    f = torch.from_numpy(U.random_state(lat, *dims, np.float32, seed=16)).to(dev)
    gen = torch.Generator(device=dev).manual_seed(17)
    lam = torch.randn(f.shape, generator=gen, device=dev)
    slots = engine.stats_partials_bytes(lat, *dims) // 40
    got = []
    for aligned in (True, False):
        cur, nxt, out = (f, lam, _like(f, True)) if aligned else (_off(f), _off(lam), _like(f, False))
        tau = torch.zeros(slots, dtype=torch.float64, device=dev)
        engine.check(engine.adjoint_step_async(lat, "float", op, cur, nxt, out, *dims, 0.7, tau))
        got.append((out.double(), tau.sum()))
    torch.cuda.synchronize()
    (a, ta), (b, tb) = got
    assert float((a - b).norm() / b.norm()) <= 1e-6
    scale = float((lam.double().abs() * f.double().abs()).sum())  # of the terms that the tau sum adds
    assert abs(float(ta - tb)) <= 2e-6 * scale


@pytest.mark.parametrize("op,storage", [("TRT", None), ("BGK", None), ("MRT", "f16s"), ("TRT", "q15s")])
def test_gradient_in_slabs(engine, dev, op, storage):
    dims = (64, 64, 64)
    rho, u, a, b = fields("D3Q19", dims[::-1], dev, torch.float32, seed=92)
    want = whole_box("D3Q19", "float", op, "mean_product", rho, u, a, b, dims, 4, 2, storage)
    results, ga, gb, gu = slabs("D3Q19", "float", op, "mean_product", rho, u, a, b, dims, 4, 2, 2, storage)
    w = want[0]
    assert np.all(np.abs(results[0] - w) <= 1e-10 * np.abs(w) + 1e-300), (results[0], w)
    for name, got, ref in (("dJ/dA0", ga, want[1]), ("dJ/dB0", gb, want[2]), ("dJ/du0", gu, want[3])):
        assert U.same_bits(got, ref), name
