"""GPU: z-slabs large enough that their interior planes run the several-cell
kernels (tests/test_gpu_slab.py and tests/test_gpu_slab_adjoint.py stay below
that): launches from plane 1 on, with statistics partials and gradient slots placed by
absolute plane, against the whole box.

* Fluid step, FP32 and 16-bit, and the coupled step: bit for bit.
* Statistics of the coupled step: bit for bit on one rank, to 1e-12 across two (the
  sums are added in another order).
* Reactive gradient: the bars of tests/test_gpu_slab_adjoint.py."""
import numpy as np
import pytest
import torch

import _util as U
import lbcube as E
import slab
from test_gpu_adjoint_reactive import fields
from test_gpu_slab_adjoint import slabs, whole_box

pytestmark = pytest.mark.gpu


def _split(doms, x):
    return [x[:, d.z0:d.z0 + d.nz].contiguous() for d in doms]


def _run(doms, cur, steps, compute):
    nxt = [tuple(torch.empty_like(t) for t in c) if isinstance(c, tuple) else torch.empty_like(c) for c in cur]
    ex = slab.LocalExchange(doms)
    for d, c in zip(doms, cur):
        d.pack(c)
    ex.exchange_all()
    for s in range(steps):
        for d, c, n in zip(doms, cur, nxt):
            compute(d, c, n, s)
        ex.exchange_all()
        cur, nxt = nxt, cur
    return cur


@pytest.mark.parametrize("lat,op,dims", [("D3Q19", "TRT", (64, 64, 130)), ("D3Q19", "MRT", (66, 62, 132)),
                                         ("D3Q27", "BGK", (72, 66, 130))])
@pytest.mark.parametrize("world", [1, 2])
def test_fluid(engine, dev, lat, op, dims, world):
    nx, ny, nz = dims
    f = torch.from_numpy(U.random_state(lat, nx, ny, nz, np.float32, seed=51)).to(dev)
    a, b = f.clone(), torch.empty_like(f)
    for _ in range(3):
        E.check(E.step_async(lat, "float", op, a, b, nx, ny, nz, 1 / 0.6))
        a, b = b, a
    doms = [slab.SlabDomain(torch, lat, "float", op, nx, ny, nz, 1 / 0.6, r, world, dev) for r in range(world)]
    cur = _run(doms, _split(doms, f.view(-1, nz, ny, nx)), 3, lambda d, c, n, s: d.compute(c, n))
    torch.cuda.synchronize()
    assert torch.equal(torch.cat(cur, 1).view(torch.int32), a.view(-1, nz, ny, nx).view(torch.int32))


@pytest.mark.parametrize("fmt,op", [("f16s", "TRT"), ("q15s", "MRT")])
def test_fluid_16bit(engine, dev, fmt, op):
    nx, ny, nz = 64, 64, 130
    f = torch.from_numpy(U.random_state("D3Q19", nx, ny, nz, np.float32, seed=52)).to(dev)
    h = torch.empty(f.shape, dtype=torch.int16, device=dev)
    E.check(E.encode_shifted_async("D3Q19", fmt, "float", f, h, nx, ny, nz, 1.0))
    a, b = h.clone(), torch.empty_like(h)
    for _ in range(3):
        E.check(E.step_shifted_async("D3Q19", fmt, op, a, b, nx, ny, nz, 1 / 0.6, 1.0))
        a, b = b, a
    doms = [slab.SlabDomain(torch, "D3Q19", "float", op, nx, ny, nz, 1 / 0.6, r, 2, dev, storage=fmt) for r in range(2)]
    cur = _run(doms, _split(doms, h.view(-1, nz, ny, nx)), 3, lambda d, c, n, s: d.compute(c, n))
    torch.cuda.synchronize()
    assert torch.equal(torch.cat(cur, 1), a.view(-1, nz, ny, nx))


@pytest.mark.parametrize("op", ["TRT", "MRT"])
@pytest.mark.parametrize("world", [1, 2])
def test_coupled_with_statistics(engine, dev, op, world):
    nx, ny, nz = 64, 64, 130
    lat, steps, omega, omega_c, k = "D3Q19", 3, 1 / 0.6, 1 / 0.8, 0.3
    state = [torch.from_numpy(x).to(dev) for x in (
        U.random_state(lat, nx, ny, nz, np.float32, seed=53), U.random_scalar("D3Q7", nx, ny, nz, np.float32, seed=54),
        U.random_scalar("D3Q7", nx, ny, nz, np.float32, seed=55))]
    whole, other = [t.clone() for t in state], [torch.empty_like(t) for t in state]
    nbytes = E.stats_partials_bytes(lat, nx, ny, nz)
    part = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=dev)
    want = torch.empty(8, dtype=torch.float64, device=dev)
    for s in range(steps):
        last = s == steps - 1
        E.check(E.fluid_reaction_ab_async(lat, "float", op, whole[0], other[0], whole[1], other[1], whole[2], other[2],
                                          nx, ny, nz, omega, omega_c, k, part if last else None, nbytes if last else 0))
        whole, other = other, whole
    E.check(E.reactive_stats_finalize_async(lat, "float", nx, ny, nz, k, part, nbytes, want))
    doms = [slab.ReactiveSlabDomain(torch, lat, "float", op, nx, ny, nz, omega, omega_c, k, r, world, dev)
            for r in range(world)]
    for d in doms:
        d.partials.fill_(float("nan"))
    cur = list(zip(*(_split(doms, t.view(-1, nz, ny, nx)) for t in state)))
    cur = _run(doms, cur, steps, lambda d, c, n, s: d.compute(c, n, stats=s == steps - 1))
    sums = sum(d.rank_sums() for d in doms) if world > 1 else doms[0].rank_sums()
    got = slab.diagnostics_from_sums(torch, "float", sums, nx * ny * nz, k)
    torch.cuda.synchronize()
    for i in range(3):
        assert torch.equal(torch.cat([c[i] for c in cur], 1).view(torch.int32),
                           whole[i].view(-1, nz, ny, nx).view(torch.int32))
    g, w = got.cpu().numpy(), want.cpu().numpy()
    if world == 1:
        assert U.same_bits(g, w)
    else:
        assert np.all(np.abs(g - w) <= 1e-12 * np.maximum(np.abs(w), 1e-300)), (g, w)


@pytest.mark.parametrize("op,storage,world", [("TRT", None, 2), ("MRT", None, 1), ("BGK", "f16s", 2), ("TRT", "q15s", 2)])
def test_reactive_gradient(engine, dev, op, storage, world):
    dims = (64, 64, 130)
    rho, u, a, b = fields("D3Q19", dims[::-1], dev, torch.float32, seed=93)
    want = whole_box("D3Q19", "float", op, "mean_product", rho, u, a, b, dims, 4, 2, storage)
    results, ga, gb, gu = slabs("D3Q19", "float", op, "mean_product", rho, u, a, b, dims, 4, 2, world, storage)
    w = want[0]
    assert np.all(np.abs(results[0] - w) <= 1e-10 * np.abs(w) + 1e-300), (results[0], w)
    for name, got, ref in (("dJ/dA0", ga, want[1]), ("dJ/dB0", gb, want[2]), ("dJ/du0", gu, want[3])):
        assert U.same_bits(got, ref), name
