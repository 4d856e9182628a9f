"""GPU: the D3Q27 MRT step at the edges of its fast path, against the CPU oracle
bit for bit.

A cell takes the fast transforms (no divisions, exact products in FMAs) only
inside the bounds of collide_mrt_d3q27 and when every dividend by 6 is 0 or at
least 2^-123; every other cell runs the reference's expression. Both must give
the oracle's bits, so the states here sit on either side of each bound: scaled
towards the underflow range and across 2^60, a relaxation rate above 2^10, and
cells of exact zeros of both signs and of exact symmetry (zero moments)."""
import numpy as np
import pytest
import torch

import _util as U
import oracle as O

pytestmark = pytest.mark.gpu

NX, NY, NZ = 37, 5, 4
REALS = {"float": np.float32, "double": np.float64}


def _check(engine, dev, real, f0, omega):
    cur = torch.from_numpy(f0).to(dev)
    nxt = torch.empty_like(cur)
    engine.check(engine.launch_step_gpu("D3Q27", real, "MRT", cur, nxt, NX, NY, NZ, omega))
    torch.cuda.synchronize()
    want = O.step(f0, "D3Q27", "MRT", NX, NY, NZ, omega, steps=1)
    assert U.same_bits(nxt.cpu().numpy(), want)


@pytest.mark.parametrize("real", ["float", "double"])
@pytest.mark.parametrize("exponent", [-960, -950, -120, -116, -112, -108, -104, 58, 60, 61, 62, 100])
def test_scaled_states(engine, dev, real, exponent):
    if real == "float" and exponent < -149:
        pytest.skip("below the FP32 range")
    f0 = U.random_state("D3Q27", NX, NY, NZ, np.float64, seed=33, neq=2e-2)
    # a different scale per cell, so cells of one warp take both paths
    spread = np.ldexp(1.0, (np.arange(f0.shape[-1]) * 7) % 5 + exponent)
    _check(engine, dev, real, (f0 * spread).astype(REALS[real]), 1 / 0.6)


@pytest.mark.parametrize("real", ["float", "double"])
@pytest.mark.parametrize("omega", [1000.0, 1030.0, 0.0])
def test_relaxation_rates_beyond_the_bound(engine, dev, real, omega):
    f0 = U.random_state("D3Q27", NX, NY, NZ, REALS[real], seed=34)
    _check(engine, dev, real, f0, omega)


@pytest.mark.parametrize("real", ["float", "double"])
def test_zero_and_symmetric_cells(engine, dev, real):
    n = NX * NY * NZ
    f0 = np.zeros((27, n), REALS[real])
    f0[:, 1::4] = -0.0
    f0[:, 2::4] = O.init_equilibrium("D3Q27", np.ones(n), np.zeros((3, n)), NX, NY, NZ, REALS[real])[:, 2::4]
    f0[::2, 3::4] = REALS[real](0.125)
    f0[1::2, 3::4] = REALS[real](-0.0)
    _check(engine, dev, real, f0, 1 / 0.6)
