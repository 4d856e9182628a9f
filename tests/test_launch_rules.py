"""CPU: the host side of the kernels' launch rules (csrc/common.cuh and the rules of
the several-cell kernels), compiled from the engine's own headers
(host_rules.cu) and asked on the host.

* FastDiv equals floor division.
* Blocks cover every cell of a plane, at most one of them partly, and never more
  than the partial sums that callers size their scratch by; a small box gets
  blocks small enough to reach the SMs.
* Which boxes take several cells per thread. Each expectation is the faster
  kernel of the two as timed on a B200 (the figures stand beside the rules)."""
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
BGK, TRT, MRT, RLBM = range(4)
F16, BF16, E3M12, Q15 = range(4)


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("rules") / "host_rules")
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "host_rules.cu")], check=True)

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", check=True, capture_output=True, text=True).stdout
        rows = [[int(v) for v in line.split()] for line in out.splitlines()]
        assert len(rows) == len(lines)
        return rows

    return run


def test_fast_div(ask):
    rng = random.Random(6)
    top = 2 ** 31 - 1
    ds = {1, 2, 3, 5, 7, 127, 128, 129, 1024, top, top - 1}
    ds |= {(1 << k) + e for k in range(1, 31) for e in (-1, 0, 1)} | {int(2 ** rng.uniform(0, 31)) for _ in range(200)}
    pairs = []
    for d in sorted(d for d in ds if 1 <= d <= top):
        ns = {0, 1, d - 1, d, min(top, 2 * d - 1), top, top // d * d, max(0, top // d * d - 1)}
        ns |= {min(top, rng.randint(0, top // d) * d + e) for _ in range(10) for e in (0, d - 1)}
        pairs += [(n, d) for n in sorted(ns)]
    for (n, d), (q,) in zip(pairs, ask([f"div {n} {d}" for n, d in pairs])):
        assert q == n // d, (n, d)


def test_blocks_cover_the_plane_within_the_partials(ask):
    rng = random.Random(7)
    boxes = [(nx, ny, nz) for nx in (1, 5, 31, 32, 33, 96, 127, 128, 129, 256, 1000) for ny in (1, 2, 7, 64, 300)
             for nz in (1, 3, 40)]
    boxes += [tuple(int(2 ** rng.uniform(0, 9)) for _ in range(3)) for _ in range(300)]
    for (nx, ny, nz), row in zip(boxes, ask(["grid %d %d %d" % b for b in boxes])):
        assert row[-1] == -(-nx // 128) * ny * nz
        for bx, tiles, launched in (row[0:3], row[3:6], row[6:9]):
            where = (nx, ny, nz, bx)
            assert bx % 32 == 0 and 32 <= bx <= 128, where
            assert (tiles - 1) * bx < nx * ny <= tiles * bx, where
            assert launched == tiles * nz <= row[-1], where


def test_small_boxes_get_small_blocks(ask):
    """Threads per block: plain launches, statistics, FP64 launches of a 3-D lattice."""
    want = {(16, 16, 16): (128, 32, 32), (32, 32, 8): (128, 32, 32), (32, 32, 32): (128, 32, 128), (8, 8, 8): (64, 32, 64),
            (24, 24, 24): (128, 32, 32), (28, 28, 28): (128, 32, 32), (30, 30, 30): (128, 32, 64), (16, 16, 1): (128, 32, 32), (40, 40, 40): (128, 128, 128),
            (64, 64, 1): (128, 64, 64),      # the partials of 64-cell rows allow 64
            (128, 128, 1): (128, 128, 128),  # and those of 128-cell rows 128
            (64, 64, 32): (128, 128, 128), (256, 256, 256): (128, 128, 128)}
    got = ask(["grid %d %d %d" % b for b in want])
    assert {b: (r[0], r[3], r[6]) for b, r in zip(want, got)} == want


COUPLED = [
    # lattice, format, resident one-cell blocks per SM, box, four cells per thread
    (19, F16, 9, (8, 8, 8), 0), (19, F16, 9, (32, 32, 32), 0), (19, F16, 9, (40, 40, 40), 0),
    (19, F16, 9, (48, 48, 48), 1), (19, F16, 9, (64, 64, 32), 1), (19, F16, 9, (56, 56, 56), 0),
    (19, F16, 9, (64, 64, 64), 1), (19, F16, 9, (192, 192, 192), 1), (19, BF16, 12, (32, 32, 32), 0),
    (19, BF16, 12, (48, 48, 48), 0), (19, BF16, 12, (64, 64, 32), 1), (19, E3M12, 10, (32, 32, 32), 0),
    (19, E3M12, 10, (64, 64, 64), 0), (19, E3M12, 10, (72, 72, 72), 0), (19, E3M12, 10, (80, 80, 80), 1),
    (19, Q15, 10, (64, 64, 64), 0), (19, Q15, 10, (64, 64, 36), 1), (19, Q15, 10, (52, 52, 52), 0),
    (19, F16, 9, (52, 52, 52), 1), (19, Q15, 10, (192, 96, 48), 1), (19, F16, 9, (128, 2, 1024), 0),
    (19, F16, 9, (4, 4, 16384), 0), (19, F16, 9, (40, 40, 200), 0),
    (9, F16, 16, (128, 128, 1), 0), (9, F16, 16, (256, 256, 1), 0), (9, F16, 16, (384, 384, 1), 1),
    (9, F16, 16, (512, 512, 1), 1), (9, E3M12, 12, (256, 256, 1), 0), (9, E3M12, 12, (512, 512, 1), 0),
    (9, E3M12, 12, (768, 768, 1), 1), (9, Q15, 16, (640, 640, 1), 0), (9, Q15, 16, (768, 768, 1), 1),
    (9, F16, 0, (1024, 1024, 1), 1), (9, F16, 0, (128, 128, 1), 0),
]


def test_coupled_16bit_step(ask):
    got = ask(["coupled %d %d %d %d %d %d" % (l, f, r, *b) for l, f, r, b, _ in COUPLED])
    assert [g[0] for g in got] == [c[-1] for c in COUPLED]


ADJOINT = [
    (19, BGK, (16, 16, 16), 0), (19, TRT, (24, 24, 24), 0), (19, BGK, (32, 32, 32), 0), (19, BGK, (40, 40, 40), 1),
    (19, TRT, (44, 44, 44), 0), (19, TRT, (48, 48, 48), 1), (19, BGK, (128, 128, 128), 1), (19, MRT, (32, 32, 32), 0),
    (19, MRT, (64, 64, 64), 0), (19, MRT, (52, 52, 52), 1), (19, MRT, (80, 80, 80), 1), (19, BGK, (8, 8, 4096), 0),
    (19, MRT, (4, 4, 16384), 0), (19, BGK, (65, 64, 64), 0),
    (9, BGK, (128, 128, 1), 0), (9, MRT, (256, 256, 1), 0), (9, TRT, (272, 272, 1), 1), (9, MRT, (512, 512, 1), 1),
]


def test_adjoint_step(ask):
    got = ask(["adjoint %d %d %d %d %d" % (l, op, *b) for l, op, b, _ in ADJOINT])
    assert [g[0] for g in got] == [c[-1] for c in ADJOINT]


FLUID = [
    # lattice, operator, with diagnostics, box, two cells per thread
    (19, BGK, 0, (64, 64, 32), 1), (19, TRT, 0, (64, 64, 32), 1), (19, TRT, 1, (64, 64, 32), 1),
    (19, BGK, 0, (48, 48, 56), 1), (19, BGK, 0, (52, 52, 52), 1), (19, MRT, 0, (52, 52, 52), 0), (19, BGK, 0, (56, 56, 56), 0),
    (19, BGK, 0, (64, 64, 64), 1), (19, BGK, 0, (32, 32, 32), 0), (19, RLBM, 0, (64, 64, 32), 0),
    (19, RLBM, 0, (4, 4, 16384), 0), (27, RLBM, 0, (4, 4, 16384), 0), (27, RLBM, 0, (96, 96, 96), 1),
    (27, BGK, 0, (96, 96, 96), 1), (27, TRT, 1, (96, 96, 96), 0), (27, RLBM, 1, (128, 128, 128), 0),
    (9, BGK, 0, (512, 512, 1), 0), (9, BGK, 1, (1024, 1024, 1), 1),
]


def test_fluid_step(ask):
    got = ask(["fluid %d %d %d %d %d %d" % (l, op, d, *b) for l, op, d, b, _ in FLUID])
    assert [g[0] for g in got] == [c[-1] for c in FLUID]
