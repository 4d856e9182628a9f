"""CPU: the division by a row length in the kernels' cell mapping (FastDiv,
lb-cube_b200/csrc/common.cuh), restated in integers, against Python's //: the
edges of every power of two and random pairs over the whole range n, d < 2^31."""
import random


def fast_div(d):
    shift = 0
    while (1 << shift) < d:
        shift += 1
    mul = ((1 << (31 + shift)) + d - 1) // d
    assert mul < 1 << 32
    return lambda n: (((2 * n) * mul) >> 32) >> shift


def test_fast_div_is_floor_division():
    rng = random.Random(5)
    top = 2 ** 31 - 1
    ds = {1, 2, 3, 5, 7, 127, 128, 129, 1024, top, top - 1}
    ds |= {(1 << k) + e for k in range(1, 31) for e in (-1, 0, 1)}
    ds |= {rng.randint(1, top) for _ in range(300)} | {int(2 ** rng.uniform(0, 31)) for _ in range(300)}
    for d in ds:
        if not 1 <= d <= top:
            continue
        div = fast_div(d)
        ns = {0, 1, d - 1, d, min(top, 2 * d - 1), top, top // d * d, max(0, top // d * d - 1)}
        ns |= {rng.randint(0, top) for _ in range(20)}
        ns |= {min(top, rng.randint(0, top // d) * d + e) for _ in range(20) for e in (0, d - 1)}
        for n in ns:
            assert div(n) == n // d, (n, d)
