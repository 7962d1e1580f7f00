"""Launch shapes of the band-limited chains: every grid that pb_masked_rows_table accepts can be launched with a full
chunk of maps and all rows (the table is refused otherwise, and callers take whole transforms)."""
import ctypes

import pytest

from polybin3d_b200 import _native as nat


def status(n):
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], 0.01
    size = ctypes.c_size_t()
    return nat.load().pb_masked_rows_table(ctypes.byref(g), None, ctypes.byref(size))


def plan_length(n):
    """n is a product of at most three factors of 2 .. 16."""
    return n >= 2 and any(n // a // b <= 16 for a in range(1, 17) if n % a == 0 for b in range(1, 17) if n // a % b == 0)


@pytest.mark.parametrize("shape", [lambda n: (n, n, n), lambda n: (1024, 1024, n), lambda n: (n, 2, 1024),
                                   lambda n: (2, n, 1000)], ids=["cube", "rows", "x", "y"])
def test_every_length_can_be_launched(shape):
    for n in range(2, 1025):
        dims = shape(n)
        if dims[2] % 2:
            continue
        assert (status(dims) == 0) == plan_length(n), dims
