"""The multiplication that replaces the division by an image's row length
(row_of in csrc/common.cuh), at the indices where it could be off by one."""

import random

import pytest


def _magic(nx):
    c = (nx - 1).bit_length()
    shift = 29 + c
    return ((1 << shift) + nx - 1) // nx, shift


def _widths():
    rng = random.Random(5)
    fixed = [2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 255, 257, 4097, 8193, 16385, (1 << 28) - 1, 1 << 28, (1 << 28) + 1]
    return fixed + [rng.randrange(2, 1 << rng.randrange(2, 29)) + 1 for _ in range(400)]


@pytest.mark.parametrize("part", range(4))
def test_row_by_multiplication(part):
    rng = random.Random(part)
    for nx in _widths()[part::4]:
        m, shift = _magic(nx)
        assert m < 1 << 32 and (1 << 29) * m < 1 << 64
        top = (1 << 29) // nx
        rows = {0, 1, top - 1, top} | {rng.randrange(0, top + 1) for _ in range(40)}
        for q in rows:
            for l in (q * nx - 1, q * nx, q * nx + 1, q * nx + nx - 1):
                if 0 <= l < 1 << 29:
                    assert (l * m) >> shift == l // nx
