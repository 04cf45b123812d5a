"""Quotients beside a power of two, where the spacing of the doubles changes.

The FP32 seed of a quotient may lie below the power of two and the quotient
above it, so the rounding test has to take its unit from the quotient.  The
operands are full significands a few to 2^36 units apart (quotients just above
and below one) and pairs whose quotient is also close to a midpoint: with
b near 2k / (2j + 1) and a = b + k units, a / b = 1 + (j + 1/2) units, nearly.
Every result must be the IEEE one, bit for bit.
"""
import numpy as np
import pytest

from test_gpu_exact64 import check, lib, significands  # noqa: F401  (lib: the compiled operations, a fixture)

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -52


def test_a_midpoint_above_one(lib):  # noqa: F811
    a, b = float.fromhex("0x1.38a31d7eaf324p+0"), float.fromhex("0x1.38a31d7eaf2dfp+0")
    check(lib, [a, -a, b, 4.0 * a, a / 1024.0], [b, b, a, b, -b])


@pytest.mark.parametrize("exponent", [0, -300, 500])
def test_operands_units_apart(lib, exponent):  # noqa: F811
    rng = np.random.default_rng(1000 + exponent)
    n = 1 << 22
    b = significands(rng, n)
    near = b + ULP * rng.integers(-4096, 4097, n)
    far = b + ULP * rng.choice([-1.0, 1.0], n) * np.floor(2.0 ** rng.uniform(0.0, 36.0, n))
    for a in (near, far):
        check(lib, np.ldexp(a, exponent), b)


def test_midpoints_beside_powers_of_two(lib):  # noqa: F811
    rng = np.random.default_rng(6)
    n = 1 << 22
    k = rng.integers(1, 4097, n).astype(np.float64)
    m, _ = np.frexp(2.0 * k / (2.0 * rng.integers(0, 4096, n) + 1.0))
    b = 2.0 * m + ULP * rng.integers(-(1 << 28), 1 << 28, n)
    for a in (b + k * ULP, b - k * ULP):
        check(lib, a, b)
        check(lib, -np.ldexp(a, 40), np.ldexp(b, -30))
