"""Pivots of the 64-tile Cholesky (csrc/tile64.cuh, `sqrt_rcp` and its careful form for far
exponents) against the correctly rounded square root and reciprocal.

The reduced matrix is block diagonal with 2×2 blocks [[a, b], [b, c]]; a and b are read back
from it.  Then L₁₁ = fl(√a) and L₂₁ = fl(b·fl(1/L₁₁)), bit for bit.  The one exception
that the kernel's comment states: the reciprocal of 2 − 2⁻⁵² (times powers of two) may be
off by one unit in the last place, and L₂₁ then by two (its own rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(p, exponent):
    """p: mantissas, exponent: of each 2×2 block's entries."""
    from sdpx_b200.normal import NormalSystem
    n = 2 * len(p)
    i = np.arange(len(p))
    s = np.ldexp(1.0, exponent)
    B = np.zeros((n, n))
    B[2 * i, 2 * i] = p * s
    B[2 * i, 2 * i + 1] = s
    B[2 * i + 1, 2 * i + 1] = s
    with NormalSystem(np.asfortranarray(B), n) as ns:
        assert ns.factor_reduced(np.ones(n), 0.0, max_attempts=1)[0]
        Q, L = ns.matrix(0), ns.matrix(1)
    a, b = Q[2 * i, 2 * i], Q[2 * i + 1, 2 * i]
    assert np.array_equal(b, p * s * s)
    l = np.sqrt(a)
    assert np.array_equal(L[2 * i, 2 * i], l)
    want, got = b * (1.0 / l), L[2 * i + 1, 2 * i]
    last = np.frexp(l)[0] == 1.0 - 2.0 ** -53  # l = 2 − 2⁻⁵² times a power of two
    assert np.array_equal(got[~last], want[~last])
    assert (np.abs(got - want) <= 2 * np.spacing(want)).all()
    return last


@pytest.mark.parametrize("seed", range(4))
def test_random_pivots(seed):
    rng = np.random.default_rng(seed)
    _check(rng.uniform(1.0, 2.0, 700), rng.integers(-400, 400, 700))


# both sides of the exponents ±830 of a pivot, alone and side by side in a block of eight
@pytest.mark.parametrize("e", [414, 415, 416, 500, -414, -415, -416, -500])
def test_far_exponents(e):
    rng = np.random.default_rng(abs(e))
    p = rng.uniform(1.0, 2.0, 300)
    _check(p, np.full(300, e))
    mixed = np.full(300, e)
    mixed[::3] = 0
    _check(p, mixed)


def test_ends_of_the_mantissa():
    k = np.arange(1, 60)
    p = np.concatenate([1.0 + k * 2.0 ** -52, 2.0 - k * 2.0 ** -52, np.sqrt(2.0) + (k - 30) * 2.0 ** -52, [1.0, 1.5]])
    assert _check(p, np.zeros(len(p), dtype=int)).any()
