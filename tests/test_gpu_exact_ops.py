"""The reference arithmetic's roots, reciprocals and quotients without the operators' slow path:
bit for bit numpy's, which are IEEE's correctly rounded ones, over the ranges the transport
takes them from."""
import numpy as np
import pytest

from lightpropagation_b200 import _native

pytestmark = pytest.mark.gpu


def on_device(op, a, b=None):
    a = np.ascontiguousarray(a, np.float32)
    b = a if b is None else np.ascontiguousarray(b, np.float32)
    out = np.empty_like(a)
    _native.check(_native.lib().lp_exact_ops(0, op, a.size, _native.fptr(a), _native.fptr(b), _native.fptr(out)))
    return out


def same_bits(got, want):
    bad = np.flatnonzero(got.view(np.uint32) != want.view(np.uint32))
    assert bad.size == 0, (bad.size, got[bad[:4]], want[bad[:4]])


def mantissas(exponent):
    """Every float in [2^exponent, 2^(exponent + 1))."""
    return (np.arange(1 << 23, dtype=np.uint32) | np.uint32((exponent + 127) << 23)).view(np.float32)


def spread(n, lo, hi, rng):
    """Floats between lo and hi, evenly over their bit patterns."""
    a, b = (int(np.float32(x).view(np.uint32)) for x in (lo, hi))
    return rng.integers(a, b, n, dtype=np.uint32, endpoint=True).view(np.float32)


@pytest.mark.parametrize("exponent", [-99, -2, -1, 0, 1, 126])   # two in a row: all roots
def test_root_of_every_mantissa(exponent):
    a = mantissas(exponent)
    same_bits(on_device(0, a), np.sqrt(a))


def test_root_over_the_range_and_at_its_ends():
    rng = np.random.default_rng(1)
    lowest = np.float32(1e-30)
    a = np.concatenate([spread(1 << 22, 1e-30, 3e38, rng), [lowest, np.nextafter(lowest, np.float32(1)), 3e38]])
    same_bits(on_device(0, a), np.sqrt(a.astype(np.float32)))
    # below the range: 0; outside of the domain: not a number
    below = np.concatenate([spread(1 << 12, 1e-45, 9.99e-31, rng), np.float32([0.0])]).astype(np.float32)
    assert not on_device(0, below).any()
    assert np.isnan(on_device(0, np.float32([-1e-7, -1.0, np.nan]))).all()


@pytest.mark.parametrize("exponent", [-100, -1, 0, 1, 99])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_reciprocal_of_every_mantissa(exponent, sign):
    a = mantissas(exponent) * np.float32(sign)
    same_bits(on_device(1, a), np.float32(1) / a)


@pytest.mark.parametrize("kind", ["any", "near ties", "near floats", "mesh units"])
def test_quotients(kind):
    """Divisors of div_range and beyond it (lengths); numerators at random, at products that put
    the quotient next to a tie or to a float, and as coordinates over a bin width."""
    rng = np.random.default_rng(2)
    n = 1 << 24
    b = spread(n, 1e-12, 1e12, rng)
    if kind == "any":
        a = spread(n, 1e-18, 1e18, rng)
    elif kind == "mesh units":
        a = rng.uniform(-300, 300, n).astype(np.float32)
        b = rng.choice(np.float32([0.1, 0.2, 0.25, 0.3, 0.5, 0.7, 1.0, 1.3, 2.0, 3.0, 10.0]), n)
    else:
        q = spread(n, 1e-9, 1e9, rng).astype(np.float64)
        if kind == "near ties":
            q *= 1.0 + 2.0 ** -24 * rng.choice([0.5, 1.0, 1.0 + 2.0 ** -20], n)
        a = (q * b.astype(np.float64)).astype(np.float32)
        a = np.nextafter(a, rng.choice(np.float32([0.0, 1e30]), n))
        a[::3] = (q[::3] * b[::3].astype(np.float64)).astype(np.float32)
    a[::2] *= np.float32(-1)
    a[:2] = 0.0, -0.0
    same_bits(on_device(2, a, b), a / b)
    same_bits(on_device(2, a, -b), a / -b)
