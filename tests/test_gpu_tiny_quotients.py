"""div_rn.cuh's quotients of tiny numerators -- scaled up, divided, and brought
down to normal and subnormal results -- against numpy's float32 division bit for
bit: every exponent down to the least subnormal, exact ties between two
subnormals and their neighbours on both sides."""
import numpy as np
import pytest

from test_gpu_division import _pairs, _same, harness  # noqa: F401

pytestmark = pytest.mark.gpu


def _check(harness, a, b):
    a, b = np.concatenate([a, -a]).astype(np.float32), np.concatenate([b, b]).astype(np.float32)
    with np.errstate(all="ignore"):
        want = a / b
    got = _pairs(harness, a, b)
    bad = np.flatnonzero(~_same(got, want))
    assert bad.size == 0, f"{bad.size} of {a.size}, e.g. {a[bad[0]]!r} / {b[bad[0]]!r}: {got[bad[0]]!r} {want[bad[0]]!r}"
    return want


@pytest.mark.parametrize("low,high", [(-149, -127), (-127, -100), (-100, -84), (-84, -39)])
def test_tiny_numerators(harness, low, high):  # noqa: F811
    rng = np.random.default_rng(-low)
    n = 1 << 21
    a = rng.uniform(1, 2, n) * np.exp2(rng.integers(low, high + 1, n))
    b = rng.uniform(1, 2, n) * np.exp2(rng.integers(-24, 40, n))
    b[::5] = np.exp2(rng.integers(-24, 41, b[::5].size))
    want = _check(harness, a, b)
    assert np.count_nonzero((np.abs(want) < 2.0 ** -126) & (want != 0)) > n // 64 or low > -110


def test_ties_between_subnormals(harness):  # noqa: F811
    rng = np.random.default_rng(3)
    n = 1 << 20
    # a / b = h 2^-150 with an odd h: exactly between two subnormals
    h = 2 * rng.integers(0, 1 << 14, n) + 1
    b = (2 * rng.integers(0, 1 << 8, n) + 1) * np.exp2(rng.integers(1, 31, n))
    a = (b * h * 2.0 ** -150).astype(np.float32)
    assert np.array_equal(a.astype(np.float64), b * h * 2.0 ** -150)
    for step in (None, np.float32(0), np.float32(np.inf)):
        _check(harness, a if step is None else np.nextafter(a, step), b)
