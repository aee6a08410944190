"""The range test of div_rn.cuh at its edges: divisors and numerators one ulp
inside, at and outside [2^-24, 2^40] and [2^-84, 2^100], zeros of both signs
and random significands at those exponents, against numpy's float32 division
bit for bit."""
import numpy as np
import pytest

from test_gpu_division import _pairs, _same, harness  # noqa: F401

pytestmark = pytest.mark.gpu


def _around(exponents, rng):
    edge = np.exp2(np.array(exponents, np.float64)).astype(np.float32)
    near = [edge, np.nextafter(edge, np.float32(0)), np.nextafter(edge, np.float32(np.inf))]
    near += [edge * rng.uniform(1, 2, edge.size).astype(np.float32) for _ in range(400)]
    return np.concatenate(near).astype(np.float32)


@pytest.mark.parametrize("numerators", [(-84, 100), (-85, -83, 99, 101), (-126, -40, 0, 33, 127)])
@pytest.mark.parametrize("divisors", [(-24, 40), (-25, -23, 39, 41), (-126, 0, 7, 127)])
def test_quotients_at_the_range_edges(harness, numerators, divisors):  # noqa: F811
    rng = np.random.default_rng(len(numerators) * 16 + len(divisors))
    a = np.concatenate([_around(numerators, rng), np.array([0.0], np.float32)])
    a = np.concatenate([a, -a])
    b = _around(divisors, rng)
    b = np.concatenate([b, -b])
    A, B = (v.ravel() for v in np.meshgrid(a, b))
    with np.errstate(all="ignore"):
        want = A / B
    ok = _same(_pairs(harness, A, B), want)
    assert ok.all(), f"{(~ok).sum()} mismatches"
