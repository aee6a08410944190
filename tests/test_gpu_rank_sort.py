"""Small sorts by rank: sizes around a CTA's 32 keys, a tile and the line to
the digit passes, partial bit ranges, equal and extreme keys, stability."""
import numpy as np
import pytest

from diomedes_gb300 import compute as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 4095, 4096, 4097, 8191, 8192, 8193])
def test_matches_stable_argsort(bits, n):
    rng = np.random.default_rng(n + bits)
    kind = np.uint32 if bits == 32 else np.uint64
    top = 2**bits - 1
    for begin, end, keys in ((0, bits, rng.integers(0, top, n, dtype=np.uint64, endpoint=True)),
                             (0, 7, rng.integers(0, 128, n, dtype=np.uint64)),
                             (5, bits - 3, rng.integers(0, top, n, dtype=np.uint64, endpoint=True)),
                             (0, bits, np.full(n, top, np.uint64)),
                             (0, bits, rng.choice(np.array([0, 1, top - 1, top], np.uint64), n))):
        keys = keys.astype(kind)
        vals = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
        digit = keys.astype(np.uint64) >> np.uint64(begin)
        if end - begin < 64:
            digit = digit & np.uint64((1 << (end - begin)) - 1)
        order = np.argsort(digit, kind="stable")
        ko, vo = C.device_sort_pairs(keys, vals, begin, end)
        assert np.array_equal(ko, keys[order]) and np.array_equal(vo, vals[order])
