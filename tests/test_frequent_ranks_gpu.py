"""Digits whose most frequent value holds more or less than 5/16 of the keys (where the passes rank by
votes), with a second value as frequent, rare or absent, in short and whole tiles of both pass schemes.
Bits and stability against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["lookback", "chunked"])
def sctx(request):
    c = native.Context(0, pass_scheme=request.param)
    yield c
    c.close()


def _keys(dt, n, one, two, seed):
    """Bytes that hold 17 with probability `one`, 200 with probability `two`, else any value."""
    rng = np.random.default_rng(seed)
    w = np.dtype(native.NP_OF[dt]).itemsize
    b = rng.integers(0, 256, size=(n, w), dtype=np.uint8)
    r = rng.random((n, w))
    b[r < one] = 17
    b[r >= 1.0 - two] = 200
    return b.view(native.NP_OF[dt]).reshape(-1)


@pytest.mark.parametrize("one,two", [(0.29, 0.0), (0.33, 0.01), (0.4, 0.4), (0.5, 0.5), (0.999, 0.0), (1.0, 0.0)])
@pytest.mark.parametrize("dt", ["u32", "u64"])
def test_frequent_values(sctx, orc, dt, one, two):
    for n in (2, 31, 4097, 8191, 20481, 1_300_003, 3_100_001):
        keys = _keys(dt, n, one, two, seed=n)
        want, got = keys.copy(), keys.copy()
        orc.sort_radix_lsd(want)
        sctx.sort(got)
        assert np.array_equal(got, want), (dt, n)
        items = np.arange(n, dtype=np.uint32)
        ko, io = keys.copy(), items.copy()
        orc.sort_pairs(ko, io)
        sctx.sort_pairs(keys, items)
        assert np.array_equal(keys, ko) and np.array_equal(items, io), (dt, n)
