"""The look-back passes at the edges of their three tile sizes: one tile (no scanner CTA), two tiles,
one key around a whole number of tiles, and the sizes where the tile changes (one small tile per SM,
two middle tiles per SM), ragged 16-byte tails included.  Bits and stability against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu

NT = 512
SMS = 148
LARGE = {("u32", False): 40, ("u64", False): 24, ("u32", True): 24, ("u64", True): 16}
SMALL, MIDDLE = NT * 8, NT * 16
SMALL_MAX, MIDDLE_MAX = SMS * SMALL, 2 * SMS * MIDDLE


@pytest.fixture(scope="module")
def lctx():
    c = native.Context(0, pass_scheme="lookback")
    yield c
    c.close()


def _sizes(width, pairs):
    large = NT * LARGE[width, pairs]
    whole = (MIDDLE_MAX // large + 1) * large
    return [2, 33, SMALL - 1, SMALL, SMALL + 1, 2 * SMALL + 3, SMALL_MAX, SMALL_MAX + 1, SMALL_MAX + MIDDLE, MIDDLE_MAX,
            MIDDLE_MAX + 1, whole - 1, whole, whole + 1]


@pytest.mark.parametrize("dt", ["u32", "f32", "u64", "i64"])
def test_lookback_tile_edges_plain(lctx, orc, dt):
    for n in _sizes("u64" if dt in ("u64", "i64") else "u32", False):
        a = datagen.by_name(dt, n, seed=n)
        want, got = a.copy(), a.copy()
        orc.sort_radix_lsd(want)
        lctx.sort(got)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), (dt, n)


@pytest.mark.parametrize("dt", ["u32", "u64"])
def test_lookback_tile_edges_pairs(lctx, orc, dt):
    for n in _sizes(dt, True):
        keys = datagen.by_name(dt, n, seed=n) % np.array(3001, dtype=native.NP_OF[dt])  # equal keys show the order
        items = np.arange(n, dtype=np.uint32)
        ko, io = keys.copy(), items.copy()
        orc.sort_pairs(ko, io)
        lctx.sort_pairs(keys, items)
        assert np.array_equal(keys, ko) and np.array_equal(items, io), (dt, n)
