"""The one-launch small sort at its edges: the smallest arrays, one slice of each shape exactly full and
one key more, one key into the next slice of a cluster, 16 full slices of each shape and one key more
(the look-back passes), passes left out, both ranking modes.  Bits and stability against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 12289, 65536, 65537, 131071, 131072, 131073, 262144,
         262145]


@pytest.fixture(scope="module", params=[0, 1])
def cctx(request):
    c = native.Context(0, rank_mode=request.param)
    yield c
    c.close()


@pytest.mark.parametrize("dt", ["u32", "i32", "f32", "u64", "f64"])
def test_small_sort_edges_plain(cctx, orc, dt):
    for n in SIZES:
        a = datagen.by_name(dt, n, seed=n)
        want, got = a.copy(), a.copy()
        orc.sort_radix_lsd(want)
        cctx.sort(got)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), (dt, n)


@pytest.mark.parametrize("dt", ["u32", "i64"])
def test_small_sort_edges_pairs(cctx, orc, dt):
    for n in SIZES:
        keys = (datagen.by_name(dt, n, seed=n) % np.array(501, dtype=native.NP_OF[dt])).astype(native.NP_OF[dt])
        items = np.arange(n, dtype=np.uint32)
        ko, io = keys.copy(), items.copy()
        orc.sort_pairs(ko, io)
        cctx.sort_pairs(keys, items)
        assert np.array_equal(keys, ko) and np.array_equal(items, io), (dt, n)


@pytest.mark.parametrize("bits", [0, 8, 16, 24])
def test_small_sort_one_digit(cctx, orc, bits):
    """Only one byte varies (and, shifted out of range, none): every other pass is the identity."""
    for n in (100, 5000, 70_001):
        a = (datagen.u32_uniform(n, seed=n) & np.uint32(0xFF)) << np.uint32(bits)
        a |= np.uint32(0x5A5A5A5A & ~(0xFF << bits))
        want = np.sort(a)
        cctx.sort(a)
        assert np.array_equal(a, want), (bits, n)
