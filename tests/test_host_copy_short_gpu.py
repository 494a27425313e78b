"""Host-array entry points on short pageable arrays: the sizes at which the copies change, which are
the first staged size (32 KiB), the first chunk shared among threads (256 KiB), one chunk and a
little more (512 KiB), equal quarters and their remainders, the largest short array and the first
long one (32 MiB).  Bit-exact against the oracle and with the staged copies off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KIB = 1 << 10
EDGES = [32 * KIB, 256 * KIB, 512 * KIB, 2048 * KIB, 8192 * KIB, 32768 * KIB]


@pytest.fixture(scope="module")
def plain_ctx():
    from hpcsharp_b200 import native

    c = native.Context(0, staged_host_copies=False)
    yield c
    c.close()


@pytest.mark.parametrize("delta", [-4, 0, 4])
@pytest.mark.parametrize("edge", EDGES)
def test_u32_and_pairs_around_the_edges(ctx, plain_ctx, orc, edge, delta):
    n = (edge + delta) // 4
    keys = np.random.default_rng(edge + delta).integers(0, 1 << 32, n, dtype=np.uint32)
    want = keys.copy()
    orc.sort_radix_par(want)
    buf = np.empty(n + 3, dtype=np.uint32)  # a start that is aligned to the element only
    got = buf[3:]
    got[:] = keys
    ctx.sort(got)
    np.testing.assert_array_equal(got, want)
    plain = keys.copy()
    plain_ctx.sort(plain)
    np.testing.assert_array_equal(plain, want)
    k, v = keys >> 20, np.arange(n, dtype=np.uint32)
    k2, v2 = k.copy(), v.copy()
    ctx.sort_pairs(k, v)
    orc.sort_pairs(k2, v2)
    np.testing.assert_array_equal(k, k2)
    np.testing.assert_array_equal(v, v2)


@pytest.mark.parametrize("n", [16 * KIB + 1, 300 * KIB + 1, 3 * 1024 * KIB + 7])
def test_odd_byte_counts(ctx, n):
    for dt in (np.uint8, np.uint16):
        a = np.random.default_rng(n).integers(0, np.iinfo(dt).max, n, dtype=dt, endpoint=True)
        got = a.copy()
        ctx.sort(got)
        np.testing.assert_array_equal(got, np.sort(a))


def test_short_and_long_arrays_in_turn(ctx):
    rng = np.random.default_rng(5)
    for n in (9_000_000, 9_000, 300_000, 9_000_001, 3_000_000, 70_000, 300_001):
        a = rng.integers(0, 1 << 32, n, dtype=np.uint32)
        got = a.copy()
        ctx.sort(got)
        np.testing.assert_array_equal(got, np.sort(a))
