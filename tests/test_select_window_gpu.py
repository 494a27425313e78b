"""The sampled-window select, its partition and the k largest at their edges: sizes around a tile and
around the sampling threshold, ranks at the ends, candidates for the one-cluster finish and for the
level launches, a sample that misleads, equal keys, unaligned arrays.  Bits against numpy."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu

SAMPLE = {4: 32768, 8: 8192}


def _ordered(a):
    """The reference's key order as unsigned integers."""
    w = a.dtype.itemsize * 8
    u = a.view(f"u{a.dtype.itemsize}")
    top = np.array(1 << (w - 1), dtype=u.dtype)
    if a.dtype.kind == "i":
        return u ^ top
    if a.dtype.kind == "f":
        return np.where(u & top, ~u, u ^ top)
    return u


def _partitioned(a, k):
    o = _ordered(a)
    v = np.partition(o, k)[k]
    return np.concatenate([a[o < v], a[o == v], a[o > v]])


def _largest(a, k):
    o = _ordered(a)
    return a[np.argsort(o, kind="stable")][a.size - k:]


def _same(x, y):
    return np.array_equal(x.view(np.uint8), y.view(np.uint8))


def _check(ctx, a, ks, what):
    for k in ks:
        got = a.copy()
        ctx.select_topk(got, k)
        assert _same(got, _partitioned(a, k)), (what, "select", a.size, k)
        kk = min(k + 1, 70_000)
        assert _same(ctx.topk_largest(a, kk), _largest(a, kk)), (what, "top-k", a.size, kk)


@pytest.mark.parametrize("dt", ["u32", "f32", "i64", "f64"])
def test_window_edges(ctx, dt):
    w = np.dtype(native.NP_OF[dt]).itemsize
    tile, s4 = 32768 // w, 4 * SAMPLE[w]
    for n in (1, 2, tile - 1, tile, tile + 1, s4 - 1, s4, s4 + 5, 9 * tile + 33):
        a = datagen.by_name(dt, n, seed=n)
        _check(ctx, a, sorted({0, n // 2, n - 1}), dt)


@pytest.mark.parametrize("dt", ["u32", "f64"])
def test_window_level_launches(ctx, dt):
    """Enough expected candidates for a launch per level."""
    n = 20_000_003 if dt == "u32" else 12_000_001
    a = datagen.by_name(dt, n, seed=3)
    _check(ctx, a, [n // 2, 17], dt)


@pytest.mark.parametrize("dt", ["u32", "u64"])
@pytest.mark.parametrize("planted", ["max", "zero"])
def test_window_misled(ctx, dt, planted):
    t = native.NP_OF[dt]
    s = SAMPLE[np.dtype(t).itemsize]
    n = 40 * s + 11
    a = datagen.by_name(dt, n, seed=5)
    a[np.arange(s, dtype=np.int64) * (n // s)] = np.iinfo(t).max if planted == "max" else 0
    _check(ctx, a, [n // 3, n - 2], planted)
    assert _same(ctx.topk_largest(a, 3 * s), _largest(a, 3 * s))


@pytest.mark.parametrize("kind", ["equal", "two", "lowest", "special"])
def test_window_duplicates(ctx, kind):
    n = 300_001
    rng = np.random.default_rng(7)
    if kind == "equal":
        a = np.full(n, 77, dtype=np.uint32)
    elif kind == "two":
        a = rng.integers(0, 2, n).astype(np.uint32)
    elif kind == "lowest":
        a = np.where(rng.random(n) < 0.6, np.iinfo(np.int32).min, 5).astype(np.int32)
    else:
        a = rng.choice(np.array([np.nan, -np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-45], dtype=np.float32), n)
    _check(ctx, a, [0, n // 2, n - 1], kind)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_window_unaligned_device(ctx, shift):
    import torch

    n = 500_003
    a = datagen.u32_uniform(n, seed=9)
    t = torch.empty(n + 8, dtype=torch.int32, device="cuda")
    v = t[shift:shift + n]
    v.copy_(torch.from_numpy(a.view(np.int32)))
    out = torch.empty(1001, dtype=torch.int32, device="cuda")
    ctx.topk_largest_dev(v, 1001, out, dtype="u32", stream=native.torch_stream())
    ctx.select_topk_dev(v, n // 4, dtype="u32", stream=native.torch_stream())
    torch.cuda.synchronize()
    assert _same(out.cpu().numpy().view(np.uint32), _largest(a, 1001))
    assert _same(v.cpu().numpy().view(np.uint32), _partitioned(a, n // 4))
