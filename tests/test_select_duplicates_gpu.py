"""Select and the k largest where copies of few values fill the sampled window: the rank on the copies of
either end of the window, and strictly between the ends with many copies on one or both sides; keys above
the selected one present or not.  Bits against numpy (unsigned keys: equal order, equal bits)."""
import numpy as np
import pytest

from hpcsharp_b200 import native

pytestmark = pytest.mark.gpu

N = 3_000_017  # more copies than the one-cluster finish takes


def _keys(dt, kind, rng):
    t = np.iinfo(native.NP_OF[dt])
    a = rng.integers(1 << 20, t.max - (1 << 20), N, dtype=native.NP_OF[dt], endpoint=True)
    if kind == "equal":
        a[:] = 77
    elif kind == "two":
        a = rng.integers(0, 2, N).astype(native.NP_OF[dt])
    elif kind == "lowest":
        a[rng.random(N) < 0.5] = 0
    elif kind == "highest":
        a[rng.random(N) < 0.5] = t.max
    elif kind == "middle":
        a[rng.random(N) < 0.4] = t.max // 2
    else:  # 1500 keys above a value that half the keys have, 300 of them the largest there is
        a //= 4
        a[rng.random(N) < 0.5] = t.max // 2
        top = rng.choice(N, 1500, replace=False)
        a[top] = rng.integers(t.max // 2 + 1, t.max, 1500, dtype=native.NP_OF[dt])
        a[top[:300]] = t.max
    return a


@pytest.mark.parametrize("dt", ["u32", "u64"])
@pytest.mark.parametrize("kind", ["equal", "two", "lowest", "highest", "middle", "above"])
def test_select_and_topk_with_copies(ctx, dt, kind):
    rng = np.random.default_rng(11)
    a = _keys(dt, kind, rng)
    srt = np.sort(a)
    edges = np.flatnonzero(np.diff(srt) != 0) + 1  # first rank of every further value
    runs = np.diff(np.concatenate([[0], edges, [N]]))
    first = int(np.concatenate([[0], edges])[np.argmax(runs)])  # the rank where the longest run begins
    end = first + int(runs.max())
    ranks = {0, first - 100, first - 1, first, first + 50, first + int(runs.max()) // 2, end - 50, end - 1, end, end + 100, N - 1}
    for k in sorted(r for r in ranks if 0 <= r < N):
        v = srt[k]
        got = a.copy()
        ctx.select_topk(got, k)
        np.testing.assert_array_equal(got, np.concatenate([a[a < v], a[a == v], a[a > v]]), err_msg=f"{kind} {k}")
    for k in (1, 200, 300, 1000, 1499, 1500, 1501, 10_000):
        np.testing.assert_array_equal(ctx.topk_largest(a, k), srt[N - k:], err_msg=f"{kind} top {k}")


@pytest.mark.parametrize("dt", ["u32", "u64"])
@pytest.mark.parametrize("planted", ["max", "zero"])
def test_misled_sample(ctx, dt, planted):
    """Keys planted at every sampled position (32768 4-byte keys, 8192 8-byte keys, at stride n // samples):
    the rank lies outside the window.  Both expected-candidate ranges: the one-cluster finish and, with the
    larger n and k, a launch per level on the rebuilt candidates."""
    t = native.NP_OF[dt]
    samples = 32768 if dt == "u32" else 8192
    for n, ks in ((1_500_007, (10, 1000)), (24_000_011 if dt == "u32" else 8_000_009, (2_000_000,))):
        a = np.random.default_rng(n).integers(1, np.iinfo(t).max, n, dtype=t)
        a[np.arange(samples, dtype=np.int64) * (n // samples)] = np.iinfo(t).max if planted == "max" else 0
        srt = np.sort(a)
        for k in ks + (samples + 5,):
            np.testing.assert_array_equal(ctx.topk_largest(a, k), srt[n - k:])
        for k in (n // 2, n // 3):
            v = srt[k]
            got = a.copy()
            ctx.select_topk(got, k)
            np.testing.assert_array_equal(got, np.concatenate([a[a < v], a[a == v], a[a > v]]))


def test_topk_time_with_copies():
    """Half the keys equal to the largest: every copy is a candidate.  They are counted by all SMs, not by
    one cluster (which took 16 times the uniform call here; by all SMs it is about 3 times)."""
    import torch

    c = native.Context(0)
    s = native.torch_stream()
    n, k = 1 << 26, 1000
    uniform = torch.randint(0, 1 << 30, (n,), dtype=torch.int32, device="cuda")
    copies = uniform.clone()
    copies[::2] = (1 << 31) - 1
    out = torch.empty(k, dtype=torch.int32, device="cuda")

    def us(keys):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            c.topk_largest_dev(keys, k, out, dtype="u32", stream=s)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return sorted(times[2:])[2]

    try:
        assert us(copies) < 8 * us(uniform)
    finally:
        c.close()
