"""The one-launch small sort where digits are the same in every key: one CTA and clusters of every slice
shape, each digit alone varying, none varying, the lowest constant; negative floats and signed keys; items;
skipping switched off; both ranking modes.  Bits and stability against numpy's stable sort."""
import numpy as np
import pytest

from hpcsharp_b200 import native

pytestmark = pytest.mark.gpu

SIZES = {"u32": [2, 1000, 5000, 8192, 8193, 40_000, 100_003, 131_073, 262_144], "i32": [3000, 200_003], "f32": [3000, 200_003],
         "u64": [2, 1000, 8192, 8193, 60_001, 131_072], "i64": [5000, 100_003], "f64": [5000, 100_003]}


def _ordered(a):
    w = a.dtype.itemsize * 8
    u = a.view(f"u{a.dtype.itemsize}")
    top = np.array(1 << (w - 1), dtype=u.dtype)
    if a.dtype.kind == "i":
        return u ^ top
    if a.dtype.kind == "f":
        return np.where(u & top, ~u, u ^ top)
    return u


def _inputs(dt, n):
    """Keys whose bits vary in one byte, in none, and in all but the lowest and one other."""
    t = np.dtype(native.NP_OF[dt])
    u = np.dtype(f"u{t.itemsize}")
    rng = np.random.default_rng(n)
    bits = rng.integers(0, np.iinfo(u).max, n, dtype=u, endpoint=True)
    base = u.type(0xC1B2A39485766758 >> (64 - 8 * t.itemsize))  # negative as signed and as float
    out = [np.full(n, base, dtype=u)]
    for j in range(t.itemsize):
        m = u.type(0xFF << (8 * j))
        out.append((base & ~m) | (bits & m))
    m = u.type(0xFF | 0xFF << (8 * (t.itemsize // 2)))
    out.append((bits & ~m) | (base & m))
    return [x.view(t) for x in out]


@pytest.fixture(scope="module", params=[(0, True), (0, False), (1, True)], ids=["skip", "noskip", "peer"])
def cctx(request):
    mode, skip = request.param
    c = native.Context(0, rank_mode=mode, skip_trivial_passes=skip)
    yield c
    c.close()


@pytest.mark.parametrize("dt", sorted(SIZES))
def test_constant_digits(cctx, dt):
    for n in SIZES[dt]:
        for i, a in enumerate(_inputs(dt, n)):
            order = np.argsort(_ordered(a), kind="stable")
            got = a.copy()
            cctx.sort(got)
            assert np.array_equal(got.view(np.uint8), a[order].view(np.uint8)), (dt, n, i)
            if n <= 131_072:
                keys, items = a.copy(), np.arange(n, dtype=np.uint32)
                cctx.sort_pairs(keys, items)
                assert np.array_equal(keys.view(np.uint8), a[order].view(np.uint8)), (dt, n, i, "pairs")
                assert np.array_equal(items, order.astype(np.uint32)), (dt, n, i, "items")


def test_constant_digits_cost_no_pass():
    """262,144 equal keys take no longer than uniform ones (ranking every constant digit took 1.4 times as
    long: all lanes of a warp on one counter)."""
    import torch

    c = native.Context(0)
    s = native.torch_stream()
    n = 262_144
    uniform = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda")
    work = torch.empty_like(uniform)

    def us(keys):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                work.copy_(keys)
                c.sort_dev(work, dtype="u32", stream=s)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times)[1]

    try:
        assert us(torch.full_like(uniform, 12345)) < us(uniform)
    finally:
        c.close()
