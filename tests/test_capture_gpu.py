"""Device sorts, pairs sorts, top-k and select captured into a CUDA graph and replayed on new keys: the
one-launch small sort (one CTA and clusters), the look-back passes and the select's launches, which are not
chained under capture.  Bits against numpy."""
import numpy as np
import pytest

from hpcsharp_b200 import native

pytestmark = pytest.mark.gpu


def _random(dt, n, seed):
    t = native.NP_OF[dt]
    return np.random.default_rng(seed).integers(0, np.iinfo(t).max, n, dtype=t, endpoint=True)


def _dev(a):
    import torch

    return torch.from_numpy(a.view(f"i{a.dtype.itemsize}").copy()).cuda()


def _captured(call, refill):
    """The call captured once (after an eager run, which sizes the scratch) and replayed on refilled inputs."""
    import torch

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        refill(0)
        call(native.torch_stream())
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call(native.torch_stream())
        for seed in (1, 2):
            refill(seed)
            g.replay()
            s.synchronize()
            yield seed


@pytest.mark.parametrize("dt", ["u32", "u64"])
@pytest.mark.parametrize("n", [1000, 9000, 100_003, 262_144, 700_001, 3_000_017])
def test_sorts_captured(dt, n):
    import torch

    c = native.Context(0)
    try:
        keys = _dev(_random(dt, n, 0))
        items = torch.empty(n, dtype=torch.int32, device="cuda")

        def refill(seed):
            keys.copy_(_dev(_random(dt, n, seed) % np.array(n // 2 + 1, dtype=native.NP_OF[dt])))
            items.copy_(torch.arange(n, dtype=torch.int32, device="cuda"))

        for seed in _captured(lambda s: c.sort_dev(keys, dtype=dt, stream=s), refill):
            want = np.sort(_random(dt, n, seed) % np.array(n // 2 + 1, dtype=native.NP_OF[dt]))
            assert np.array_equal(keys.cpu().numpy().view(want.dtype), want)
        for seed in _captured(lambda s: c.sort_pairs_dev(keys, items, dtype=dt, stream=s), refill):
            a = _random(dt, n, seed) % np.array(n // 2 + 1, dtype=native.NP_OF[dt])
            order = np.argsort(a, kind="stable")
            assert np.array_equal(keys.cpu().numpy().view(a.dtype), a[order])
            assert np.array_equal(items.cpu().numpy().view(np.uint32), order.astype(np.uint32))
        c.synchronize()
    finally:
        c.close()


@pytest.mark.parametrize("dt", ["u32", "u64"])
@pytest.mark.parametrize("n", [5000, 300_007, 20_000_003])
def test_topk_and_select_captured(dt, n):
    import torch

    c = native.Context(0)
    try:
        keys = _dev(_random(dt, n, 0))
        out = torch.empty(min(n // 2, 3000), dtype=keys.dtype, device="cuda")
        k = out.numel()

        def refill(seed):
            keys.copy_(_dev(_random(dt, n, seed)))

        for seed in _captured(lambda s: c.topk_largest_dev(keys, k, out, dtype=dt, stream=s), refill):
            assert np.array_equal(out.cpu().numpy().view(native.NP_OF[dt]), np.sort(_random(dt, n, seed))[n - k:])
        for seed in _captured(lambda s: c.select_topk_dev(keys, n // 3, dtype=dt, stream=s), refill):
            a = _random(dt, n, seed)
            v = np.partition(a, n // 3)[n // 3]
            assert np.array_equal(keys.cpu().numpy().view(a.dtype), np.concatenate([a[a < v], a[a == v], a[a > v]]))
        c.synchronize()
    finally:
        c.close()
