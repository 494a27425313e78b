"""Sorts and top-k calls under a scratch budget that holds their ping-pong buffers and little more: large
ones with the count tables of the chunked passes in place of the look-back rows, middle ones with the rows of
the large tile, a small sort and the sort of a top-k call's output with none.  Bits against numpy."""
import numpy as np
import pytest

from hpcsharp_b200 import native

pytestmark = pytest.mark.gpu

PLAN = 32 << 10  # the plan and the small words
KIB = 1 << 10


def _random(dt, n, seed):
    t = native.NP_OF[dt]
    return np.random.default_rng(seed).integers(0, np.iinfo(t).max, n, dtype=t, endpoint=True)


def _dev(a):
    import torch

    return torch.from_numpy(a.view(f"i{a.dtype.itemsize}").copy()).cuda()


# dtype, items, keys, bytes of rows that have to be enough
CASES = [("u32", False, 50 << 20, 148 * 7 * KIB), ("u64", False, 8 << 20, 148 * 11 * KIB), ("u32", True, 8 << 20, 148 * 7 * KIB),
         ("u64", True, 4 << 20, 148 * 11 * KIB), ("u32", False, 1_200_000, 2 * 74 * KIB), ("u32", False, 262_144, 0),
         ("u64", True, 100_003, 0)]


@pytest.mark.parametrize("rank_mode", [0, 1], ids=["ordered", "peer"])
@pytest.mark.parametrize("dt,items,n,rows", CASES, ids=[f"{c[0]}-{'pairs' if c[1] else 'keys'}-{c[2]}" for c in CASES])
def test_sort_under_budget(ctx, dt, items, n, rows, rank_mode):
    import torch

    keys = _random(dt, n, n)
    keys[::5] = keys[0]
    small = n <= 262_144
    budget = (0 if small else n * (keys.itemsize + (4 if items else 0))) + rows + PLAN
    c = native.Context(0, pool_bytes=budget, rank_mode=rank_mode)
    try:
        d = _dev(keys)
        s = native.torch_stream()
        if small and rank_mode == 1 and n > 131_072:
            pytest.skip("above the peer-mask ranking's one-launch sizes")
        if items:
            v = torch.arange(n, dtype=torch.int32, device="cuda")
            c.sort_pairs_dev(d, v, dtype=dt, stream=s)
        else:
            c.sort_dev(d, dtype=dt, stream=s)
        torch.cuda.synchronize()
        c.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(d.cpu().numpy().view(keys.dtype), keys[order])
        if items:
            assert np.array_equal(v.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    finally:
        c.close()


def test_topk_under_budget(ctx):
    import torch

    a = _random("u32", 1_000_003, 3)
    c = native.Context(0, pool_bytes=a.nbytes + 8 * KIB)
    try:
        d, out = _dev(a), torch.empty(8192, dtype=torch.int32, device="cuda")
        c.topk_largest_dev(d, 8192, out, dtype="u32", stream=native.torch_stream())
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.sort(a)[-8192:])
    finally:
        c.close()


def test_still_refused(ctx):
    """A budget without room for the ping-pong buffer, and a forced scheme's rows, are refused as before."""
    a = _random("u32", 8 << 20, 4)
    for kw, budget in (({}, a.nbytes // 2), ({"pass_scheme": "lookback"}, a.nbytes + 148 * 7 * KIB // 4)):
        c = native.Context(0, pool_bytes=budget, **kw)
        try:
            with pytest.raises(native.HpcsError) as e:
                c.sort_dev(_dev(a), dtype="u32", stream=native.torch_stream())
            assert e.value.status == native.HPCS_ERR_OOM
        finally:
            c.close()


def test_first_context_of_a_process_with_a_budget():
    """The ranking probe of a process's first context has scratch of its own: a 12 MiB budget is enough for a
    context and a million keys, whichever context comes first."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = ("import numpy as np\nfrom hpcsharp_b200 import native\nc = native.Context(0, pool_bytes=12 << 20)\n"
            "a = np.random.default_rng(1).integers(0, 1 << 32, 1_000_000, dtype=np.uint32)\nw = np.sort(a)\nc.sort(a)\n"
            "assert np.array_equal(a, w)\nassert c.rank_mode in (0, 1)\nc.close()\nprint('sorted')\n")
    res = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert "sorted" in res.stdout, res.stderr[-2000:]
