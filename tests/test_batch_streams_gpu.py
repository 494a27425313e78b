"""How a batch's launches are spread over the streams: a batch bound by one array's time (a few long arrays
among many short ones of every class), one bound by the GPU's throughput, batches of one and of two
launches; as a planned call and as a direct one.  Bits against the oracle, and the time of the first kind:
nothing may run behind its longest array."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu

SETS = {
    "one array's time": [(100, 40), (200, 40), (400, 30), (1500, 30), (3500, 20), (7000, 20), (13_000, 6)],
    "throughput": [(100, 400), (400, 300), (1500, 300), (3500, 300), (7000, 300), (13_000, 330)],
    "one launch": [(100, 5)],
    "two launches": [(100, 5), (20_000, 2)],
}


def _make(lengths, dtypes):
    import torch

    arrays, segs, keep = [], [], []
    i = 0
    for n, count in lengths:
        for _ in range(count):
            dt = dtypes[i % len(dtypes)]
            a = datagen.by_name(dt, n + i % 7, seed=i)
            t = torch.from_numpy(a.view(np.uint8)).cuda()
            arrays.append((a, t))
            segs.append(((t.data_ptr(), a.size), dt))
            i += 1
    return arrays, segs


@pytest.mark.parametrize("kind", sorted(SETS))
@pytest.mark.parametrize("planned", [True, False], ids=["plan", "direct"])
def test_batch_streams(ctx, orc, kind, planned):
    import torch

    arrays, segs = _make(SETS[kind], ["u32", "f32", "u64", "i64"])
    torch.cuda.synchronize()
    if planned:
        plan = ctx.segplan(segs)
        plan.execute()
        ctx.synchronize()
        plan.close()
    else:
        ctx.sort_segmented_dev(segs)
        ctx.synchronize()
    for a, t in arrays:
        want = a.copy()
        orc.sort_radix_lsd(want)
        assert np.array_equal(t.cpu().numpy(), want.view(np.uint8)), (kind, a.dtype, a.size)


def _us(ctx, segs):
    import torch

    plan = ctx.segplan(segs)
    s = native.torch_stream()
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            plan.execute(stream=s)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 100)
    plan.close()
    return sorted(times)[2]


def test_nothing_behind_the_longest(ctx):
    """1024 arrays of log-uniform lengths, the longest four u64 arrays of more than 8192 keys: they take little
    longer than those four alone (1.04 times; 1.47 with other launches queued behind them)."""
    from hpcsharp_b200 import workloads

    lengths, dtypes = workloads.batched_lengths(count=1024, target_total=1_024_000)
    arrays, segs = [], []
    for n, dt in zip(lengths, dtypes):
        a, s = _make([(int(n), 1)], [dt])
        arrays += a
        segs += s
    longest = [s for s in segs if s[1] == "u64" and s[0][1] > 8192]
    assert 2 <= len(longest) <= 8
    assert _us(ctx, segs) < 1.2 * _us(ctx, longest)


def test_more_equal_tiled_arrays_than_sms(ctx, orc):
    """Equal tiled arrays, a few more than SMs: two to an SM, not a second round of one to an SM (which took
    1.76 times as long as one round; two to an SM take 1.42 times)."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    arrays, segs = _make([(23_560, sms + sms // 12)], ["u32"])
    assert _us(ctx, segs) < 1.6 * _us(ctx, segs[:sms])
    for a, t in arrays[::20]:
        want = a.copy()
        orc.sort_radix_lsd(want)
        assert np.array_equal(t.cpu().numpy(), want.view(np.uint8))
