"""Batches whose tiled arrays number one less than, exactly and one more than two per SM (where the tiled
shape changes) and a handful, planned and direct, with short arrays among them.  Bits against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiled", [1, 7, 295, 296, 297])
def test_few_tiled_arrays(orc, tiled):
    import torch

    ctx = native.Context(0)
    rng = np.random.default_rng(tiled)
    arrays, tensors, segs = [], [], []
    dtypes = ["u32", "f32", "u64", "i64"]
    for i in range(tiled + 40):
        dt = dtypes[i % 4]
        w = np.dtype(native.NP_OF[dt]).itemsize
        lo = 16385 if w == 4 else 8193  # the first length of the tiled path
        n = lo + (0 if i < 4 else int(rng.integers(0, 9000))) if i < tiled else int(rng.integers(1, 8192))
        a = datagen.by_name(dt, n, seed=i)
        t = torch.from_numpy(a.view(np.uint8).copy()).cuda()
        arrays.append(a)
        tensors.append(t)
        segs.append(((t.data_ptr(), n), dt))
    torch.cuda.synchronize()
    ctx.sort_segmented_dev(segs)
    ctx.synchronize()
    wants = []
    for a, t in zip(arrays, tensors):
        want = a.copy()
        orc.sort_radix_lsd(want)
        wants.append(want)
        assert np.array_equal(t.cpu().numpy(), want.view(np.uint8)), (a.dtype, a.size)
        t.copy_(torch.from_numpy(a.view(np.uint8).copy()))
    torch.cuda.synchronize()
    plan = ctx.segplan(segs)
    plan.execute()
    ctx.synchronize()
    for want, t in zip(wants, tensors):
        assert np.array_equal(t.cpu().numpy(), want.view(np.uint8)), (want.dtype, want.size)
    plan.close()
    ctx.close()
