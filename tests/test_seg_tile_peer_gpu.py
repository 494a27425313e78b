"""The tiled batched kernel's wide shape with the peer-mask ranking, and the copy for u64 keys in both rankings:
one key over a tile, whole tiles and one key more or less, a constant digit, arrays off the 16-byte boundary.
Bits against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1], ids=["ordered", "peer"])
def test_wide_shape(orc, mode):
    import torch

    c = native.Context(0, rank_mode=mode, seg_grid_min_keys=-1)
    try:
        table = c.seg_tuning
        for w in range(2):
            table[w][6] = table[w][7] = 8
        c.seg_tuning = table
        arrays, segs = [], []
        for dt in ("u64", "u32", "i64", "f64"):
            w = np.dtype(native.NP_OF[dt]).itemsize
            for j, n in enumerate([8193, 9001] + [m * 512 * k * 4 // w + d for k in (32, 46) for m in (1, 2, 3) for d in (-1, 0, 1)]):
                if n <= 8192:
                    continue
                a = datagen.by_name(dt, n, seed=j)
                if dt[0] == "u" and j % 4 == 1:
                    a = (a & np.array(0xFF00, dtype=a.dtype)) | np.array(3, dtype=a.dtype)
                t = torch.empty(n * w + 64, dtype=torch.uint8, device="cuda")
                off = w * (j % 2)
                t[off:off + n * w].copy_(torch.from_numpy(a.view(np.uint8)))
                arrays.append((a, t, off))
                segs.append(((t.data_ptr() + off, n), dt))
        torch.cuda.synchronize()
        c.sort_segmented_dev(segs)
        c.synchronize()
        for a, t, off in arrays:
            want = a.copy()
            orc.sort_radix_lsd(want)
            assert np.array_equal(t[off:off + a.nbytes].cpu().numpy(), want.view(np.uint8)), (a.dtype, a.size)
    finally:
        c.close()
