"""The batched sort's tiled kernel (both shapes) around its tiles: one key over the in-shared-memory
limit, whole tiles and one key more or less, ragged 16-byte tails, arrays off the 16-byte boundary,
digits that all keys share, all six key types, both ranking modes.  Bits against the oracle."""
import numpy as np
import pytest

from hpcsharp_b200 import datagen, native

pytestmark = pytest.mark.gpu

DTYPES = ["u32", "i32", "f32", "u64", "i64", "f64"]


@pytest.fixture(scope="module", params=[(8, 0), (9, 0), (9, 1)], ids=["wide", "narrow", "narrow-peer"])
def tctx(request):
    variant, mode = request.param
    c = native.Context(0, rank_mode=mode, seg_grid_min_keys=-1)
    table = c.seg_tuning
    for w in range(2):
        table[w][6] = table[w][7] = variant
    c.seg_tuning = table
    yield c
    c.close()


def _lengths(width):
    tiles = [256 * 32 * 4 // width, 512 * 46 * 4 // width, 512 * 32 * 4 // width]
    out = [8193, 16385]
    for t in tiles:
        out += [2 * t - 1, 2 * t, 2 * t + 1, 3 * t + 7]
    return [n for n in out if n > 8192]


def test_seg_tile_edges(tctx, orc):
    import torch

    arrays, segs, keep = [], [], []
    for i, dt in enumerate(DTYPES):
        w = np.dtype(native.NP_OF[dt]).itemsize
        for j, n in enumerate(_lengths(w)):
            a = datagen.by_name(dt, n, seed=100 * i + j)
            if dt in ("u32", "u64") and j % 4 == 1:
                a = (a & np.array(0xFF00, dtype=a.dtype)) | np.array(3, dtype=a.dtype)  # one digit varies
            t = torch.empty(n * w + 64, dtype=torch.uint8, device="cuda")
            off = w * (j % 3)  # every third array on a 16-byte boundary
            t[off:off + n * w].copy_(torch.from_numpy(a.view(np.uint8)))
            keep.append(t)
            arrays.append((a, t, off))
            segs.append(((t.data_ptr() + off, n), dt))
    torch.cuda.synchronize()
    tctx.sort_segmented_dev(segs)
    tctx.synchronize()
    for a, t, off in arrays:
        want = a.copy()
        orc.sort_radix_lsd(want)
        got = t[off:off + a.nbytes].cpu().numpy()
        assert np.array_equal(got, want.view(np.uint8)), (a.dtype, a.size)
