"""The probe that licenses the ordered-atomic ranking runs every kernel shape that a sort of 4-byte keys takes:
its list of sorts against the shapes of all lengths.  Both come from the library; no GPU is needed."""
import ctypes as C

import pytest

from hpcsharp_b200 import build, native

AUTO, LOOKBACK, CHUNKED = 0, 1, 2


@pytest.fixture(scope="module")
def lib():
    build.build_gpu()
    lib = native.load()
    lib.hpcs_sort_shape.argtypes = [C.c_int, C.c_int, C.c_int, C.c_int64, C.c_int]
    lib.hpcs_probe_sort.argtypes = [C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int32), C.POINTER(C.c_int64)]
    return lib


def _lengths(sms):
    """Around every power of two and every multiple of the SM count times one, and in between."""
    out = set()
    for base in (1, sms * 512, sms * 512 * 3):
        x = 2
        while x * base < 1 << 31:
            out |= {x * base - 1, x * base, x * base + 1, x * base * 5 // 4, x * base * 3 // 2}
            x *= 2
    return sorted(n for n in out if n >= 2)


@pytest.mark.parametrize("items", [0, 1])
@pytest.mark.parametrize("sms", [148, 132, 74, 20])
def test_every_shape_is_probed(lib, items, sms):
    probed, i = set(), 0
    scheme, n = C.c_int32(), C.c_int64()
    while lib.hpcs_probe_sort(i, items, sms, C.byref(scheme), C.byref(n)):
        probed.add(lib.hpcs_sort_shape(4, items, scheme.value, n.value, sms))
        i += 1
    taken = {lib.hpcs_sort_shape(4, items, s, m, sms) for m in _lengths(sms) for s in (AUTO, LOOKBACK, CHUNKED)}
    assert taken <= probed, (sorted(taken - probed), sorted(probed))


def test_known_shapes(lib):
    """The lines between the shapes of u32 keys, as documented."""
    shape = lambda n, items=0: lib.hpcs_sort_shape(4, items, AUTO, n, 148)
    assert [shape(n) for n in (1000, 2048, 2049, 4096, 4097, 8192, 8193, 65_536, 65_537, 131_072, 131_073, 262_144)] == \
        [204, 204, 208, 208, 216, 216, 308, 308, 316, 316, 332, 332]
    assert [shape(n) for n in (262_145, 606_208, 606_209, 2_424_832, 2_424_833)] == [108, 108, 116, 116, 140]
    assert shape(131_073, 1) == 108
