"""The halo items of open blocks hold slots of levels of any size the device
takes: also past 2^31 (a level of more than 2 10^9 cells fits in FP16)."""
import ctypes

import pytest


@pytest.mark.parametrize("to,src", [(0, 0), (2 ** 31 - 1, 2 ** 31), (2 ** 31, 5), (2 ** 32 - 1, 2 ** 32), (2 ** 40 + 3, 2 ** 33 + 7),
                                    (2 ** 48 - 1, 2 ** 48 - 1)])
@pytest.mark.parametrize("pop,fill", [(1, 0), (18, 1)])
def test_slots_round_trip(ob, to, src, pop, fill):
    out = (ctypes.c_longlong * 4)()
    f = ob.capi.lib().octlb_gpu_debug_open_item
    f.restype, f.argtypes = None, [ctypes.c_longlong] * 2 + [ctypes.c_int] * 2 + [ctypes.POINTER(ctypes.c_longlong)]
    f(to, src, pop, fill, out)
    assert list(out) == [to, src, pop, fill]
