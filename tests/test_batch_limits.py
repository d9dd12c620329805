"""cb_batch_create refuses a block whose padded box 32-bit node indices cannot
address, as cb_create does, before it touches a device (no GPU needed)."""
import ctypes

import pytest


def _lib():
    from chimera_comp_les_b200 import build
    return ctypes.CDLL(build.build())


@pytest.mark.parametrize("dims", [(1300, 1300, 1300), (2147483647, 6, 6), (100000, 100000, 100000)])
def test_block_too_large_for_32_bit_indices(dims):
    from chimera_comp_les_b200._lib import CB_E_ARG, CbConfig
    lib = _lib()
    c = CbConfig()
    lib.cb_config_default(ctypes.byref(c), 16, 16, 16)
    d = (ctypes.c_int * 6)(16, 16, 16, *dims)
    out = ctypes.c_void_p()
    lib.cb_batch_create.restype = ctypes.c_int
    assert lib.cb_batch_create(ctypes.byref(c), 2, d, ctypes.byref(out)) == CB_E_ARG
    assert not out.value
