"""Launches of few tiles reserve an SM's shared memory, which spreads their CTAs
over the SMs, on the legacy default stream only: on other streams the kernels of
several plans share the SMs."""
import ctypes as C

import pytest

SM, CTA = 228 * 1024, 226 * 1024


@pytest.mark.parametrize("smem", [0, 9 * 1024, 70 * 1024, 200 * 1024])
@pytest.mark.parametrize("tiles,fit", [(1, 148), (64, 2368), (128, 296), (147, 148), (512, 1184),
                                       (1183, 1184), (1184, 1184), (5000, 1184), (7, 0)])
def test_reserved_shared_memory(emu, smem, tiles, fit):
    f = emu.pac_emu_vec_smem
    f.argtypes = [C.c_size_t, C.c_longlong, C.c_longlong, C.c_int, C.c_int]
    f.restype = C.c_size_t
    assert f(smem, tiles, fit, 148, 0) == smem
    got = f(smem, tiles, fit, 148, 1)
    if fit == 0 or tiles >= fit:
        assert got == smem
    else:
        per_sm = -(-tiles // 148)
        assert smem <= got <= CTA
        assert got * per_sm <= SM or got == smem  # an even share still fits
