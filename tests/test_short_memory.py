"""What is allocated for speed alone is done without where memory is short: the
fft.h functions' third pair of arrays on the device and their pinned memory, a
plan's whole 4-step tables.  On the host replay, whose allocations above a limit
fail; every shape is one that no other test caches."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import O, pac, rng

MB = 1 << 20


@pytest.fixture
def limits(emu):
    emu.pac_emu_alloc_limits.argtypes = [C.c_size_t, C.c_size_t]
    yield emu.pac_emu_alloc_limits
    emu.pac_emu_alloc_limits(0, 0)


def check_dropin(L, shape, r):
    g = rng(5)
    a = [g.standard_normal(shape) for _ in range(4)]
    x, h = a[0] + 1j * a[1], a[2] + 1j * a[3]
    fh = np.fft.fftn(h)
    rev = np.ix_(*[P.digit_reversal(r, n) for n in shape])
    for method, spectrum in ((O.METHOD_PAC, fh[rev]), (O.METHOD_FFT_BASED, fh)):
        y = pac.dropin_convolution(L, method, r, *a)
        assert L.pac_get_last_status() == 0
        assert P.crel(y[0] + 1j * y[1], np.fft.ifftn(np.fft.fftn(x) * fh)) < P.TOL
        assert P.crel(y[2] + 1j * y[3], spectrum) < P.TOL
    y = pac.dropin_transform(L, 0, r, *a[:2])
    assert P.crel(y[0] + 1j * y[1], np.fft.fftn(x)) < P.TOL


@pytest.mark.parametrize("shape,r,limit", [((2, 1 << 16), 2, 32 << 17), ((2, 128), 2, 32 << 8)])
def test_two_pairs_on_the_device(emu, limits, shape, r, limit):
    limits(limit, 0)  # two pairs fit, three do not
    check_dropin(emu, shape, r)


@pytest.mark.parametrize("shape", [(4, 64), (4, 1 << 16)])
def test_no_pinned_memory(emu, limits, shape):
    limits(0, 16)
    check_dropin(emu, shape, 2)


@pytest.mark.parametrize("form,table", [(pac.PAC_FORM_F64, 16 << 15), (pac.PAC_FORM_F32, 8 << 15)])
def test_no_whole_tables(emu, limits, form, table):
    dims, batch = (1 << 15,), 2
    g = rng(6)
    x = g.standard_normal((batch,) + dims) + 1j * g.standard_normal((batch,) + dims)
    d = P.Dev(emu)
    dt = np.float64 if form == pac.PAC_FORM_F64 else np.float32
    try:
        a = [d.put(v.astype(dt)) for v in (x.real, x.imag)]
        y = [d.zeros(x.shape, dt) for _ in range(2)]
        limits(table - 1, 0)
        plan = pac.Plan(emu, dims, batch, 2, form)
        plan.transform(pac.OP_AT, *a, *y)
        plan.transform(pac.OP_CONJ_A, *y, *y)
        plan.close()
        z = (d.get(y[0], x.shape, dt) + 1j * d.get(y[1], x.shape, dt)) / dims[0]
    finally:
        d.free()
    assert P.crel(z, x) < (P.TOL if form == pac.PAC_FORM_F64 else P.TOL_F32)
