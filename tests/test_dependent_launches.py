"""Passes that may start before the launch ahead of them has ended: the memory
that the launch ahead still writes (signals, intermediates, filter spectra) is
read by ordinary loads, never through the read-only path, which the hardware
need not keep coherent while a kernel runs.  The host replay counts read-only
loads that fall into a pass's own arrays.  On the GPU, calls queued without a
wait -- one-stage columns, bases 4 and 8, spectra of changing filters read at
once by the pass that follows -- give bit for bit what the same calls give
when each is waited for."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import pac, rng

F64, F32 = pac.PAC_FORM_F64, pac.PAC_FORM_F32
# one-stage columns of every length, short and long columns, rows, split axes
# with both kinds of 4-step twiddles (whole table, two-level above 2^20)
SHAPES = [((2, 256), 1, 2), ((4, 8, 256), 1, 2), ((8, 512), 1, 8), ((16, 64), 3, 4),
          ((64, 64), 2, 8), ((256, 64), 1, 4), ((512, 64), 1, 8), ((1024, 64), 1, 2),
          ((4096,), 3, 2), ((1 << 14,), 3, 2), ((1 << 16,), 2, 4)]
LONG = [((1 << 21,), 1, 2)]


def convolutions(L, dims, batch, base, form, wait):
    """Filters that change before every convolution, in place, and a
    transform pair in between."""
    dt = np.float64 if form == F64 else np.float32
    g = rng(23)
    shape = (batch,) + dims
    d = P.Dev(L)
    plan = pac.Plan(L, dims, batch, base, form)
    try:
        h = []
        for k in range(4):
            v = np.zeros(shape)
            v[(slice(None),) + (0,) * len(dims)] = 0.9
            v[(slice(None),) + (0,) * (len(dims) - 1) + (k + 1,)] = 0.3
            h.append([d.put(v), d.put(0.4 * v)])
        H = [d.zeros(shape, dt) for _ in range(2)]
        x = [d.put(g.standard_normal(shape).astype(dt)) for _ in range(2)]

        def done():
            if wait:
                pac.check(L, L.pac_stream_synchronize(None), "sync")

        for k in range(16):
            plan.filter_spectrum(*h[k % 4], *H, nfilters=batch)
            done()
            plan.convolve(*x, *H, *x, per_problem=1)
            done()
            if k % 4 == 3:
                for op in (pac.OP_AT, pac.OP_CONJ_A, pac.OP_FFT, pac.OP_IFFT):
                    plan.transform(op, *x, *x)
                    done()
        return [d.get(p, shape, dt) for p in x]
    finally:
        plan.close()
        d.free()


@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", SHAPES + LONG)
def test_data_is_not_read_only(emu, dims, batch, base, form):
    before = emu.pac_emu_read_only_data_loads()
    convolutions(emu, dims, batch, base, form, False)
    assert emu.pac_emu_read_only_data_loads() == before


@pytest.mark.parametrize("form", [F64, F32])
def test_uneven_batch_data_is_not_read_only(emu, form):
    before = emu.pac_emu_read_only_data_loads()
    P.check_multi(emu, [(256,), (64, 32), (256,), (1 << 14,), (8, 256), (1 << 14,)], form)
    assert emu.pac_emu_read_only_data_loads() == before


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", SHAPES + LONG)
def test_queued_calls(lib, dims, batch, base, form):
    a = convolutions(lib, dims, batch, base, form, True)
    b = convolutions(lib, dims, batch, base, form, False)
    for u, v in zip(a, b):
        assert np.isfinite(u).all()
        assert np.array_equal(u, v)


# the no-allocation entry point fills its tables on the caller's stream, so
# the first pass over them may not start early; the largest and the smallest
# sizes, and the one whose split depends on the batch
NOALLOC = [(6, 5), (12, 3), (13, 3), (13, 70), (14, 2), (15, 1), (16, 2)]
SCRATCH = 1280 * 1024  # its static array


@pytest.mark.parametrize("logn,batch", NOALLOC)
def test_tables_are_waited_for(emu, logn, batch):
    n = 1 << logn
    g = rng(logn)
    x = g.standard_normal((batch, n)) + 1j * g.standard_normal((batch, n))
    h = g.standard_normal(n) + 1j * g.standard_normal(n)
    d = P.Dev(emu)
    emu.pac_emu_conv_in_scratch.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_int] + [C.c_void_p] * 6
    before = emu.pac_emu_early_tables()
    try:
        a = [d.put(np.ascontiguousarray(v)) for v in (x.real, x.imag, h.real, h.imag)]
        y = [d.zeros((batch, n), np.float64) for _ in range(2)]
        scratch = d.put(np.full(SCRATCH, 255, np.uint8))  # NaN
        for _ in range(2):
            pac.check(emu, emu.pac_emu_conv_in_scratch(scratch, SCRATCH, logn, batch, *a, *y), "conv")
        y = [d.get(p, (batch, n), np.float64) for p in y]
    finally:
        d.free()
    assert P.crel(y[0] + 1j * y[1], np.fft.ifft(np.fft.fft(x) * np.fft.fft(h))) < P.TOL
    assert emu.pac_emu_early_tables() == before


@pytest.mark.parametrize("form", [F64, F32])
def test_plan_tables_are_waited_for(emu, form):
    before = emu.pac_emu_early_tables()
    convolutions(emu, (1 << 14,), 2, 2, form, False)
    P.check_multi(emu, [(256,), (1 << 14,), (8, 256)], form)
    assert emu.pac_emu_early_tables() == before
