"""Bounded waits of the passes over 8-byte elements.  With a wait limit of a
few SM cycles every wait for a copied tile gives up; the call still returns,
the status says so once (PAC_ERROR_TIMEOUT, then cleared), and with the default
limit the same plan is right again.  Plans (fused rows, copied columns),
multi-plans -- their spectra, the first call and the recorded ones -- and the
no-allocation entry point, which has no limit to set: the host replay sets
it."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import pac, rng

F64, F32 = pac.PAC_FORM_F64, pac.PAC_FORM_F32
TIMEOUT = 8  # PAC_ERROR_TIMEOUT
ENV = ("PAC_COLTMA", "PAC_PIPE", "PAC_CLUSTER_VARIANT", "PAC_SPECIAL_VARIANT")
# one row pass; copied 512-point columns; a split axis, whose conj(A) columns
# are copied
PLANS = [((4096,), 3, 2), ((512, 64), 2, 2), ((1 << 14,), 2, 2)]


def check_plan(L, dims, batch, base, form):
    dt = np.float64 if form == F64 else np.float32
    g = rng(9)
    shape = (batch,) + dims
    x = g.standard_normal(shape) + 1j * g.standard_normal(shape)
    h = g.standard_normal(dims) + 1j * g.standard_normal(dims)
    d = P.Dev(L)
    plan = pac.Plan(L, dims, batch, base, form)
    try:
        H, y = [d.zeros(dims, dt) for _ in range(2)], [d.zeros(shape, dt) for _ in range(2)]
        plan.filter_spectrum(d.put(h.real), d.put(h.imag), *H)
        xp = [d.put(v.astype(dt)) for v in (x.real, x.imag)]
        assert L.pac_plan_check_status(plan.h, None) == 0
        pac.check(L, L.pac_plan_set_wait_limit(plan.h, 4), "limit")
        plan.convolve(*xp, *H, *y)
        assert L.pac_plan_check_status(plan.h, None) == TIMEOUT
        plan.transform(pac.OP_CONJ_A, *xp, *y)
        assert L.pac_plan_check_status(plan.h, None) == TIMEOUT
        assert L.pac_plan_check_status(plan.h, None) == 0
        pac.check(L, L.pac_plan_set_wait_limit(plan.h, 0), "limit")
        plan.convolve(*xp, *H, *y)
        assert L.pac_plan_check_status(plan.h, None) == 0
        got = d.get(y[0], shape, dt) + 1j * d.get(y[1], shape, dt)
    finally:
        plan.close()
        d.free()
    z = P.fftconv(x, h[None], tuple(range(1, len(shape))))
    assert P.crel(got, z) < (P.TOL if form == F64 else P.TOL_F32)


def check_multi(L, form, stream):
    dt = np.float64 if form == F64 else np.float32
    shapes = [(256,), (64, 32), (256,), (1 << 14,), (4096,), (1 << 14,)]
    m = pac.MultiPlan(L, shapes, 2, form)
    n = int(m.offsets[-1])
    g = rng(10)
    x = g.standard_normal(n) + 1j * g.standard_normal(n)
    h = g.standard_normal(n) + 1j * g.standard_normal(n)
    d = P.Dev(L)
    s = C.c_void_p()
    try:
        if stream:
            pac.check(L, L.pac_stream_create(C.byref(s)), "stream")
        hp = [d.put(h.real), d.put(h.imag)]
        H, y = [d.zeros(n, dt) for _ in range(2)], [d.zeros(n, dt) for _ in range(2)]
        xp = [d.put(v.astype(dt)) for v in (x.real, x.imag)]
        assert L.pac_multi_check_status(m.h, s) == 0
        pac.check(L, L.pac_multi_set_wait_limit(m.h, 4), "limit")
        m.filter_spectra(*hp, *H, s)
        assert L.pac_multi_check_status(m.h, s) == TIMEOUT
        for _ in range(3):  # issued, captured, replayed
            m.convolve(*xp, *H, *y, s)
            assert L.pac_multi_check_status(m.h, s) == TIMEOUT
            assert b"multi-plan gave up" in L.pac_last_error()
            assert L.pac_multi_check_status(m.h, s) == 0
        pac.check(L, L.pac_multi_set_wait_limit(m.h, 0), "limit")
        m.filter_spectra(*hp, *H, s)
        for _ in range(3):
            m.convolve(*xp, *H, *y, s)
            assert L.pac_multi_check_status(m.h, s) == 0
        got = d.get(y[0], (n,), dt) + 1j * d.get(y[1], (n,), dt)
        if stream:
            pac.check(L, L.pac_stream_destroy(s), "stream")
    finally:
        m.close()
        d.free()
    for p, shape in enumerate(shapes):
        o, e = int(m.offsets[p]), int(m.offsets[p + 1])
        z = np.fft.ifftn(np.fft.fftn(x[o:e].reshape(shape)) * np.fft.fftn(h[o:e].reshape(shape)))
        assert P.crel(got[o:e].reshape(shape), z) < (P.TOL if form == F64 else P.TOL_F32), shape
    assert L.pac_multi_check_status(None, None) == 1  # PAC_ERROR_INVALID_VALUE
    assert L.pac_multi_set_wait_limit(None, 1) == 1


@pytest.fixture(autouse=True)
def default_kernels(monkeypatch):
    for name in ENV:
        monkeypatch.delenv(name, raising=False)


@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", PLANS)
def test_plan_replay(emu, dims, batch, base, form):
    check_plan(emu, dims, batch, base, form)


@pytest.mark.parametrize("form", [F64, F32])
def test_multi_replay(emu, form):
    check_multi(emu, form, False)


@pytest.mark.parametrize("logn", [12, 14])
def test_noalloc_replay(emu, logn):
    n, size = 1 << logn, 1280 * 1024
    emu.pac_emu_conv_in_scratch.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_int] + [C.c_void_p] * 6
    emu.pac_emu_noalloc_wait_limit.argtypes = [C.c_longlong]
    d = P.Dev(emu)
    try:
        a = [d.put(np.ones(n)) for _ in range(6)]
        scratch = d.put(np.zeros(size, np.uint8))
        for limit, want in ((4, TIMEOUT), (0, 0)):
            emu.pac_emu_noalloc_wait_limit(limit)
            pac.check(emu, emu.pac_emu_conv_in_scratch(scratch, size, logn, 1, *a), "conv")
            assert emu.pac_noalloc_check_status(None) == want
            assert emu.pac_noalloc_check_status(None) == 0
    finally:
        emu.pac_emu_noalloc_wait_limit(0)
        d.free()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", PLANS)
def test_plan_gpu(lib, dims, batch, base, form):
    check_plan(lib, dims, batch, base, form)


@pytest.mark.gpu
@pytest.mark.parametrize("stream", [False, True])
@pytest.mark.parametrize("form", [F64, F32])
def test_multi_gpu(lib, form, stream):
    check_multi(lib, form, stream)


@pytest.mark.gpu
def test_noalloc_gpu(lib):
    d = P.Dev(lib)
    try:
        a = [d.put(np.ones(4096)) for _ in range(6)]
        assert lib.pac_noalloc_check_status(None) == 0
        pac.check(lib, lib.pac_convolve_1d_noalloc(*a, 4096, 1, None), "conv")
        assert lib.pac_noalloc_check_status(None) == 0
    finally:
        d.free()
