"""Passes over 8-byte elements (FP64 lines, FP32 line pairs): every line
length of the fused rows, the DIF and DIT rows and the columns, at the edges
of their tiles -- one line, an odd number of lines (the last FP32 pair has
one), tiles as wide as the stride, outer factors with 4-step twiddles from the
whole table and (above 2^20 points) from the two-level ones -- against numpy.

Relative L2 errors of an FFT of 2^m points grow with the number of butterfly
levels; 1e-13 (FP64) and 1e-6 (FP32) are hundreds of roundings at m <= 21."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

F64, F32 = pac.PAC_FORM_F64, pac.PAC_FORM_F32

# rows of every length and base (dims, batch, base); 8192-point rows are one
# pass from 64 line units on
ROWS = ([((1 << k,), b, 2) for k in range(5, 14) for b in (1, 3)] +
        [((8192,), 131, 2), ((64,), 67, 2), ((256,), 9, 2), ((512,), 2, 2), ((1024,), 5, 2)] +
        [((4 ** k,), 5, 4) for k in range(3, 7)] + [((8 ** k,), 5, 8) for k in range(2, 5)])
# columns of every length and base: at the narrowest stride that has a tile
# of both types, and one with several tiles
COLS = ([((1 << k, 256), 1, 2) for k in range(1, 12)] + [((32, 128), 3, 2), ((64, 64), 3, 2),
        ((128, 32), 3, 2), ((2048, 8), 2, 2), ((512, 16), 1, 2), ((1024, 8), 1, 2)] +
        [((4 ** k, 64), 2, 4) for k in range(1, 6)] + [((8 ** k, 64), 1, 8) for k in range(1, 4)])
# split axes: 1D of 2 and 3 factors, long columns, a middle axis, per-axis bases
SPLIT = [((1 << 14,), 3, 2), ((1 << 15,), 1, 2), ((1 << 17,), 2, 2), ((4 ** 7,), 3, 4),
         ((8 ** 5,), 2, 8), ((4096, 32), 1, 2), ((4, 4096, 16), 1, 2), ((16, 8192), 1, 2),
         ((64, 128, 32), 1, (8, 2, 2))]
LONG = [((1 << 21,), 1, 2)]


def check(L, dims, batch, base, form):
    g = rng(77)
    shape = (batch,) + dims
    axes = tuple(range(1, len(shape)))
    tol = P.TOL if form == F64 else P.TOL_F32
    x = g.standard_normal(shape) + 1j * g.standard_normal(shape)
    fx = np.fft.fftn(x, axes=axes)
    n = int(np.prod(dims))
    bases = base if isinstance(base, tuple) else (base,) * len(dims)
    rev = np.ix_(np.arange(batch), *[P.digit_reversal(b, v) for b, v in zip(bases, dims)])
    want = {pac.OP_AT: fx[rev], pac.OP_CONJ_A: n * np.fft.ifftn(x[rev], axes=axes),
            pac.OP_FFT: fx, pac.OP_IFFT: np.fft.ifftn(x, axes=axes),
            pac.OP_UIFFT: np.fft.ifftn(x[rev], axes=axes)}
    for op, z in want.items():
        assert P.crel(P.native_transform(L, dims, batch, base, form, op, x), z) < tol, op
    h = g.standard_normal(dims) + 1j * g.standard_normal(dims)
    y = P.native_conv(L, dims, batch, base, form, x, h)
    assert P.crel(y, np.fft.ifftn(fx * np.fft.fftn(h), axes=axes)) < tol
    h = g.standard_normal(shape) + 1j * g.standard_normal(shape)
    y = P.native_conv(L, dims, batch, base, form, x, h, per_problem=True)
    assert P.crel(y, np.fft.ifftn(fx * np.fft.fftn(h, axes=axes), axes=axes)) < tol


# uneven batches: problems of one shape apart from each other (an odd number
# of them, so the last FP32 pair of rows has one line), every short-column
# length, and two-element problems after which nothing starts at a multiple of
# 16 bytes (those take the work queue)
UNEVEN = [[(256,), (64, 32), (256,), (2 ** 14,), (512,), (256,), (2 ** 14,), (8192,), (64, 32)],
          [(1 << k, 256) for k in range(1, 9)] + [(2 ** 15,), (4, 8, 256), (2 ** 15,), (1024, 64)],
          [(256,), (2048,), (2,), (256,), (2048,), (64, 64), (2,), (2,), (2,), (256,)]]


@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("shapes", UNEVEN)
def test_uneven_replay(emu, shapes, form):
    P.check_multi(emu, shapes, form)


@pytest.mark.gpu
@pytest.mark.parametrize("stream", [False, True])
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("shapes", UNEVEN + [[(2 ** 20,), (256,), (2048, 512), (2 ** 20,), (256,)]])
def test_uneven_gpu(lib, shapes, form, stream):
    P.check_multi(lib, shapes, form, stream=stream)


@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", ROWS + COLS + SPLIT)
def test_replay(emu, dims, batch, base, form):
    check(emu, dims, batch, base, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", ROWS + COLS + SPLIT + LONG)
def test_gpu(lib, dims, batch, base, form):
    check(lib, dims, batch, base, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,batch,base", [((4096,), 3, 2), ((256, 256), 1, 2), ((1 << 16,), 5, 2),
                                             ((1024, 512), 2, 2), ((64, 64, 64), 1, 4)])
def test_queued_calls(lib, dims, batch, base, form):
    """Calls queued on one stream that each overwrite their own input (every
    kernel may start before the one ahead of it has ended) give bit for bit
    what the same calls give when each is waited for."""
    dt = np.float64 if form == F64 else np.float32
    g = rng(5)
    shape = (batch,) + dims
    n = int(np.prod(dims))
    h = np.zeros(dims)
    h[(0,) * len(dims)] = 0.9
    h[(1,) * len(dims)] = 0.3
    d = P.Dev(lib)
    got = []
    try:
        plan = pac.Plan(lib, dims, batch, base, form)
        hr, hi = d.put(h), d.put(0.5 * h)
        Hr, Hi = d.zeros(dims, dt), d.zeros(dims, dt)
        plan.filter_spectrum(hr, hi, Hr, Hi)
        x = [g.standard_normal(shape).astype(dt) for _ in range(2)]
        for wait in (True, False):
            xr, xi = d.put(x[0]), d.put(x[1])
            for k in range(24):
                if k % 3 == 2:
                    plan.transform(pac.OP_FFT, xr, xi, xr, xi)
                    plan.transform(pac.OP_IFFT, xr, xi, xr, xi)
                else:
                    plan.convolve(xr, xi, Hr, Hi, xr, xi)
                if wait:
                    pac.check(lib, lib.pac_stream_synchronize(None), "sync")
            got.append((d.get(xr, shape, dt), d.get(xi, shape, dt)))
        plan.close()
    finally:
        d.free()
    assert n and np.isfinite(got[0][0]).all()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


# filter spectra stored in plan order by the transform's last pass: every row
# length, several filters, and a plan whose main schedule has other lines (the
# reorder stays a pass of its own); FP32 with h and hhat in the same memory
SPECTRA = ([((1 << k,), 3, 2, None) for k in (5, 6, 7, 8, 9, 10, 11, 12)] +
           [((8192,), 65, 2, None), ((1 << 15,), 2, 2, None), ((32, 512), 1, 2, None),
            ((4 ** 5,), 2, 4, None), ((8 ** 3,), 3, 8, None),
            ((1 << 14,), 2, 2, {"max_factor_log": 5}), ((1024,), 2, 2, {"max_radix_log": 3})])


def check_spectrum(L, dims, nf, base, tune, form):
    dt = np.float64 if form == F64 else np.float32
    shape = (nf,) + dims
    g = rng(3)
    h = [g.standard_normal(shape) for _ in range(2)]
    d = P.Dev(L)
    try:
        plan = pac.Plan(L, dims, nf, base, form, tune=tune)
        want = [d.zeros(shape, dt) for _ in range(2)]
        p64 = pac.Plan(L, dims, nf, base, F64)
        hp, at = [d.put(v) for v in h], [d.zeros(shape, np.float64) for _ in range(2)]
        p64.transform(pac.OP_AT, *hp, *at)
        pac.check(L, L.pac_spectrum_to_plan_order(plan.h, *at, nf, *want, 0.25, None), "order")
        want = [d.get(p, shape, dt) for p in want]
        got = []
        for alias in (False, True):  # hhat apart from h, and on top of it
            hp = [d.put(v) for v in h]
            out = hp if alias else [d.zeros(shape, dt) for _ in range(2)]
            plan.filter_spectrum(*hp, *out, nfilters=nf, scale=0.25)
            got.append([d.get(p, shape, dt) for p in out])
        plan.close()
        p64.close()
    finally:
        d.free()
    z = want[0] + 1j * want[1]
    for a in got:
        assert P.crel(a[0] + 1j * a[1], z) < (P.TOL if form == F64 else P.TOL_F32)


@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,nf,base,tune", SPECTRA)
def test_spectrum_replay(emu, dims, nf, base, tune, form):
    check_spectrum(emu, dims, nf, base, tune, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32])
@pytest.mark.parametrize("dims,nf,base,tune", SPECTRA)
def test_spectrum_gpu(lib, dims, nf, base, tune, form):
    check_spectrum(lib, dims, nf, base, tune, form)


# tensor-core plans: passes without a radix-16 stage run here, the others on
# the tensor cores, in one plan (64 x 256: the columns here, the rows there)
TC = [((64, 512), 1, 2), ((8, 64, 32), 2, 2), ((8 ** 4,), 3, 8), ((64, 256), 1, 2), ((512, 16), 3, 2)]


@pytest.mark.parametrize("dims,batch,base", TC)
def test_tc_replay(emu, orc, dims, batch, base):
    P.check_tc(emu, orc, dims, batch, base, ops=len(dims) < 3 and base == 2)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,batch,base", TC)
def test_tc_gpu(lib, orc, dims, batch, base):
    P.check_tc(lib, orc, dims, batch, base, ops=len(dims) < 3 and base == 2)
