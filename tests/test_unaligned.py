"""Arrays that do not start at a multiple of 16 bytes (slices of larger ones)
run on the kernels over 8-byte elements, whose tiles the CTA's threads then copy
in: the same results bit for bit as with aligned arrays wherever every pass can
(rows at any offset, columns at multiples of 8 bytes), for every line length,
base and operator, one array at a time and all of them; and numpy's within the
tolerance everywhere, FP32 columns at odd offsets among them."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import pac, rng

F64, F32 = pac.PAC_FORM_F64, pac.PAC_FORM_F32
ROWS = ([((1 << k,), b, 2) for k in range(5, 13) for b in (1, 3)] + [((8192,), 131, 2)] +
        [((4 ** k,), 5, 4) for k in range(3, 7)] + [((8 ** k,), 5, 8) for k in range(2, 5)])
COLS = ([((1 << k, 256), 1, 2) for k in range(1, 11)] + [((4 ** k, 64), 2, 4) for k in range(1, 6)] +
        [((8 ** k, 64), 1, 8) for k in range(1, 4)] + [((1 << 14,), 3, 2), ((1 << 17,), 1, 2),
         ((8 ** 5,), 1, 8), ((64, 128, 32), 1, (8, 2, 2))])
LONG = [((1 << 20,), 1, 2), ((1 << 21,), 1, 2)]
# arrays off their boundary: all; the input alone; one part of the output alone
OFF = [(1, 1, 1, 1), (1, 0, 0, 0), (0, 0, 0, 1)]


class Placed:
    """Device arrays, each `off` elements into a block of its own."""

    def __init__(self, L):
        self.d = P.Dev(L)

    def put(self, a, off):
        flat = np.concatenate([np.zeros(off, a.dtype), a.ravel(), np.zeros(8, a.dtype)])
        return C.c_void_p(self.d.put(flat).value + off * a.itemsize)

    def get(self, p, shape, dt):
        return self.d.get(p, shape, dt)


def results(L, dims, batch, base, form, step, off):
    """spectrum, convolution and every operator with (in re, in im, out re, out
    im) off by `step` elements where `off` says so"""
    dt = np.float64 if form == F64 else np.float32
    g = rng(6)
    shape = (batch,) + dims
    x = [g.standard_normal(shape).astype(dt) for _ in range(2)]
    h = [g.standard_normal(dims) for _ in range(2)]
    o = [step * v for v in off]
    a = Placed(L)
    plan = pac.Plan(L, dims, batch, base, form)
    out = {}
    try:
        H = [a.put(np.zeros(dims, dt), v) for v in o[2:]]
        plan.filter_spectrum(*[a.put(v, k) for v, k in zip(h, o)], *H)
        out["spectrum"] = [a.get(p, dims, dt) for p in H]
        xs = [a.put(v, k) for v, k in zip(x, o)]
        y = [a.put(np.zeros(shape, dt), v) for v in o[2:]]
        plan.convolve(*xs, *H, *y)
        out["conv"] = [a.get(p, shape, dt) for p in y]
        for op in (pac.OP_AT, pac.OP_A, pac.OP_CONJ_A, pac.OP_FFT, pac.OP_IFFT):
            plan.transform(op, *xs, *y)
            out[op] = [a.get(p, shape, dt) for p in y]
    finally:
        plan.close()
        a.d.free()
    z = np.fft.fftn(x[0].astype(np.float64) + 1j * x[1], axes=tuple(range(1, len(shape))))
    tol = P.TOL if form == F64 else P.TOL_F32
    assert P.crel(out[pac.OP_FFT][0] + 1j * out[pac.OP_FFT][1], z) < tol
    y = np.fft.ifftn(z * np.fft.fftn(h[0] + 1j * h[1]), axes=tuple(range(1, len(shape))))
    c = out["conv"]
    n = float(np.prod(dims))  # the plan's default scale is 1 / n of the filter
    assert P.crel(c[0] + 1j * c[1], y) < tol, n
    return out


def check(L, dims, batch, base, form, step, exact):
    want = results(L, dims, batch, base, form, 0, (0, 0, 0, 0))
    for off in OFF:
        got = results(L, dims, batch, base, form, step, off)
        for k in want:
            if exact:
                assert all(np.array_equal(u, v) for u, v in zip(got[k], want[k])), (off, k)


# (form, elements off, columns too)
STEPS = [(F64, 1, True), (F32, 2, True), (F32, 1, False), (F32, 3, False)]


@pytest.mark.parametrize("form,step,cols", STEPS)
@pytest.mark.parametrize("dims,batch,base", ROWS)
def test_rows_replay(emu, dims, batch, base, form, step, cols):
    check(emu, dims, batch, base, form, step, True)


@pytest.mark.parametrize("form,step,cols", STEPS)
@pytest.mark.parametrize("dims,batch,base", COLS)
def test_columns_replay(emu, dims, batch, base, form, step, cols):
    check(emu, dims, batch, base, form, step, cols)


@pytest.mark.gpu
@pytest.mark.parametrize("form,step,cols", STEPS)
@pytest.mark.parametrize("dims,batch,base", ROWS)
def test_rows_gpu(lib, dims, batch, base, form, step, cols):
    check(lib, dims, batch, base, form, step, True)


@pytest.mark.gpu
@pytest.mark.parametrize("form,step,cols", STEPS)
@pytest.mark.parametrize("dims,batch,base", COLS + LONG)
def test_columns_gpu(lib, dims, batch, base, form, step, cols):
    check(lib, dims, batch, base, form, step, cols)


UNEVEN = [(256,), (64, 32), (256,), (1 << 14,), (4096,), (8, 256), (1 << 14,)]


def check_uneven(L, form, step):
    dt = np.float64 if form == F64 else np.float32
    m = pac.MultiPlan(L, UNEVEN, 2, form)
    n = int(m.offsets[-1])
    g = rng(12)
    x = [g.standard_normal(n).astype(dt) for _ in range(2)]
    h = [g.standard_normal(n) for _ in range(2)]
    a = Placed(L)
    got = []
    try:
        for off in (0, step):
            H = [a.put(np.zeros(n, dt), off) for _ in range(2)]
            y = [a.put(np.zeros(n, dt), off) for _ in range(2)]
            m.filter_spectra(*[a.put(v, off) for v in h], *H)
            m.convolve(*[a.put(v, off) for v in x], *H, *y)
            got.append([a.get(p, (n,), dt) for p in y])
    finally:
        m.close()
        a.d.free()
    for p, shape in enumerate(UNEVEN):
        s = slice(int(m.offsets[p]), int(m.offsets[p + 1]))
        z = np.fft.ifftn(np.fft.fftn((x[0][s].astype(np.float64) + 1j * x[1][s]).reshape(shape)) *
                         np.fft.fftn((h[0][s] + 1j * h[1][s]).reshape(shape)))
        for y in got:
            e = P.crel((y[0][s] + 1j * y[1][s]).reshape(shape), z)
            assert e < (P.TOL if form == F64 else P.TOL_F32)


@pytest.mark.parametrize("form,step", [(F64, 1), (F32, 1), (F32, 2)])
def test_uneven_replay(emu, form, step):
    check_uneven(emu, form, step)


@pytest.mark.gpu
@pytest.mark.parametrize("form,step", [(F64, 1), (F32, 1), (F32, 2)])
def test_uneven_gpu(lib, form, step):
    check_uneven(lib, form, step)
