"""The operator A (and the unordered FFT, which is A) runs on the kernels of
conj(A): A x = swap(conj(A) swap(x)) with real and imaginary parts exchanged,
bit for bit, and both agree with numpy; every kind of pass, in and out of
place."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

F64, F32, TC = pac.PAC_FORM_F64, pac.PAC_FORM_F32, pac.PAC_FORM_TC
SHAPES = [((16,), 3, 2), ((256,), 5, 2), ((4096,), 3, 2), ((8192,), 2, 2), ((1 << 14,), 3, 2),
          ((1 << 17,), 1, 2), ((4 ** 5,), 3, 4), ((8 ** 5,), 1, 8), ((2048, 8), 1, 2), ((4, 4096, 2), 1, 2),
          ((64, 32), 3, 2), ((64, 128, 32), 1, (8, 2, 2)), ((1, 1), 2, 2)]


def transform(L, dims, batch, base, form, op, x, inplace):
    dt = np.float64 if form == F64 else np.float32
    d = P.Dev(L)
    plan = pac.Plan(L, dims, batch, base, form)
    try:
        a = [d.put(v) for v in x]
        b = a if inplace else [d.zeros(x[0].shape, dt) for _ in range(2)]
        plan.transform(op, *a, *b)
        return [d.get(p, x[0].shape, dt) for p in b]
    finally:
        plan.close()
        d.free()


def check(L, dims, batch, base, form):
    dt = np.float64 if form == F64 else np.float32
    g = rng(2)
    shape = (batch,) + dims
    axes = tuple(range(1, len(shape)))
    x = [g.standard_normal(shape).astype(dt) for _ in range(2)]
    bases = base if isinstance(base, tuple) else (base,) * len(dims)
    rev = np.ix_(np.arange(batch), *[P.digit_reversal(b, v) for b, v in zip(bases, dims)])
    z = np.fft.fftn((x[0].astype(np.float64) + 1j * x[1])[rev], axes=axes)
    for inplace in (False, True):
        c = transform(L, dims, batch, base, form, pac.OP_CONJ_A, x[::-1], inplace)
        for op in (pac.OP_A, pac.OP_UFFT):
            a = transform(L, dims, batch, base, form, op, x, inplace)
            assert np.array_equal(a[0], c[1]) and np.array_equal(a[1], c[0])
            assert P.crel(a[0] + 1j * a[1], z) < (P.TOL if form == F64 else P.TOL_F32)


@pytest.mark.parametrize("form", [F64, F32, TC])
@pytest.mark.parametrize("dims,batch,base", SHAPES)
def test_replay(emu, dims, batch, base, form):
    check(emu, dims, batch, base, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [F64, F32, TC])
@pytest.mark.parametrize("dims,batch,base", SHAPES)
def test_gpu(lib, dims, batch, base, form):
    check(lib, dims, batch, base, form)
