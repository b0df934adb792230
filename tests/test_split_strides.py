"""Factors of an axis are chosen for the stride that the passes will meet: a
trailing axis of one point changes nothing, and an axis beside a very short
one is not split for column tiles that do not fit between its neighbours."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

FORMS = [pac.PAC_FORM_F64, pac.PAC_FORM_F32]


def passes(L, dims, batch, base, form):
    plan = pac.Plan(L, dims, batch, base, form)
    n = plan.info().conv_passes
    plan.close()
    return n


def check(L, dims, batch, base, form):
    g = rng(int(np.prod(dims)))
    shape = (batch,) + dims
    axes = tuple(range(1, len(shape)))
    tol = P.TOL if form == pac.PAC_FORM_F64 else P.TOL_F32
    x = g.standard_normal(shape) + 1j * g.standard_normal(shape)
    h = g.standard_normal(dims) + 1j * g.standard_normal(dims)
    assert P.crel(P.native_conv(L, dims, batch, base, form, x, h), P.fftconv(x, h[None], axes)) < tol
    fx = np.fft.fftn(x, axes=axes)
    assert P.crel(P.native_transform(L, dims, batch, base, form, pac.OP_FFT, x), fx) < tol
    y = P.native_transform(L, dims, batch, base, form, pac.OP_IFFT, fx)
    assert P.crel(y, x) < tol


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,base", [((4096,), 2), ((8192,), 2), ((1 << 16,), 2), ((2048,), 2),
                                       ((64, 512), 2), ((4096,), 4), ((512,), 8)])
@pytest.mark.parametrize("batch", [1, 200])
def test_trailing_ones(emu, dims, base, form, batch):
    n = passes(emu, dims, batch, base, form)
    while len(dims) < 3:
        dims += (1,)
        assert passes(emu, dims, batch, base, form) == n


NARROW = [((4096, 2), 3, 2), ((4096, 4), 1, 2), ((4096, 1), 5, 2), ((8192, 1, 1), 2, 2), ((64, 2), 7, 2),
          ((128, 4), 2, 2), ((256, 2, 2), 2, 2), ((1024, 2), 1, 2), ((2048, 2), 1, 2), ((2048, 4), 1, 2),
          ((2048, 8), 1, 2), ((2, 4096, 2), 1, 2), ((4096, 4), 1, 4), ((512, 8), 1, 8),
          ((1 << 14, 2), 1, 2), ((4 ** 7, 4), 1, 4)]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch,base", NARROW)
def test_narrow_replay(emu, dims, batch, base, form):
    check(emu, dims, batch, base, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch,base", NARROW)
def test_narrow_gpu(lib, dims, batch, base, form):
    check(lib, dims, batch, base, form)
