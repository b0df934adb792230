"""One-stage columns run in CTAs of 64 units while they leave SMs empty, of 256
from there on: batches around a CTA's units and around the change (256 units to
an SM, 148 SMs), FP64 units and FP32 pairs of them, against numpy."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

CASES = [((16, 2), 31), ((16, 2), 33), ((4, 8), 8), ((8, 16), 5), ((2, 64), 1), ((16, 32), 1183),
         ((16, 32), 1185), ((16, 32), 2367), ((16, 32), 2369)]


def check(L, dims, batch, form):
    g = rng(batch)
    dt = np.float64 if form == pac.PAC_FORM_F64 else np.float32
    shape = (batch,) + dims
    x = (g.standard_normal(shape) + 1j * g.standard_normal(shape)).astype(
        np.complex128 if dt == np.float64 else np.complex64).astype(np.complex128)
    y = P.native_transform(L, dims, batch, 2, form, pac.OP_FFT, x)
    assert P.crel(y, np.fft.fftn(x, axes=(1, 2))) < (P.TOL if dt == np.float64 else P.TOL_F32)


@pytest.mark.parametrize("form", [pac.PAC_FORM_F64, pac.PAC_FORM_F32])
@pytest.mark.parametrize("dims,batch", CASES)
def test_replay(emu, dims, batch, form):
    check(emu, dims, batch, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [pac.PAC_FORM_F64, pac.PAC_FORM_F32])
@pytest.mark.parametrize("dims,batch", CASES)
def test_gpu(lib, dims, batch, form):
    check(lib, dims, batch, form)
