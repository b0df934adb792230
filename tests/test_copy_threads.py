"""Host copies of the fft.h functions start threads only for arrays that gain
from them: below 2 MiB an array the calling thread copies alone (results at
sizes around it: test_host_copies.py)."""
import os

import numpy as np
import pytest

import parity as P
from conftest import O, pac, rng


@pytest.mark.parametrize("log2,most", [(12, 0), (16, 1), (17, 1), (18, 4), (19, 4)])
def test_threads(emu, log2, most):
    n = 1 << log2
    g = rng(log2)
    a = [g.standard_normal((2, n // 2)) for _ in range(4)]
    emu.pac_emu_copy_threads()
    y = pac.dropin_convolution(emu, O.METHOD_PAC, 2, *a)
    threads = emu.pac_emu_copy_threads()
    x, h = a[0] + 1j * a[1], a[2] + 1j * a[3]
    assert P.crel(y[0] + 1j * y[1], np.fft.ifft2(np.fft.fft2(x) * np.fft.fft2(h))) < P.TOL
    if most <= 1:
        assert threads == most
    elif os.cpu_count() > 1:
        assert threads > 1
