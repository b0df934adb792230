"""FP32 filter spectra that share memory with the FP64 filters they come from:
the transform rounds 8-byte values to 4-byte ones, so the place of a line's
output holds the input of another line.  hhat packed on the first half of
h_re's bytes, on its second half, and part by part on h, with more lines than
a tile (the last alias is the one that only an order of the lines can get
right), against the same call with memory of its own, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import pac, rng

# one factor (a pass reads h and writes hhat), and two
SHAPES = [((256,), 96, 2), ((512,), 64, 2), ((1024,), 96, 2), ((4096,), 33, 2), ((64,), 200, 4),
          ((512,), 64, 8), ((1 << 14,), 8, 2), ((64, 256), 8, 2)]


def at(p, n):
    return C.c_void_p(p.value + n)


def check(L, dims, nf, base):
    shape = (nf,) + dims
    n = int(np.prod(shape))
    g = rng(11)
    h = [g.standard_normal(shape) for _ in range(2)]
    d = P.Dev(L)
    plan = pac.Plan(L, dims, nf, base, pac.PAC_FORM_F32)
    try:
        hp, out = [d.put(v) for v in h], [d.zeros(shape, np.float32) for _ in range(2)]
        plan.filter_spectrum(*hp, *out, nfilters=nf, scale=0.25)
        want = [d.get(p, shape, np.float32) for p in out]
        fh = np.fft.fftn(h[0] + 1j * h[1], axes=tuple(range(1, len(shape))))
        assert np.isclose(np.linalg.norm(want), 0.25 * np.linalg.norm(fh), rtol=1e-5)
        for where in ("first half", "second half", "part on part"):
            hp = [d.put(v) for v in h]
            if where == "part on part":
                out = hp
            else:
                out = [at(hp[0], 0), at(hp[0], 4 * n)]
                if where == "second half":
                    out.reverse()
            plan.filter_spectrum(*hp, *out, nfilters=nf, scale=0.25)
            got = [d.get(p, shape, np.float32) for p in out]
            for a, b in zip(got, want):
                assert np.array_equal(a, b), where
    finally:
        plan.close()
        d.free()


@pytest.mark.parametrize("dims,nf,base", SHAPES)
def test_replay(emu, dims, nf, base):
    check(emu, dims, nf, base)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,nf,base", SHAPES)
def test_gpu(lib, dims, nf, base):
    check(lib, dims, nf, base)
