"""Host copies of the fft.h functions: small calls through an entry's pinned
block, large ones through the pool of copy threads (arrays below and above a
pool slot of 1 MiB), several callers at once (one has the pool, the others
take the driver's way), against numpy."""
import threading

import numpy as np
import pytest

import parity as P
from conftest import O, pac, rng

# the largest shape of a pinned block is 2^15 elements
SHAPES = [((1 << 15,), 2), ((1 << 16,), 4), ((256, 512), 2), ((64, 64, 64), 4)]
SHAPES_GPU = SHAPES + [((1 << 18,), 2), ((512, 1024), 2), ((1 << 20,), 4)]


def check(L, shape, r, threads):
    g = rng(int(np.prod(shape)) + r)
    data = [[g.standard_normal(shape) for _ in range(4)] for _ in range(threads)]
    out, err = [None] * threads, []

    def call(k):
        try:
            out[k] = [pac.dropin_convolution(L, O.METHOD_PAC, r, *data[k]) for _ in range(2)]
            out[k].append(pac.dropin_transform(L, 0, r, *data[k][:2]))
        except Exception as e:  # told by the main thread
            err.append(e)

    ts = [threading.Thread(target=call, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not err and L.pac_get_last_status() == 0
    rev = np.ix_(*[P.digit_reversal(r, n) for n in shape])
    for k in range(threads):
        x, h = data[k][0] + 1j * data[k][1], data[k][2] + 1j * data[k][3]
        fx, fh = np.fft.fftn(x), np.fft.fftn(h)
        for y in out[k][:2]:
            assert P.crel(y[0] + 1j * y[1], np.fft.ifftn(fx * fh)) < P.TOL
            assert P.crel(y[2] + 1j * y[3], fh[rev]) < P.TOL
        assert P.crel(out[k][2][0] + 1j * out[k][2][1], fx) < P.TOL


@pytest.mark.parametrize("threads", [1, 3])
@pytest.mark.parametrize("shape,r", SHAPES)
def test_replay(emu, shape, r, threads):
    check(emu, shape, r, threads)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [1, 3])
@pytest.mark.parametrize("shape,r", SHAPES_GPU)
def test_gpu(lib, shape, r, threads):
    check(lib, shape, r, threads)
