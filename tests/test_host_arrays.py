"""Host arrays of the fft.h functions that are not plain memory of their own:
a device or managed array beside ordinary ones (copied by the driver, never
through the pinned slots that the copy threads read and write on the host), in
small and large calls and while another shape holds the slots; arrays shared
between the signal and the filter, whose last writer is the signal.

On the host replay a "device" array is an address range whose bytes live
elsewhere and that only copies reach; on the GPU it is managed memory."""
import ctypes as C

import numpy as np
import pytest

import parity as P
from conftest import pac, rng

DP = C.POINTER(C.c_double)
# all arrays of the first two fit a pinned block, the others use the slots
SHAPES = [((64,), 2), ((1 << 12,), 2), ((1 << 16,), 2), ((256, 1024), 2)]
LARGE = (1 << 17,)


def ptr(a):
    return a.ctypes.data_as(DP) if isinstance(a, np.ndarray) else C.cast(a, DP)


def call(L, fn, shape, r, arrays):
    nd = len(shape)
    name = fn + ("" if nd == 1 else f"_{nd}d")
    tw = [None] * (2 * nd + (fn == "fft_based_convolution"))
    f = getattr(L, name)
    f(ptr(arrays[0]), ptr(arrays[1]), *shape, r, *tw, ptr(arrays[2]), ptr(arrays[3]))
    assert L.pac_get_last_status() == 0


def want(shape, r, data, fn):
    x, h = data[0] + 1j * data[1], data[2] + 1j * data[3]
    fh = np.fft.fftn(h)
    y = np.fft.ifftn(np.fft.fftn(x) * fh)
    rev = np.ix_(*[P.digit_reversal(r, n) for n in shape])
    s = fh[rev] if fn.startswith("perm") else fh
    return [y.real, y.imag, s.real, s.imag]


def check_mixed(L, shape, r, make):
    """make(array) -> (pointer, read, release)"""
    g = rng(3)
    big = [g.standard_normal(LARGE) for _ in range(4)]
    call(L, "permutation_avoiding_convolution", LARGE, 2, big)  # the slots exist
    for fn in ("permutation_avoiding_convolution", "fft_based_convolution"):
        for which in ((1,), (0, 3), (2, 3), (0, 1, 2, 3)):
            data = [g.standard_normal(shape) for _ in range(4)]
            arrays, read, drop = [], [], []
            for k, a in enumerate(data):
                if k in which:
                    p, get, rel = make(a)
                    arrays.append(p)
                    read.append(get)
                    drop.append(rel)
                else:
                    b = a.copy()
                    arrays.append(b)
                    read.append(lambda b=b: b)
            call(L, fn, shape, r, arrays)
            got = [f().copy() for f in read]
            for rel in drop:
                rel()
            for k, (u, v) in enumerate(zip(got, want(shape, r, data, fn))):
                assert np.abs(u.reshape(shape) - v).max() < 1e-9, (fn, which, k)


def check_shared(L, shape, r):
    """im and h_im are one array; then every array is the same one."""
    g = rng(4)
    for fn in ("permutation_avoiding_convolution", "fft_based_convolution"):
        re, hr, zero = g.standard_normal(shape), g.standard_normal(shape), np.zeros(shape)
        z = want(shape, r, [re, zero, hr, zero], fn)
        im = zero.copy()
        a, b = re.copy(), hr.copy()
        call(L, fn, shape, r, [a, im, b, im])
        for u, v in zip((a, im, b), (z[0], z[1], z[2])):
            assert np.abs(u - v).max() < 1e-9, fn
        z = want(shape, r, [re, re, re, re], fn)
        a = re.copy()
        call(L, fn, shape, r, [a] * 4)
        assert np.abs(a - z[1]).max() < 1e-9, fn


@pytest.mark.parametrize("shape,r", SHAPES)
def test_mixed_replay(emu, shape, r):
    emu.pac_emu_device_array.argtypes = [C.c_void_p, C.c_size_t, C.c_void_p]

    def make(a):
        shadow, face = a.copy(), np.full(a.shape, 1e30)
        emu.pac_emu_device_array(face.ctypes.data, face.nbytes, shadow.ctypes.data)

        def release():
            emu.pac_emu_device_array(face.ctypes.data, 0, None)
            assert (face == 1e30).all()  # the host wrote nothing there
        return face, (lambda: shadow), release

    check_mixed(emu, shape, r, make)


@pytest.mark.parametrize("shape,r", SHAPES)
def test_shared_replay(emu, shape, r):
    check_shared(emu, shape, r)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,r", SHAPES)
def test_mixed_gpu(lib, shape, r):
    from cuda.bindings import runtime as rt

    def make(a):
        err, p = rt.cudaMallocManaged(a.nbytes, rt.cudaMemAttachGlobal)
        assert int(err) == 0
        view = np.ctypeslib.as_array(C.cast(p, DP), shape=(a.size,))
        view[:] = a.ravel()
        return C.c_void_p(p), (lambda: view), (lambda: rt.cudaFree(p))

    check_mixed(lib, shape, r, make)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,r", SHAPES)
def test_shared_gpu(lib, shape, r):
    check_shared(lib, shape, r)
