"""Kernel choices of the environment: PAC_PIPE=0 and PAC_SPECIAL_VARIANT=0 are
the built-in choices, bit for bit; under a choice of the scalar kernels a plan
has the factors that those are made for (the ones that the max_factor_log knob
gives at its largest value), so its spectrum order is that of such a plan."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

NAMES = ("PAC_COLTMA", "PAC_PIPE", "PAC_CLUSTER_VARIANT", "PAC_SPECIAL_VARIANT")


@pytest.fixture(autouse=True)
def unset(monkeypatch):
    for name in NAMES + ("PAC_MAX_FACTOR_LOG",):
        monkeypatch.delenv(name, raising=False)


def run(L, dims, batch, form, tune=None):
    """(spectrum, convolution)"""
    dt = np.float64 if form == pac.PAC_FORM_F64 else np.float32
    g = rng(8)
    shape = (batch,) + dims
    d = P.Dev(L)
    plan = pac.Plan(L, dims, batch, 2, form, tune=tune)
    try:
        H, y = [d.zeros(dims, dt) for _ in range(2)], [d.zeros(shape, dt) for _ in range(2)]
        plan.filter_spectrum(*[d.put(g.standard_normal(dims)) for _ in range(2)], *H)
        plan.convolve(*[d.put(g.standard_normal(shape).astype(dt)) for _ in range(2)], *H, *y)
        return np.array([d.get(p, dims, dt) for p in H]), np.array([d.get(p, shape, dt) for p in y])
    finally:
        plan.close()
        d.free()


def check_zero(L, dims, batch, form, monkeypatch, name):
    want = run(L, dims, batch, form)
    monkeypatch.setenv(name, "0")
    got = run(L, dims, batch, form)
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])


def check_choice(L, dims, batch, form, monkeypatch, name, value):
    want = run(L, dims, batch, form, tune={"max_factor_log": 13})
    monkeypatch.setenv(name, value)
    got = run(L, dims, batch, form)
    tol = P.TOL if form == pac.PAC_FORM_F64 else P.TOL_F32
    for u, v in zip(got, want):
        assert P.crel(u[0] + 1j * u[1], v[0] + 1j * v[1]) < tol


CASES = [((1 << 16,), 2), ((512, 64), 1), ((4096,), 3)]
FORMS = [pac.PAC_FORM_F64, pac.PAC_FORM_F32]
CHOICES = [("PAC_COLTMA", "0"), ("PAC_PIPE", "1"), ("PAC_CLUSTER_VARIANT", "0"),
           ("PAC_SPECIAL_VARIANT", "1")]


@pytest.mark.parametrize("name", ["PAC_PIPE", "PAC_SPECIAL_VARIANT"])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch", CASES)
def test_zero_replay(emu, monkeypatch, dims, batch, form, name):
    check_zero(emu, dims, batch, form, monkeypatch, name)


@pytest.mark.parametrize("name,value", CHOICES)
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch", CASES)
def test_choice_replay(emu, monkeypatch, dims, batch, form, name, value):
    check_choice(emu, dims, batch, form, monkeypatch, name, value)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["PAC_PIPE", "PAC_SPECIAL_VARIANT"])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch", CASES)
def test_zero_gpu(lib, monkeypatch, dims, batch, form, name):
    check_zero(lib, dims, batch, form, monkeypatch, name)


@pytest.mark.gpu
@pytest.mark.parametrize("name,value", CHOICES)
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,batch", CASES)
def test_choice_gpu(lib, monkeypatch, dims, batch, form, name, value):
    check_choice(lib, dims, batch, form, monkeypatch, name, value)
