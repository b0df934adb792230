"""Knobs of 0, and no knobs, are a multi-plan's built-in choices: the plan that
pac_multi_create makes, tile for tile and with the same spectra -- what the
tuner measures its candidates against."""
import numpy as np
import pytest

import parity as P
from conftest import pac, rng

SHAPES = [(1 << 18,), (256,), (1024, 64), (1 << 15,), (256,), (4096, 32)]


def made(L, form, tune):
    dt = np.float64 if form == pac.PAC_FORM_F64 else np.float32
    m = pac.MultiPlan(L, SHAPES, 2, form, tune=tune)
    n = int(m.offsets[-1])
    g = rng(1)
    d = P.Dev(L)
    try:
        h = [d.put(g.standard_normal(n)) for _ in range(2)]
        H, y = [d.zeros(n, dt) for _ in range(2)], [d.zeros(n, dt) for _ in range(2)]
        m.filter_spectra(*h, *H)
        m.convolve(*[d.put(g.standard_normal(n).astype(dt)) for _ in range(2)], *H, *y)
        info = m.info()
        return (info["items"], info["fast_items"]), [d.get(p, (n,), dt) for p in H + y]
    finally:
        m.close()
        d.free()


def check(L, form):
    items, want = made(L, form, None)
    got_items, got = made(L, form, {})
    assert got_items == items
    for u, v in zip(got, want):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("form", [pac.PAC_FORM_F64, pac.PAC_FORM_F32, pac.PAC_FORM_TC])
def test_replay(emu, monkeypatch, form):
    monkeypatch.delenv("PAC_TUNE_CACHE", raising=False)
    check(emu, form)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [pac.PAC_FORM_F64, pac.PAC_FORM_F32, pac.PAC_FORM_TC])
def test_gpu(lib, monkeypatch, form):
    monkeypatch.delenv("PAC_TUNE_CACHE", raising=False)
    check(lib, form)
