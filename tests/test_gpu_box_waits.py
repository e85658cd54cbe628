"""Every bounded wait on a box of the step kernels runs out and is reported by
itself: bulk tiles and interface tiles, in the single launch and in the two
kernels (which a step with statistics and GP_SPLIT_KERNELS take), FP64 and FP32,
and the bulk tiles of a sweep.  The barriers of one kind expect more bytes than a
box brings (GP_TEST_TMA_SHORTFALL, GP_TEST_TMA_KIND), the other kind's are as always;
the GPU stays usable, and a new context steps as the oracle does.
"""
import numpy as np
import pytest

import eshwar_dipan_b200 as gp
from gp_cases import write_case
from oracle_py import Oracle, bits_equal

pytestmark = pytest.mark.gpu


def _case(tmp_path):
    ip, fp = write_case(str(tmp_path), "w", dict(N=2, K=1, mesh=(160, 224), dab=0.03, d_solid=0.0),
                        seeds=[(0, 80, 100, 20.0)])
    p = gp.load_params(ip)
    return (p,) + gp.fill(p, fp)


def _short(monkeypatch, kind):
    monkeypatch.setenv("GP_TEST_TMA_SHORTFALL", "16")
    monkeypatch.setenv("GP_TEST_TMA_KIND", kind)


def _usable(monkeypatch, p, phi, mu):
    monkeypatch.delenv("GP_TEST_TMA_SHORTFALL")
    monkeypatch.delenv("GP_TEST_TMA_KIND")
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    o.smooth(2)
    o.step(3)
    with gp.Simulation(p, phi, mu) as s:
        s.smooth(2)
        s.step(3, stats=False)
        for a, b in zip(s.get(), o.get()):
            assert bits_equal(a, b)


@pytest.mark.parametrize("kind", ["bulk", "interface"])
@pytest.mark.parametrize("form", ["single", "split", "stats"])
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
def test_step(tmp_path, monkeypatch, kind, form, prec):
    p, phi, mu = _case(tmp_path)
    if form == "split":
        monkeypatch.setenv("GP_SPLIT_KERNELS", "1")
    monkeypatch.setenv("GP_NO_TUNING", "1")
    with gp.Simulation(p, phi, mu, precision=getattr(gp, "GP_" + prec)) as s:
        s.smooth(2)
        assert s.kernel_times(1)["fused"] == (form != "split")
    _short(monkeypatch, kind)
    with gp.Simulation(p, phi, mu, precision=getattr(gp, "GP_" + prec)) as s:
        with pytest.raises(gp.GpError, match="did not arrive") as ei:
            s.step(1, stats=form == "stats")
        assert ei.value.code == gp.GP_ETIMEOUT
    _usable(monkeypatch, p, phi, mu)


@pytest.mark.parametrize("kind", ["bulk", "interface"])
def test_sweep(tmp_path, monkeypatch, kind):
    """Four simulations sweep by tile kinds: bulk tiles from boxes, the others by
    ordinary loads."""
    p, phi, mu = _case(tmp_path)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    o.smooth(2)
    _short(monkeypatch, kind)
    b = gp.Batch([p] * 4, [(phi, mu)] * 4, precision=gp.GP_FP64)
    try:
        if kind == "bulk":
            with pytest.raises(gp.GpError, match="did not arrive") as ei:
                b.smooth(2)
            assert ei.value.code == gp.GP_ETIMEOUT
        else:
            b.smooth(2)
            for x, y in zip(b.get(2), o.get()):
                assert np.array_equal(x, y)
    finally:
        b.close()
    _usable(monkeypatch, p, phi, mu)
