"""Infinities, NaN and values far beyond any phase fraction in the tiles that an
interface crosses, and spacings far from 1, against the CPU oracle: the step, the
allocation-free step, the sweeps by tile kinds and the progress record's extremes.

Kernels leave terms out that are +-0 for ordinary values (a phase that is zero on
a stencil, off-diagonal constants that are zero); for others those terms are NaN or
an infinity and have to be there.  FP64 results are the oracle's to the last bit
(zeros of either sign and all NaN are equal), so there is no tolerance.
"""
import ctypes

import numpy as np
import pytest

import eshwar_dipan_b200 as gp
from eshwar_dipan_b200 import _abi
from gp_cases import PARITY_CASES, write_case
from oracle_py import Oracle, bits_equal, mismatch_report

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")
MESH = (88, 104)
SEEDS = [(0, 22, 24, 12.0), (1, 62, 30, 11.0), (0, 50, 78, 13.0), (1, 24, 70, 10.0)]
# mu at places across the interfaces; phi of one phase there; phi of all but the liquid
PLANTS = {
    "mu_inf": ("mu", [INF, -INF]),
    "mu_nan": ("mu", [NAN]),
    "mu_huge": ("mu", [1e19, -1e160, 1e300]),
    "phi_inf": ("phi", [INF, -INF]),
    "phi_nan": ("phi", [NAN]),
    "phi_huge": ("phi", [1e19, -1e19, 1e160, -1e300]),
    "phi_out_of_range": ("phi", [1.5, -0.25, 40.0, -3.0]),
}
SYSTEMS = {
    "three_aniso": dict(N=3, K=2, dab=0.02),
    "three_rotated": dict(N=3, K=1, dab=[0.0, 0.02, 0.02], rot={(0, 2): 30.0, (1, 2): 45.0}, bc_phi=(3, 3, 1, 1)),
    "four_iso": dict(N=4, K=2, aniso=False, dab=0.0, dx=1.5, dt=0.04),
    "four_aniso_coupled": dict(N=4, K=2, dab=0.02, A_off=0.25, bc_phi=(3, 3, 3, 3)),
    "two_aniso": dict(N=2, K=1, dab=0.03),
}


def _same(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    return np.array_equal(na, nb) and bits_equal(np.where(na, 0.0, a), np.where(nb, 0.0, b))


def _diff(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    w = np.argwhere(~((na & nb) | (a == b)))
    return "%d differ, first %s: %r, oracle %r" % (len(w), w[0], a[tuple(w[0])], b[tuple(w[0])]) if len(w) else "same"


def _state(tmp_path, system, plant):
    kw = dict(SYSTEMS[system])
    seeds = [(min(a, kw["N"] - 2), x, y, r) for a, x, y, r in SEEDS]
    ip, fp = write_case(str(tmp_path), system, dict(kw, mesh=MESH, d_solid=0.0), seeds=seeds)
    p = gp.load_params(ip)
    o = Oracle(p, recip_div=1)
    o.set(*gp.fill(p, fp))
    o.smooth(9)
    o.step(4)
    phi, mu = o.get()
    o.close()
    field, values = PLANTS[plant]
    # around every seed from inside the interface to three cells outside, no two
    # within each other's stencils
    q, rng = 0, np.random.default_rng(11)
    for s, (_, cx, cy, r) in enumerate(seeds):
        for i in range(8):
            ang = 2 * np.pi * (i + 0.3 * s) / 8
            d = r + (-3, -1, 0, 1, 2, 3, 4, 5)[(i + 3 * s) % 8]
            x, y = int(round(cx + d * np.cos(ang))), int(round(cy + d * np.sin(ang)))
            f = mu if field == "mu" else phi
            f[int(rng.integers(f.shape[0])), x, y] = values[q % len(values)]
            q += 1
    return p, phi, mu


@pytest.mark.parametrize("plant", sorted(PLANTS))
@pytest.mark.parametrize("system", sorted(SYSTEMS))
def test_step(tmp_path, system, plant):
    p, phi, mu = _state(tmp_path, system, plant)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    with gp.Simulation(p, phi, mu) as sim:
        for n in range(2):
            o.step(1)
            try:
                st = sim.step(1)
            except gp.NonFiniteError as e:
                st = e.stats
            for what, a, b in zip(("phi", "mu"), sim.get(), o.get()):
                assert _same(a, b), "%s after step %d: %s" % (what, n + 1, _diff(a, b))
            ost = o.stats()
            for k in ("phi_max", "phi_min", "mu_max", "mu_min"):
                assert st[k] == ost[k], (k, n)
    if plant not in ("phi_out_of_range", "mu_huge"):
        assert not np.isfinite(np.concatenate(o.get())).all() or plant == "phi_huge"


@pytest.mark.parametrize("plant", sorted(PLANTS))
@pytest.mark.parametrize("system", ["three_aniso", "three_rotated", "four_iso"])
def test_noalloc(tmp_path, system, plant):
    import torch
    p, phi, mu = _state(tmp_path, system, plant)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    o.step(1)
    L = _abi.lib()
    src = [torch.from_numpy(np.array(a)).cuda() for a in (phi, mu)]
    dst = [torch.zeros_like(a) for a in src]
    stream = torch.cuda.current_stream()
    rc = L.gp_step_noalloc(ctypes.byref(p), src[0].data_ptr(), src[1].data_ptr(), dst[0].data_ptr(),
                           dst[1].data_ptr(), ctypes.c_void_p(stream.cuda_stream))
    assert rc == 0, L.gp_last_error(None)
    for what, a, b in zip(("phi", "mu"), dst, o.get()):
        assert _same(a.cpu().numpy(), b), "%s: %s" % (what, _diff(a.cpu().numpy(), b))


@pytest.mark.parametrize("plant", sorted(PLANTS))
@pytest.mark.parametrize("system", ["three_aniso", "four_iso", "four_aniso_coupled"])
def test_smooth_by_tile_kinds(tmp_path, system, plant):
    p, phi, mu = _state(tmp_path, system, plant)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    o.smooth(2)
    b = gp.Batch([p] * 4, [(phi, mu)] * 4, precision=gp.GP_FP64)
    b.smooth(2)
    for what, x, y in zip(("phi", "mu"), b.get(3), o.get()):
        assert _same(x, y), "%s: %s" % (what, _diff(x, y))
    b.close()


@pytest.mark.parametrize("system", ["three_aniso", "four_aniso_coupled", "four_iso", "two_aniso"])
@pytest.mark.parametrize("plant", ["mu_inf", "mu_nan", "mu_huge"])
def test_bulk_tiles(tmp_path, system, plant):
    """Values in liquid far from any interface, inside the domain and at its edges:
    fields, extremes and the two sweeps by tile kinds."""
    kw, mesh = SYSTEMS[system], (160, 256)
    ip, fp = write_case(str(tmp_path), "b", dict(kw, mesh=mesh, d_solid=0.0), seeds=[(0, 30, 40, 10.0)])
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    values = PLANTS[plant][1]
    for i, (x, y) in enumerate([(100, 200), (100, 120), (90, 40), (140, 223), (120, 160), (0, 150), (80, 255), (159, 90)]):
        mu[i % mu.shape[0], x, y] = values[i % len(values)]
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    with gp.Simulation(p, phi, mu) as sim:
        for n in range(2):
            o.step(1)
            try:
                st = sim.step(1)
            except gp.NonFiniteError as e:
                st = e.stats
            for what, a, b in zip(("phi", "mu"), sim.get(), o.get()):
                assert _same(a, b), "%s after step %d: %s" % (what, n + 1, _diff(a, b))
            ost = o.stats()
            for k in ("phi_max", "phi_min", "mu_max", "mu_min"):
                assert st[k] == ost[k], (k, n)
    o.set(phi, mu)
    o.smooth(2)
    b = gp.Batch([p] * 4, [(phi, mu)] * 4, precision=gp.GP_FP64)
    b.smooth(2)
    for what, x, y in zip(("phi", "mu"), b.get(1), o.get()):
        assert _same(x, y), "sweep, %s: %s" % (what, _diff(x, y))
    b.close()


@pytest.mark.parametrize("name", ["bin_iso_antitrap", "ternary3_aniso_periodic", "dilute_three_phase"])
@pytest.mark.parametrize("dx", [3e-20, 5e20, 0.5 ** 64])
def test_spacings_beyond_the_quick_range(tmp_path, name, dx):
    """Outside [2**-60, 2**60) every division by a spacing is a division.  The
    other lengths and the time step scale with the spacing, so the fields stay
    ordinary."""
    c = PARITY_CASES[name]
    kw = dict(c["kw"])
    old = kw.get("dx", 1.0)
    kw.update(dx=dx, dt=kw.get("dt", 0.02) * (dx / old) ** 2, eps=kw.get("eps", 4.0) * dx / old)
    ip, fp = write_case(str(tmp_path), "dx", kw, seeds=c["seeds"])
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    with gp.Simulation(p, phi, mu) as sim:
        for what, n in (("smooth", 3), ("step", 1), ("step", 3)):
            getattr(o, what)(n)
            getattr(sim, what)(n)
            for a, b in zip(sim.get(), o.get()):
                assert np.isfinite(b).all()
                assert bits_equal(a, b), "%s: %s" % (what, mismatch_report(a, b))
