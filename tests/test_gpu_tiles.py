"""Tile edges and spacings of the step, of the smoothing sweeps and of
gp_step_noalloc, against the CPU oracle, bit for bit.

A tile is 8 rows by 32 columns.  The meshes lie one cell below, at and one cell
above whole tiles, one has more tiles than blocks resident on a GPU, and the
spacings are not powers of two (their divisions are corrected multiplications).
FP64 results are the oracle's to the last bit, so there is no tolerance.
"""
import ctypes

import numpy as np
import pytest

import eshwar_dipan_b200 as gp
from eshwar_dipan_b200 import _abi
from gp_cases import random_seeds, write_case
from oracle_py import Oracle, bits_equal, mismatch_report

pytestmark = pytest.mark.gpu

# mesh, spacing, phases, solutes, further parameters
CASES = {
    "below": ((15, 31), 0.7, 2, 1, dict(dab=0.03, d_solid=0.0)),
    "whole": ((16, 64), 1.5, 3, 2, dict(dab=0.02, A_off=0.25)),
    "above": ((17, 65), 1.1, 4, 2, dict(dab=0.02, bc_phi=(3, 3, 1, 1))),
    "one_tile_periodic": ((8, 32), 3.0, 2, 1, dict(dab=0.03, bc_phi=(3, 3, 3, 3))),
    "iso": ((25, 97), 0.3, 3, 1, dict(aniso=False, dab=0.0)),
    "many_tiles": ((200, 425), 1.3, 2, 1, dict(dab=0.03, bc_phi=(1, 1, 3, 3))),
}


def _start(tmp_path, name):
    mesh, dx, N, K, kw = CASES[name]
    big = min(mesh) / 4.0
    seeds = random_seeds(max(2, mesh[0] * mesh[1] // 3000), mesh, big / 2 if big < 8 else 4.0, min(big, 8.0), N - 1, 7)
    ip, fp = write_case(str(tmp_path), name, dict(N=N, K=K, mesh=mesh, dx=dx, dt=0.02 * dx * dx, eps=4.0 * dx, **kw),
                        seeds=seeds)
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    return p, phi, mu, o


@pytest.mark.parametrize("name", sorted(CASES))
def test_smooth_and_steps(tmp_path, name):
    p, phi, mu, o = _start(tmp_path, name)
    sim = gp.Simulation(p, phi, mu)
    try:
        for what, n in (("smooth", 9), ("step", 1), ("step", 12)):
            getattr(o, what)(n)
            sim.smooth(n) if what == "smooth" else sim.step(n, stats=False)
            for a, b in zip(sim.get(), o.get()):
                assert np.isfinite(b).all()
                assert bits_equal(a, b), "%s %d: %s" % (what, n, mismatch_report(a, b))
    finally:
        sim.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_noalloc(tmp_path, name):
    import torch
    p, phi, mu, o = _start(tmp_path, name)
    o.smooth(3)
    phi, mu = o.get()
    L = _abi.lib()
    src = [torch.from_numpy(np.array(a)).cuda() for a in (phi, mu)]
    dst = [torch.full_like(a, float("nan")) for a in src]
    stream = torch.cuda.current_stream()
    for n in range(2):
        o.step(1)
        rc = L.gp_step_noalloc(ctypes.byref(p), src[0].data_ptr(), src[1].data_ptr(), dst[0].data_ptr(),
                               dst[1].data_ptr(), ctypes.c_void_p(stream.cuda_stream))
        assert rc == 0, L.gp_last_error(None)
        stream.synchronize()
        for a, b in zip(dst, o.get()):
            assert np.isfinite(b).all()
            assert bits_equal(a.cpu().numpy(), b), "call %d: %s" % (n, mismatch_report(a.cpu().numpy(), b))
        src, dst = dst, src


@pytest.mark.parametrize("name", ["above", "below", "iso", "whole"])
def test_smooth_by_tile_kinds_in_a_batch(tmp_path, name):
    """Four simulations take the sweep by tile kinds at any size (one of these
    grids alone takes one launch over every cell)."""
    p, phi, mu, o = _start(tmp_path, name)
    b = gp.Batch([p] * 4, [(phi, mu)] * 4, precision=gp.GP_FP64)
    o.smooth(9)
    o.step(1)
    b.smooth(9)
    b.step(1, stats=False)
    for s in range(4):
        for x, y in zip(b.get(s), o.get()):
            assert bits_equal(x, y), mismatch_report(x, y)
    b.close()


@pytest.mark.parametrize("tiles", [2666, 2667])
def test_smooth_on_both_sides_of_the_line(tmp_path, tiles):
    """tiles * (phases + solutes) just below and above 8000."""
    mesh = (8, 32 * tiles)
    ip, fp = write_case(str(tmp_path), "line", dict(N=2, K=1, mesh=mesh, dab=0.03, d_solid=0.0),
                        seeds=[(0, 3, 40 + 9000 * i, 6.0) for i in range(8)])
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    o = Oracle(p, recip_div=1)
    o.set(phi, mu)
    with gp.Simulation(p, phi, mu) as sim:
        sim.smooth(3)
        sim.step(1, stats=False)
        o.smooth(3)
        o.step(1)
        for a, b in zip(sim.get(), o.get()):
            assert bits_equal(a, b), mismatch_report(a, b)
