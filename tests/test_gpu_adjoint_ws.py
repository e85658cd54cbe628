"""gp_adjoint_ws: the adjoint in a block of the caller's, against gp_adjoint.

The block starts as NaN bytes, so anything read before it is written shows.
The reverse sweep accumulates with atomics: with at most 9 * 12 = 108 additions
into a value over the steps, two orders differ by 108 * 2**-53 = 1.2e-14 of the
largest partial sums; the bound leaves a factor of about 1e3 for the steps'
amplification.  A parameter's gradient is one sum over cells and steps
(3e4 terms, 3.4e-12 of its terms' size) that cancels in part.
"""
import ctypes

import numpy as np
import pytest

import eshwar_dipan_b200 as gp
from eshwar_dipan_b200 import _abi
from gp_cases import write_case

pytestmark = pytest.mark.gpu


def _call(sim, phi_bar, mu_bar, snapshots, ws):
    req, out = _abi.AdjReq(), _abi.AdjOut()
    req.nsteps, req.snapshots = 12, snapshots
    req.phi_bar, req.mu_bar = phi_bar.ctypes.data, mu_bar.ctypes.data
    g_phi, g_mu = np.zeros_like(phi_bar), np.zeros_like(mu_bar)
    out.phi0_bar, out.mu0_bar = g_phi.ctypes.data, g_mu.ctypes.data
    L = _abi.lib()
    n = L.gp_adjoint_ws_bytes(sim.handle, ctypes.byref(req))
    assert 0 < n <= 2 << 30
    if ws is None:
        rc = L.gp_adjoint(sim.handle, ctypes.byref(req), ctypes.byref(out))
    else:
        import torch
        cut, off = ws
        t = torch.full((n + 256,), 255, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        rc = L.gp_adjoint_ws(sim.handle, ctypes.byref(req), ctypes.byref(out), t.data_ptr() + off, n - cut)
        assert cut or off or bool((t[:n] != 255).any())   # the block was used
    assert rc == 0, L.gp_last_error(sim.handle)
    return g_phi, g_mu, np.array([out.d_tau, out.d_dab, out.d_epsilon, out.d_gamma]), out.snapshots


@pytest.mark.parametrize("snapshots,ws", [(0, (0, 0)), (3, (0, 0)), (0, (512, 0)), (0, (0, 8))])
def test_same_gradients(tmp_path, snapshots, ws):
    ip, fp = write_case(str(tmp_path), "a", dict(N=2, K=1, mesh=(37, 70), dab=0.03, d_solid=0.0),
                        seeds=[(0, 18, 35, 8.0)])
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    rng = np.random.default_rng(3)
    pb, mb = rng.standard_normal(phi.shape), rng.standard_normal(mu.shape)
    r = []
    for w in (None, ws):
        with gp.Simulation(p, phi, mu) as s:
            s.smooth(5)
            r.append(_call(s, pb, mb, snapshots, w) + s.get())
    a, b = r
    assert a[3] == b[3]
    for i in (4, 5):   # the final state: no atomics
        assert np.array_equal(a[i], b[i])
    for i in (0, 1):
        assert np.isfinite(a[i]).all() and np.abs(a[i]).max() > 0
        np.testing.assert_allclose(b[i], a[i], rtol=0, atol=1e-11 * np.abs(a[i]).max())
    np.testing.assert_allclose(b[2], a[2], rtol=1e-8)
