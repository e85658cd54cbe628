"""The first step of a context, on which nearly every cell's mu is a new extreme of
the progress record, takes about as long as the next one: extremes are reduced over
a warp before they go to the simulation's few addresses.  (With an atomic per cell
it took 4.3 times as long on this grid; the bound of 2 leaves the reduction twice
its time.)  The extremes themselves: test_gpu_parity.py, test_gpu_unusual_values.py.
"""
import pytest

import eshwar_dipan_b200 as gp
from gp_cases import random_seeds, write_case

pytestmark = pytest.mark.gpu


def test_first_step_costs_a_step(tmp_path):
    mesh = (2048, 2048)
    ip, fp = write_case(str(tmp_path), "first", dict(N=3, K=2, mesh=mesh, dab=0.02, d_solid=0.0),
                        seeds=random_seeds(64, mesh, 12.0, 40.0, 2, 3))
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    ms = [[], []]
    for _ in range(4):   # (the first context loads the kernels)
        with gp.Simulation(p, phi, mu) as s:
            s.smooth(9)
            for m in ms:
                t = s.kernel_times(1)
                m.append(t["step_ms"] + t["bulk_ms"] + t["iface_ms"])
    assert min(ms[0]) < 2.0 * min(ms[1]), ms
