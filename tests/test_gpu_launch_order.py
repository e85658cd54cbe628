"""Steps inside a graph are launched ahead of their predecessor's end below 4096 tiles
and in order from there; single steps always ahead.  All give the same bits: 4095
and 4096 tiles, graphs against single steps, one simulation and two."""
import pytest

import eshwar_dipan_b200 as gp
from gp_cases import random_seeds, write_case
from oracle_py import bits_equal, mismatch_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(8 * 63, 32 * 65), (8 * 64, 32 * 64)])
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
def test_graphs_against_single_steps(tmp_path, mesh, prec):
    ip, fp = write_case(str(tmp_path), "l", dict(N=3, K=2, mesh=mesh, dab=0.02, d_solid=0.0),
                        seeds=random_seeds(20, mesh, 8.0, 30.0, 2, 4))
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    precision = getattr(gp, "GP_" + prec)
    with gp.Simulation(p, phi, mu, precision=precision) as s:
        s.smooth(9)
        phi, mu = s.get()
    with gp.Simulation(p, phi, mu, precision=precision) as s:
        for _ in range(41):
            s.step(1, stats=False)
        ref = s.get()
    with gp.Simulation(p, phi, mu, precision=precision) as s:
        s.step(41, stats=False)
        for a, b in zip(s.get(), ref):
            assert bits_equal(a, b), mismatch_report(a, b)
    b = gp.Batch([p] * 2, [(phi, mu)] * 2, precision=precision)
    b.step(41, stats=False)
    for x, y in zip(b.get(1), ref):
        assert bits_equal(x, y), mismatch_report(x, y)
    b.close()
