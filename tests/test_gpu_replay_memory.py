"""gp_adjoint_replay gives back the device memory that it takes for a call."""
import pytest

import eshwar_dipan_b200 as gp
from gp_cases import write_case

pytestmark = pytest.mark.gpu


def test_replay_frees_its_buffers(tmp_path):
    import torch
    mesh, calls = (512, 512), 24
    ip, fp = write_case(str(tmp_path), "r", dict(N=2, K=1, mesh=mesh, dab=0.03, d_solid=0.0),
                        seeds=[(0, 250, 260, 20.0)])
    p = gp.load_params(ip)
    phi, mu = gp.fill(p, fp)
    with gp.Simulation(p, phi, mu) as s:
        assert s.adjoint_replay(3)[1] == 0   # modules and graphs are loaded
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for _ in range(calls):
            s.adjoint_replay(3)
        lost = before - torch.cuda.mem_get_info()[0]
    # a call takes two states (three planes each) and two planes of delta-phi
    taken = 8 * 8 * mesh[0] * mesh[1]
    assert lost < taken, "%d bytes gone after %d calls that take %d each" % (lost, calls, taken)
