"""Tensor maps of the step kernels' boxes: a map in global memory needs an
acquire fence before a block's first use of it (the copy unit may hold what lay
at its address before); a batch of one gets its maps as a kernel parameter, one of
as many tiles as its simulations squared fences them all at the start of a block, any
other where a thread moves to a simulation.

The GPU tests put different maps at the same addresses one after the other.
States are compared bit for bit.  Gradients: as in test_gpu_adjoint_ws.py.
"""
import ctypes
import os
import re

import numpy as np
import pytest

import eshwar_dipan_b200 as gp
from eshwar_dipan_b200 import _abi
from gp_cases import random_seeds, write_case
from oracle_py import Oracle, bits_equal, mismatch_report

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eshwar_dipan_b200", "csrc")
MESHES = [(40, 160), (104, 64), (64, 224)]


def test_boxes_take_their_map_from_box_map():
    with open(os.path.join(CSRC, "gp_fused.cuh")) as f:
        src = re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)
    calls = re.findall(r"(?<!void )tma_load_3d\(smem_addr\([^()]*\),\s*(\w+)", src)
    assert calls == ["box_map", "box_map"]
    def body(name):
        t = src[src.index(name):]
        return t[:t.index("\n}\n")]

    assert "fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" in body("void box_fence(")
    # the kernel parameter's map, else a fence ahead of the wait or here
    assert re.findall(r"return ([^;]*);", body("*box_map(")) == ["&maps.m[kind]", "m"]
    assert re.search(r"if \(!maps.ahead && m != ready\) \{\s*box_fence\(m\);", body("*box_map("))
    ahead = body("void box_begin(")
    assert "if (!SOLO && maps.ahead) {" in ahead
    assert ahead.index("box_fence(") < ahead.index("__syncthreads();") < ahead.index("pdl_wait();")
    for kernel, kinds in (("kf_bulk", "1u << MAP_MU"), ("kf_general", "1u << MAP_ALL"),
                          ("kf_step", "1u << MAP_MU | 1u << MAP_ALL")):
        k = src[src.index(" %s(\n" % kernel):]
        assert re.search(r"\{\s*box_begin<([^,]*),", k).group(1) == kinds
    params = re.findall(r"([\w ]*)BoxMaps maps,", src)
    assert len(params) == 3 and all(q.strip() == "const __grid_constant__" for q in params)


def _case(tmp_path, mesh, N=2, K=1, **kw):
    seeds = random_seeds(3, mesh, 5.0, 9.0, N - 1, mesh[0])
    ip, fp = write_case(str(tmp_path), "m%d_%d" % mesh, dict(N=N, K=K, mesh=mesh, dab=0.03, d_solid=0.0, **kw),
                        seeds=seeds)
    p = gp.load_params(ip)
    return (p,) + gp.fill(p, fp)


@pytest.mark.gpu
def test_adjoint_in_one_block_on_several_grids(tmp_path):
    import torch
    L = _abi.lib()
    runs = []
    for mesh in MESHES[:2]:
        p, phi, mu = _case(tmp_path, mesh)
        sim = gp.Simulation(p, phi, mu)
        sim.smooth(5)
        rng = np.random.default_rng(mesh[0])
        runs.append((sim, sim.get(), rng.standard_normal(phi.shape), rng.standard_normal(mu.shape)))

    def call(run, block):
        sim, start, pb, mb = run
        sim.set(*start)
        req, out = _abi.AdjReq(), _abi.AdjOut()
        req.nsteps, req.phi_bar, req.mu_bar = 12, pb.ctypes.data, mb.ctypes.data
        g_phi, g_mu = np.zeros_like(pb), np.zeros_like(mb)
        out.phi0_bar, out.mu0_bar = g_phi.ctypes.data, g_mu.ctypes.data
        n = L.gp_adjoint_ws_bytes(sim.handle, ctypes.byref(req))
        if block is None:
            block = torch.empty(n, dtype=torch.uint8, device="cuda")
        assert 0 < n <= block.numel()
        torch.cuda.synchronize()
        rc = L.gp_adjoint_ws(sim.handle, ctypes.byref(req), ctypes.byref(out), block.data_ptr(), block.numel())
        assert rc == 0, L.gp_last_error(sim.handle)
        return sim.get() + (g_phi, g_mu)

    try:
        alone = [call(r, None) for r in runs]
        fixed = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
        for k in range(4):
            got, ref = call(runs[k % 2], fixed), alone[k % 2]
            for a, b in zip(got[:2], ref[:2]):
                assert bits_equal(a, b), "call %d: %s" % (k, mismatch_report(a, b))
            for a, b in zip(got[2:], ref[2:]):
                assert np.abs(b).max() > 0
                np.testing.assert_allclose(a, b, rtol=0, atol=1e-11 * np.abs(b).max())
    finally:
        for r in runs:
            r[0].close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec,times", [("FP64", 1), ("FP32", 1), ("FP64", 12), ("FP32", 12), ("FP64", 64),
                                        ("FP32", 64)])
def test_batches_one_after_the_other(tmp_path, prec, times):
    """Batches of two grids (`times` of each), each in the memory that the one before gave back, and
    alone: a batch's simulations step as they do alone (maps from global memory
    and from the parameter), in FP64 as the oracle does."""
    precision = getattr(gp, "GP_" + prec)
    ref = {}
    for mesh in MESHES:
        p, phi, mu = _case(tmp_path, mesh, N=3, K=2)
        with gp.Simulation(p, phi, mu, precision=precision) as s:
            s.step(7, stats=False)
            ref[mesh] = (p, phi, mu) + s.get()
        if prec == "FP64":
            o = Oracle(p, recip_div=1)
            o.set(phi, mu)
            o.step(7)
            for a, b in zip(ref[mesh][3:], o.get()):
                assert bits_equal(a, b), mismatch_report(a, b)
    for pair in [(0, 1), (1, 2), (2, 0), (1, 0)]:
        ms = [ref[MESHES[i]] for i in pair] * times
        b = gp.Batch([m[0] for m in ms], [(m[1], m[2]) for m in ms], precision=precision)
        b.step(7, stats=False)
        for i, m in enumerate(ms):
            for x, y in zip(b.get(i), m[3:]):
                assert np.array_equal(x, y), "%s: %s" % (pair, mismatch_report(x, y))
        b.close()
