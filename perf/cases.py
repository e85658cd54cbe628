"""The work a user of this package has it do, as measurable cases.

A case is one call or one short sequence of calls through the public entry
points, from a start state to the fields (and gradients) it produces.  Kinds:

  step      a simulation on the GPU restarted from a state held in CUDA tensors,
            stepped, its statistics and new state read back (the inner loop of
            an optimisation or a data-generation run; gp_set_dev, gp_step,
            gp_get_dev)
  noalloc   one step on the caller's own device buffers (gp_step_noalloc)
  smooth    the start-up sweeps of a fresh state
  program   a whole directional-solidification run from host fields: create,
            smooth, step with the moving frame, read fields and temperature
  fp32      the FP32 storage form over host fields
  ensemble  a batch of independent binary simulations of different sizes
  rollout   the differentiable time loop: forward and backward through torch

Physics and seed layouts follow eshwar_dipan_b200.workloads (the benchmark
configurations); start states are grown seeds with the obstacle potential's
diffuse profile and a solute layer around each, made from the seed alone.
"""
import ctypes
import math
import tempfile

import numpy as np
import torch

import eshwar_dipan_b200 as gp
from eshwar_dipan_b200 import _abi
from eshwar_dipan_b200.integrator import GPRollout
from eshwar_dipan_b200.workloads import write_case

_F64 = torch.float64


def listed():
    return [
        # the smallest call: a single step in an application that owns its buffers
        dict(name="noalloc_200x152", kind="noalloc", n=2, k=1, mx=200, my=152, aniso=True, dab=0.03, bc=1, seeds=2,
             rlo=8.0, rhi=30.0, steps=1),
        # a short advance of a small grid (the first benchmark configuration): launches and gaps
        dict(name="binary_256_10steps", kind="step", n=2, k=1, mx=256, my=256, aniso=False, dab=0.0, bc=1, seeds=1,
             rlo=40.0, rhi=50.0, steps=10),
        # an ordinary dendrite run of one simulation, sides as in the ensemble of the benchmark
        dict(name="dendrite_1024", kind="step", n=2, k=1, mx=1024, my=1024, aniso=True, dab=0.04, bc=1, seeds=8,
             rlo=12.0, rhi=60.0, steps=200),
        # the 2048^2 ternary three-phase benchmark configuration
        dict(name="ternary_2048", kind="step", n=3, k=2, mx=2048, my=2048, aniso=True, dab=0.02, bc=3, seeds=64,
             rlo=6.0, rhi=40.0, steps=100),
        # the largest: the 4096^2 headline configuration
        dict(name="ternary_4096", kind="step", n=3, k=2, mx=4096, my=4096, aniso=False, dab=0.0, bc=1, seeds=256,
             rlo=6.0, rhi=40.0, steps=50),
        # ragged sides, a spacing that is no power of two, coupled diffusion, a rotated pair
        dict(name="ragged_1501x1111", kind="step", n=3, k=2, mx=1501, my=1111, aniso=True, dab=0.02, bc=1, seeds=24,
             rlo=6.0, rhi=40.0, steps=60, dx=1.5, dt=0.04, a_off=0.25, rot=45.0),
        # the widest system the kernels take: four phases, two solutes
        dict(name="four_phase_768", kind="step", n=4, k=2, mx=768, my=768, aniso=False, dab=0.0, bc=3, seeds=12,
             rlo=6.0, rhi=40.0, steps=60),
        # start-up of a large grid: the NSMOOTH-1 sweeps
        dict(name="smooth_2048", kind="smooth", n=3, k=2, mx=2048, my=2048, aniso=True, dab=0.02, bc=3, seeds=64,
             rlo=4.0, rhi=12.0, steps=9),
        # a whole run from host fields, non-isothermal with the moving frame
        dict(name="dirsolid_256x640", kind="program", n=2, k=1, mx=256, my=640, aniso=True, dab=0.03, bc=3, seeds=8,
             rlo=3.0, rhi=8.0, steps=150),
        # the FP32 form between two outputs (SAVET = 1000)
        dict(name="fp32_1536", kind="fp32", n=3, k=2, mx=1536, my=1536, aniso=False, dab=0.0, bc=1, seeds=36,
             rlo=6.0, rhi=40.0, steps=1000),
        # a parameter study: 24 simulations, sides 128..1024, in the FP32 form
        dict(name="ensemble_24", kind="ensemble", n=2, k=1, sims=24, lo=128, hi=1024, steps=500),
        # gradients of a dendrite run (the adjoint benchmark's grid)
        dict(name="rollout_grad_512", kind="rollout", n=2, k=1, mx=512, my=512, aniso=True, dab=0.04, bc=1, seeds=1,
             rlo=30.0, rhi=60.0, steps=100, every=0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["noalloc", "step", "step", "step", "smooth", "program", "fp32", "ensemble", "rollout"])
    if kind == "ensemble":
        return dict(kind=kind, n=2, k=1, sims=rng.randint(2, 24), lo=128, hi=rng.choice([256, 512, 1024]),
                    steps=rng.randint(100, 500))
    if kind == "rollout":
        mx, my = int(_log(rng, 64, 512)), int(_log(rng, 64, 512))
        return dict(kind=kind, n=2, k=1, mx=mx, my=my, aniso=rng.random() < 0.7, dab=0.04, bc=rng.choice([1, 3]),
                    seeds=rng.randint(1, 3), rlo=8.0, rhi=8.0 + min(mx, my) / 9.0, steps=rng.randint(10, 100),
                    every=rng.choice([0, 0, 10]))
    if kind == "program":
        return dict(kind=kind, n=2, k=1, mx=int(_log(rng, 64, 512)), my=int(_log(rng, 192, 640)), aniso=True,
                    dab=0.03, bc=3, seeds=rng.randint(1, 10), rlo=3.0, rhi=8.0, steps=rng.randint(50, 200))
    n, k = rng.choice([(2, 1), (2, 1), (3, 2), (3, 2), (3, 1), (4, 2)])
    top = {"noalloc": 600, "step": 3000 if n < 4 else 900, "smooth": 2048, "fp32": 1600}[kind]
    mx, my = int(_log(rng, 100, top)), int(_log(rng, 100, top))
    aniso = rng.random() < 0.6
    c = dict(kind=kind, n=n, k=k, mx=mx, my=my, aniso=aniso, dab=0.03 if aniso else 0.0, bc=rng.choice([1, 3]),
             seeds=max(1, int(mx * my * _log(rng, 4e-6, 3e-5))), rlo=6.0, rhi=6.0 + min(34.0, min(mx, my) / 6.0),
             steps={"noalloc": 1, "step": int(_log(rng, 5, 200)), "smooth": rng.randint(3, 9),
                    "fp32": rng.randint(200, 1000)}[kind])
    if rng.random() < 0.3:
        c.update(dx=1.5, dt=0.04)
    if k == 2 and rng.random() < 0.4:
        c.update(a_off=0.25)
    return c


# ---- inputs ------------------------------------------------------------------

def _members(case, seed):
    """the simulations of a case: one, or an ensemble's members (sides,
    composition, anisotropy strength and seeds of their own)"""
    if case["kind"] != "ensemble":
        return [dict(case)]
    r = np.random.RandomState(1000003)   # the ensemble's sides and physics belong to the case
    out = []
    for _ in range(case["sims"]):
        side = 32 * int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))) / 32.0))
        out.append(dict(kind="fp32", n=2, k=1, mx=side, my=side, aniso=True, dab=round(0.05 * r.uniform(), 6),
                        bc=1, seeds=1 + int(8 * r.uniform()), rlo=4.0, rhi=30.0,
                        c0=round(0.40 + 0.08 * r.uniform(), 6), T=1.0))
    return out


def _input(m):
    """input deck keywords of one simulation (workloads.input_text)"""
    n, k = m["n"], m["k"]
    bc = (1, 1, 1, 1) if m["bc"] == 1 else (3, 3, 3, 3)
    kw = dict(N=n, K=k, mesh=(m["mx"], m["my"]), dx=m.get("dx", 1.0), dt=m.get("dt", 0.02), eps=4.0, aniso=m["aniso"],
              dab=m["dab"], bc_phi=bc, d_liquid=[1.0, 0.5][:k], d_solid=0.0, A_off=m.get("a_off", 0.0),
              T=m.get("T", 0.97), tau_ab=0.28, tau=1.31, gamma=1.0, gamma_abc=10.0, Teq=1.0)
    if "rot" in m:
        kw["rot"] = {(n - 2, n - 1): m["rot"]}
    if "c0" in m:
        kw["liquid_c"] = [m["c0"]]
    if m["kind"] == "rollout":
        kw["T"], kw["liquid_c"] = 1.0, [0.42]
    if m["kind"] == "program":
        kw.update(bc_phi=(3, 3, 1, 1), T=1.0, tempgrady=(0.97, 0.06, 200.0, 40.0, 0.5), shift=True, shiftj=40,
                  liquid_c=[0.45])
    return kw


def _load(m):
    with tempfile.TemporaryDirectory() as d:
        ip, _ = write_case(d, "case", _input(m))
        return gp.load_params(ip)


def _fields(m, seed, grow=0.0):
    """start fields phi [n][mx][my], mu [k][mx][my] on the GPU: seeds of random
    place, size and solid phase.  Sharp where the start-up sweeps follow (smooth,
    program), else with the obstacle profile (width pi^2 eps / 4) and a layer of
    rejected solute that decays into the liquid."""
    r = np.random.RandomState(seed % (1 << 31))
    n, k, mx, my = m["n"], m["k"], m["mx"], m["my"]
    dx = m.get("dx", 1.0)
    model = Model(_input(m))
    half = math.pi ** 2 * 4.0 / 8.0 / dx     # half width of the diffuse interface in cells
    dist = torch.full((mx, my), 1e9, dtype=_F64, device="cuda")
    lab = torch.zeros((mx, my), dtype=torch.int64, device="cuda")
    X = torch.arange(mx, dtype=_F64, device="cuda")[:, None]
    Y = torch.arange(my, dtype=_F64, device="cuda")[None, :]
    for _ in range(m["seeds"]):
        R = r.uniform(m["rlo"], m["rhi"]) + grow
        cx, cy, ph = r.uniform(0, mx), r.uniform(0, my), int(r.randint(n - 1))
        if m["kind"] == "program":           # bumps on a flat front
            cy, ph = 56.0, 0
        reach = R + 60.0
        a0, a1 = max(0, int(cx - reach)), min(mx, int(cx + reach) + 1)
        b0, b1 = max(0, int(cy - reach)), min(my, int(cy + reach) + 1)
        d = torch.sqrt((X[a0:a1] - cx) ** 2 + (Y[:, b0:b1] - cy) ** 2) - R
        sub, sl = dist[a0:a1, b0:b1], lab[a0:a1, b0:b1]
        near = d < sub
        sl.copy_(torch.where(near, torch.full_like(sl, ph), sl))
        sub.copy_(torch.where(near, d, sub))
    if m["kind"] == "program":
        dist = torch.minimum(dist, (Y - 56.0).expand(mx, my))
    if m["kind"] in ("program", "smooth"):
        s = (dist <= 0.0).to(_F64)
    else:
        s = 0.5 - 0.5 * torch.sin((dist / half).clamp(-1.0, 1.0) * (math.pi / 2.0))
        s = torch.where(dist >= half, torch.zeros_like(s), torch.where(dist <= -half, torch.ones_like(s), s))
    phi = torch.stack([torch.where(lab == a, s, torch.zeros_like(s)) for a in range(n - 1)] + [1.0 - s])
    far, eq = model.mu_far(), model.mu_eq()
    ph0 = r.uniform(0, 2 * math.pi, size=2)
    wave = 1e-3 * torch.sin(X * (2 * math.pi / 97.0) + ph0[0]) * torch.sin(Y * (2 * math.pi / 131.0) + ph0[1])
    layer = torch.exp(-dist.clamp(min=0.0) / 12.0)
    if m["kind"] in ("program", "smooth"):
        layer = s
    mu = torch.stack([far[i] + (eq[i] - far[i]) * 0.9 * layer + wave for i in range(k)])
    return phi.contiguous(), mu.contiguous()


def prepare(case, seed):
    if case["kind"] == "ensemble":
        ms = _members(case, seed)
        fields = [tuple(f.cpu().numpy() for f in _fields(m, seed * 64 + i)) for i, m in enumerate(ms)]
        return dict(case=case, fields=fields, batch=gp.Batch([_load(m) for m in ms], fields, precision=gp.GP_FP32))
    p = _load(case)
    phi, mu = _fields(case, seed)
    s = dict(case=case, p=p)
    if case["kind"] in ("step", "smooth"):
        s.update(phi=phi, mu=mu, sim=gp.Simulation.from_tensors(p, phi, mu))
    elif case["kind"] == "noalloc":
        s.update(phi=phi, mu=mu, phi_out=torch.empty_like(phi), mu_out=torch.empty_like(mu))
    elif case["kind"] == "rollout":
        s.update(phi=phi.requires_grad_(), mu=mu.requires_grad_(), target=_fields(case, seed, grow=4.0)[0],
                 roll=GPRollout(p, case["steps"], checkpoint_every=case["every"]))
        s["theta"] = s["roll"].theta0().requires_grad_()
    else:
        s.update(phi=phi.cpu().numpy(), mu=mu.cpu().numpy())
        if case["kind"] == "fp32":
            s["sim"] = gp.Simulation(p, s["phi"], s["mu"], precision=gp.GP_FP32)
    return s


# ---- one pass ----------------------------------------------------------------

def run(s):
    case = s["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "step":
        s["sim"].set_tensors(s["phi"], s["mu"])
        st = s["sim"].step(steps)
        phi, mu = s["sim"].get_tensors()
        return dict(phi=phi, mu=mu, stats=st)
    if kind == "smooth":
        s["sim"].set_tensors(s["phi"], s["mu"])
        s["sim"].smooth(steps)
        phi, mu = s["sim"].get_tensors()
        return dict(phi=phi, mu=mu)
    if kind == "noalloc":
        rc = _abi.lib().gp_step_noalloc(ctypes.byref(s["p"]), s["phi"].data_ptr(), s["mu"].data_ptr(),
                                        s["phi_out"].data_ptr(), s["mu_out"].data_ptr(),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _abi.check(rc)
        return dict(phi=s["phi_out"], mu=s["mu_out"])
    if kind == "program":
        with gp.Simulation(s["p"], s["phi"], s["mu"]) as sim:
            sim.smooth(s["p"].nsmooth - 1)
            st = sim.step(steps)
            phi, mu = sim.get()
            return dict(phi=phi, mu=mu, T=sim.temperature(), stats=st)
    if kind == "fp32":
        s["sim"].set(s["phi"], s["mu"])
        s["sim"].step(steps, stats=False)
        phi, mu = s["sim"].get()          # float values in double arrays: kept as float
        return dict(phi=torch.from_numpy(phi).to(torch.float32), mu=torch.from_numpy(mu).to(torch.float32))
    if kind == "ensemble":
        b = s["batch"]
        for i, (phi, mu) in enumerate(s["fields"]):
            b.set(i, phi, mu)
        b.step(steps, stats=False)
        out = []
        for i in range(b.n):
            phi, mu = b.get(i)
            out.append((torch.from_numpy(phi).to(torch.float32), torch.from_numpy(mu).to(torch.float32)))
        return out
    phi, mu = s["roll"](s["phi"], s["mu"], s["theta"])
    loss = 0.5 * ((phi - s["target"]) ** 2).sum()
    g = torch.autograd.grad(loss, (s["phi"], s["mu"], s["theta"]))
    return dict(phi=phi.detach(), mu=mu.detach(), loss=loss.detach(), g_phi=g[0], g_mu=g[1], g_theta=g[2])


def work(case):
    """Bytes and operations of one pass that no implementation of these steps
    avoids: the inputs read and the outputs written once, and per step one read
    and one write of mu (phi moves at interfaces only); the operations of the
    diffusion of mu, about 20 per cell and solute, and per sweep the phase-field
    terms."""
    cells, nk = 0, case["n"] + case["k"]
    for m in _members(case, 0):
        cells += m["mx"] * m["my"]
    steps, kind = case["steps"], case["kind"]
    s = 4 if kind in ("fp32", "ensemble") else 8
    if kind == "noalloc":
        return dict(bytes=2.0 * nk * 8 * cells, flops=20.0 * case["k"] * cells)
    if kind == "smooth":
        return dict(bytes=2.0 * nk * 8 * cells * steps, flops=(20.0 * case["k"] + 60.0 * case["n"]) * cells * steps)
    b = 2.0 * case["k"] * s * cells * steps + 2.0 * nk * 8 * cells
    f = 20.0 * case["k"] * cells * steps
    if kind == "rollout":                    # the tape is read back, the adjoint moves once a step
        b, f = 3.0 * b, 4.0 * f
    return dict(bytes=b, flops=f)


# ---- the same values in plain float64 torch ---------------------------------

class Model:
    """Constants and one time step of the grand-potential model in plain
    float64 torch operations, from the input deck's numbers."""

    def __init__(self, kw):
        self.kw = kw
        N, K = kw["N"], kw["K"]
        self.N, self.K, self.L = N, K, N - 1
        self.mx, self.my = kw["mesh"]
        self.dx = self.dy = kw["dx"]
        self.dt, self.eps, self.tau = kw["dt"], kw["eps"], kw["tau"]
        self.Teq, self.T = kw["Teq"], kw["T"]
        off = kw["A_off"]
        self.A = [[[1.0 if i == j else off for j in range(K)] for i in range(K)] for _ in range(N)]
        self.cmu = [np.linalg.inv(np.array([[2.0 * a[i][j] if i == j else a[i][j] for j in range(K)]
                                            for i in range(K)])).tolist() for a in self.A]
        cl = [0.5] if K == 1 else [0.33] * K
        self.c_far = kw.get("liquid_c") or ([0.45] if K == 1 else [0.3] * K)
        cs, sl = [], []
        for a in range(N - 1):
            b = [0.2 if a % 2 == 0 else 0.8] if K == 1 else [0.7 if a == i else 0.15 for i in range(K)]
            cs.append(b)
            sl.append([0.45 if a % 2 == 0 else -0.45] + [0.1] * (K - 1))
        self.cl, self.cs = cl, cs
        self.DT = [sum(sl[a][i] * (cl[i] - cs[a][i]) for i in range(K)) for a in range(N - 1)]
        self.Beq, _ = self._BC(self.Teq)
        self.dB = [[0.0] * K for _ in range(N)]
        for a in range(N - 1):
            q = [(cl[i] - cs[a][i]) / self.DT[a] for i in range(K)]
            for i in range(K):
                self.dB[a][i] = sum((2.0 if j == i else 1.0) * (self.A[self.L][i][j] - self.A[a][i][j]) * q[j]
                                    for j in range(K))
        D = [[[(kw["d_liquid"][i] if a == self.L else kw["d_solid"]) if i == j else 0.0 for j in range(K)]
              for i in range(K)] for a in range(N)]
        self.DC = [(np.array(D[a]) @ np.array(self.cmu[a])).tolist() for a in range(N)]
        self.atf = [[1.0 - D[a][i][i] / D[self.L][i][i] for i in range(K)] for a in range(N)]
        self.gamma, self.tau_ab, self.dab = {}, {}, {}
        self.R, self.rotated = {}, False
        for a in range(N):
            for b in range(N):
                if a == b:
                    continue
                p = (min(a, b), max(a, b))
                self.gamma[a, b], self.tau_ab[a, b], self.dab[a, b] = kw["gamma"], kw["tau_ab"], kw["dab"]
                th = kw.get("rot", {}).get(p, 0.0) * math.pi / 180.0
                self.rotated |= th != 0.0
                self.R[a, b] = [[math.cos(th), -math.sin(th)], [math.sin(th), math.cos(th)]]
        bx, by = kw["bc_phi"][0], kw["bc_phi"][2]
        dev = "cuda"
        self.ix = {w: torch.tensor(_copy_rows(self.mx, bx, w), device=dev) for w in (1, 2)}
        self.iy = {w: torch.tensor(_copy_rows(self.my, by, w), device=dev) for w in (1, 2)}
        self.by = by

    def _cls(self, a, T):
        q = [(self.cl[i] - self.cs[a][i]) * (self.Teq - T) / self.DT[a] for i in range(self.K)]
        return [self.cl[i] - q[i] for i in range(self.K)], [self.cs[a][i] - q[i] for i in range(self.K)]

    def _BC(self, T):
        B, C = [], []
        for a in range(self.N):
            if a == self.L:
                B.append([0.0] * self.K)
                C.append(0.0)
                continue
            l, s = self._cls(a, T)
            AL, AS = self.A[self.L], self.A[a]
            B.append([sum((2.0 if j == i else 1.0) * (AL[j][i] * l[j] - AS[j][i] * s[j]) for j in range(self.K))
                      for i in range(self.K)])
            C.append(sum(AS[i][j] * s[i] * s[j] - AL[i][j] * l[i] * l[j] for i in range(self.K)
                         for j in range(i, self.K)))
        return B, C

    def _E(self, T):
        return [[self.Beq[a][i] + self.dB[a][i] * (T - self.Teq) for i in range(self.K)] for a in range(self.N)]

    def _Mu(self, E, c, a):
        return [sum((2.0 if i == j else 1.0) * self.A[a][i][j] * c[j] for j in range(self.K)) + E[a][i]
                for i in range(self.K)]

    def mu_far(self):
        return self._Mu(self._E(self.T), self.c_far, self.L)

    def mu_eq(self):
        return self._Mu(self._E(self.T), self.cl, self.L)

    # -- pieces
    def c_of(self, E, m, a):
        return [sum(self.cmu[a][i][j] * (m[j] - E[a][j]) for j in range(self.K)) for i in range(self.K)]

    def h(self, ph, a):
        o = [ph[b] for b in range(self.N) if b != a]
        s1 = sum((o[i] * o[j] for i in range(len(o)) for j in range(i + 1, len(o))), torch.zeros_like(ph[a]))
        return 3.0 * ph[a] * ph[a] - 2.0 * ph[a] * ph[a] * ph[a] + s1 * (2.0 * ph[a])

    def dh(self, ph, b, a):
        """d h_b / d phi_a"""
        if a == b:
            s = 6.0 * ph[a] * (1.0 - ph[a])
            o = [e for e in range(self.N) if e != b]
            for i, e in enumerate(o):
                for f in o[i + 1:]:
                    s = s + 2.0 * ph[e] * ph[f]
            return s
        return sum((2.0 * ph[e] for e in range(self.N) if e not in (a, b)), torch.zeros_like(ph[a])) * ph[b]

    def _rot(self, a, b, q0, q1, inverse=False):
        if not self.rotated:
            return q0, q1
        R = self.R[a, b]
        if inverse:
            return R[0][0] * q0 + R[1][0] * q1, R[0][1] * q0 + R[1][1] * q1
        return R[0][0] * q0 + R[0][1] * q1, R[1][0] * q0 + R[1][1] * q1

    def _an(self, a, b, q0, q1):
        """a_c, |q|^2 and dA/dq of the fourfold anisotropy"""
        d = self.dab[a, b]
        x2, y2 = q0 * q0, q1 * q1
        q2 = x2 + y2
        ok = q2 > 1.0e-15
        qs = torch.where(ok, q2, torch.ones_like(q2))
        q4 = x2 * x2 + y2 * y2
        ac = torch.where(ok, 1.0 - d * (3.0 - 4.0 * q4 / (qs * qs)), torch.ones_like(q2))
        z = torch.zeros_like(q2)
        d0 = torch.where(ok, 16.0 * d * (q0 * x2 / (qs * qs) - q0 * q4 / (qs * qs * qs)), z)
        d1 = torch.where(ok, 16.0 * d * (q1 * y2 / (qs * qs) - q1 * q4 / (qs * qs * qs)), z)
        return ac, q2, d0, d1

    def _face(self, a, b, s, g, c0, c1, xface):
        """divergence terms of the gradient energy on faces, of (a,b)'s phase a and phase b"""
        Pab = s[a] * g[b] - s[b] * g[a]
        if not self.kw["aniso"] or self.iso:
            return Pab * (-s[b]), (-Pab) * (-s[a])
        t = 0.5 * (s[a] * (c0[b] + c1[b]) - s[b] * (c0[a] + c1[a]))
        q0, q1 = self._rot(a, b, *((Pab, t) if xface else (t, Pab)))
        ac, q2, d0, d1 = self._an(a, b, q0, q1)
        r = self._rot(a, b, d0, d1, inverse=True)[0 if xface else 1]
        u = ac * ac * Pab + ac * q2 * r
        return u * (-s[b]), (-u) * (-s[a])

    def delta_phi(self, P, M, T, smooth):
        """delta-phi of the interior and a one-cell ring; P: phi with two ghost
        rows, M: mu with one"""
        N, dx, dy = self.N, self.dx, self.dy
        self.iso = smooth
        ph = [p[1:-1, 1:-1] for p in P]
        xf = [(p[1:] - p[:-1]) / dx for p in P]
        yf = [(p[:, 1:] - p[:, :-1]) / dy for p in P]
        act, gcx, gcy = [], [], []
        for a in range(N):
            f, b = xf[a][1:, 1:-1], xf[a][:-1, 1:-1]
            r, l = yf[a][1:-1, 1:], yf[a][1:-1, :-1]
            act.append(((f - b) / dx + (r - l) / dy).abs() > 0.0)
            gcx.append(0.5 * (f + b))
            gcy.append((P[a][1:-1, 2:] - P[a][1:-1, :-2]) / (2.0 * dy))
        sx = [0.5 * (p[1:, 1:-1] + p[:-1, 1:-1]) for p in P]
        sy = [0.5 * (p[1:-1, 1:] + p[1:-1, :-1]) for p in P]
        gx, gy = [f[:, 1:-1] for f in xf], [f[1:-1] for f in yf]
        cy = [(p[:, 2:] - p[:, :-2]) / (2.0 * dy) for p in P]
        cx = [0.5 * (f[1:] + f[:-1]) for f in xf]
        zero = torch.zeros_like(ph[0])
        dA, div = [zero] * N, [zero] * N
        for a in range(N):
            for b in range(a + 1, N):
                X = self._face(a, b, sx, gx, [c[:-1] for c in cy], [c[1:] for c in cy], True)
                Y = self._face(a, b, sy, gy, [c[:, :-1] for c in cx], [c[:, 1:] for c in cx], False)
                g = self.gamma[a, b]
                q0 = ph[a] * gcx[b] - ph[b] * gcx[a]
                q1 = ph[a] * gcy[b] - ph[b] * gcy[a]
                if self.kw["aniso"] and not smooth:
                    q0, q1 = self._rot(a, b, q0, q1)
                    ac, q2, d0, d1 = self._an(a, b, q0, q1)
                    e0, e1 = ac * ac * q0 + ac * q2 * d0, ac * ac * q1 + ac * q2 * d1
                else:
                    e0, e1 = q0, q1
                for me, other, sg, o in ((a, b, 1.0, 0), (b, a, -1.0, 1)):
                    w0, w1 = gcx[other], gcy[other]
                    if self.kw["aniso"] and not smooth:
                        w0, w1 = self._rot(a, b, w0, w1)
                    dA[me] = dA[me] + (2.0 * sg) * g * (e0 * w0 + e1 * w1)
                    div[me] = div[me] + 2.0 * g * ((X[o][1:] - X[o][:-1]) / dx + (Y[o][:, 1:] - Y[o][:, :-1]) / dy)
        if not smooth:
            E = self._E(T)
            B, C = self._BC(T)
            psi = []
            for b in range(N):
                c = self.c_of(E, M, b)
                f = sum(self.A[b][i][j] * c[i] * c[j] for i in range(self.K) for j in range(i, self.K))
                f = f + sum(B[b][i] * c[i] for i in range(self.K)) + C[b]
                psi.append(f - sum(M[i] * c[i] for i in range(self.K)))
        lam, sl, cnt = [], zero, zero
        for a in range(N):
            w = zero
            for b in range(N):
                if b != a:
                    v = self.gamma[a, b] * ph[b]
                    if not (smooth and self.kw["aniso"]):
                        v = torch.where(ph[a] * ph[b] >= 0.0, v, -v)
                    w = w + torch.where(act[b], v, zero)
            w = w * (16.0 / (math.pi * math.pi))
            for b in range(N):
                for c in range(b + 1, N):
                    if a not in (b, c):
                        v = self.kw["gamma_abc"] * ph[b] * ph[c]
                        if not (smooth and self.kw["aniso"]):
                            v = torch.where(ph[a] * ph[b] * ph[c] >= 0.0, v, -v)
                        w = w + torch.where(act[b] & act[c], v, zero)
            q = self.eps * (div[a] - dA[a]) - w / self.eps
            if not smooth:
                q = q - sum(psi[b] * self.dh(ph, b, a) for b in range(N))
            lam.append(q)
            sl = sl + torch.where(act[a], q, zero)
            cnt = cnt + act[a].to(_F64)
        sl = sl / cnt.clamp(min=1.0)
        s, s1 = zero, zero
        for a in range(N):
            for b in range(a + 1, N):
                s, s1 = s + self.tau_ab[a, b] * ph[a] * ph[b], s1 + ph[a] * ph[b]
        nz = s1 != 0.0
        tau = torch.where(nz, s / torch.where(nz, s1, torch.ones_like(s1)), torch.full_like(s1, self.tau))
        d = [torch.where(act[a], self.dt * (lam[a] - sl) / (tau * self.eps), zero) for a in range(N)]
        return (self._project_nw if smooth else self._project)(ph, act, d)

    def _project(self, ph, act, d):
        zero = torch.zeros_like(d[0])
        inside = [act[a] & (ph[a] + d[a] > 0.0) & (ph[a] + d[a] < 1.0) for a in range(self.N)]
        count = sum(i.to(_F64) for i in inside)
        total = sum(torch.where(inside[a], ph[a], zero) for a in range(self.N))
        D, d = zero, list(d)
        for a in range(self.N):
            v = torch.where(ph[a] + d[a] < 0.0, (ph[a] + d[a]).abs(), zero)
            d[a], D = d[a] + v, D + v
        ok = total.abs() > 0.0
        ts = torch.where(ok, total, torch.ones_like(total))
        for a in range(self.N):
            m = (D > 0.0) & act[a] & (ph[a] + d[a] > 0.0) & (ph[a] + d[a] < 1.0)
            d[a] = torch.where(m, d[a] - torch.where(ok, D * ph[a] / ts, D / count.clamp(min=1.0)), d[a])
        hit = torch.full(d[0].shape, -1, dtype=torch.int64, device=d[0].device)
        for a in range(self.N):
            hit = torch.where((hit < 0) & act[a] & (ph[a] + d[a] > 1.0), torch.full_like(hit, a), hit)
        return [torch.where(hit == a, 1.0 - ph[a], torch.where((hit >= 0) & act[a], -ph[a], d[a]))
                for a in range(self.N)]

    def _project_nw(self, ph, act, d):
        d = list(d)
        inside = [act[a] & (ph[a] + d[a] > 0.0) & (ph[a] + d[a] < 1.0) for a in range(self.N)]
        count = sum(i.to(_F64) for i in inside).clamp(min=1.0)
        done = torch.zeros_like(act[0])
        for a in range(self.N):
            live = act[a] & ~done
            v = ph[a] + d[a]
            hi, lo = live & (v > 1.0), live & (v < 0.0)
            D = v.abs()
            d[a] = torch.where(hi, 1.0 - ph[a], torch.where(lo, d[a] + D, d[a]))
            for b in range(self.N):
                if b != a:
                    m = lo & act[b] & (ph[b] + d[b] > 0.0) & (ph[b] + d[b] < 1.0)
                    d[b] = torch.where(hi & act[b], -ph[b], torch.where(m, d[b] - D / count, d[b]))
            done = done | hi
        return d

    def step(self, phi, mu, Tp=None, Tc=None, smooth=False):
        """one time step (or smoothing sweep): new phi, mu; Tp, Tc: temperature of
        the ring's columns in the phase-field and the concentration pass"""
        N, K, L, dx, dy = self.N, self.K, self.L, self.dx, self.dy
        P = [f[self.ix[2]][:, self.iy[2]] for f in phi]
        M = [f[self.ix[1]][:, self.iy[1]] for f in mu]
        d = self.delta_phi(P, M, self.T if Tp is None else Tp, smooth)
        ph = [p[1:-1, 1:-1] for p in P]
        E = self._E(self.T if Tc is None else Tc)
        cm = [self.c_of(E, M, a) for a in range(N)]
        xs = lambda q: (q[:-1, 1:-1], q[1:, 1:-1])      # the two cells of the interior's x faces
        ys = lambda q: (q[1:-1, :-1], q[1:-1, 1:])
        H = [self.h(ph, a) for a in range(N)]
        jx, jy = [0.0] * K, [0.0] * K
        if not smooth:
            xf = [(p[1:] - p[:-1]) / dx for p in P]
            yf = [(p[:, 1:] - p[:, :-1]) / dy for p in P]
            cy = [((p[:, 2:] - p[:, :-2]) / (2.0 * dy))[1:-1, 1:-1] for p in P]
            cx = [(0.5 * (f[1:] + f[:-1]))[1:-1, 1:-1] for f in xf]
            w = []
            for a in range(L):
                u = ph[a] * (1.0 - ph[a])
                ok = u > 0.0
                v = ph[a] * (1.0 - H[a]) / torch.sqrt(torch.where(ok, u, torch.ones_like(u)))
                w.append(torch.where(ok, v, torch.zeros_like(v)))
            yl = torch.arange(-1, self.my, device=M[0].device) != self.my - 5
            for xface in (True, False):
                gr = [f[1:-1, 2:-2] for f in xf] if xface else [f[2:-2, 1:-1] for f in yf]
                cn = [0.5 * (c[:-1] + c[1:]) for c in cy] if xface else [0.5 * (c[:, :-1] + c[:, 1:]) for c in cx]
                at = xs if xface else ys
                nl2 = cn[L] * cn[L] + gr[L] * gr[L]
                nl = torch.sqrt(torch.where(nl2 > 0.0, nl2, torch.ones_like(nl2)))
                for a in range(L):
                    s2 = cn[a] * cn[a] + gr[a] * gr[a]
                    on = s2 != 0.0
                    ng = torch.sqrt(torch.where(on, s2, torch.ones_like(s2)))
                    sp = gr[a] * gr[L] + cn[a] * cn[L]
                    sp = torch.where(nl2 > 0.0, sp / (nl * ng), sp)
                    on = on if xface else on & yl
                    for k in range(K):
                        q0, q1 = at(w[a] * (cm[L][k] - cm[a][k]) * d[a])
                        j = self.atf[a][k] * sp.abs() * 0.5 * (q1 + q0) * gr[a] / ng
                        j = torch.where(on, j, torch.zeros_like(j))
                        if xface:
                            jx[k] = jx[k] + j
                        else:
                            jy[k] = jy[k] + j
        flux, cst = [], -0.25 * math.pi * self.eps
        for k in range(K):
            fx = fy = 0.0
            for l in range(K):
                D = sum(self.DC[b][k][l] * ph[b] for b in range(N))
                (a0, a1), (m0, m1) = xs(D), xs(M[l])
                fx = fx + 0.5 * (a1 + a0) * ((m1 - m0) / dx)
                (a0, a1), (m0, m1) = ys(D), ys(M[l])
                fy = fy + 0.5 * (a1 + a0) * ((m1 - m0) / dy)
            v = self.dt * ((fx[1:] - fx[:-1]) / dx + (fy[:, 1:] - fy[:, :-1]) / dy)
            if not smooth:
                v = v - ((jx[k][1:] - jx[k][:-1]) * cst / dx + (jy[k][:, 1:] - jy[k][:, :-1]) * cst / dy)
            flux.append(v)
        I = lambda q: q[1:-1, 1:-1]
        p, dp, m = [I(q) for q in ph], [I(q) for q in d], [I(q) for q in M]
        Ei = [[(I(e.expand_as(M[0])) if torch.is_tensor(e) else e) for e in r] for r in E]
        c = [[I(q) for q in r] for r in cm]
        Hi = [I(q) for q in H]
        dc = list(flux)
        if not smooth:
            for a in range(N):
                t = sum(self.dh(p, a, b) * dp[b] for b in range(N))
                dc = [dc[k] - c[a][k] * t for k in range(K)]
        S = [[sum(self.cmu[a][i][j] * Hi[a] for a in range(N)) for j in range(K)] for i in range(K)]
        if K == 1:
            new = [m[0] + dc[0] / S[0][0]]
        else:
            det = S[0][0] * S[1][1] - S[0][1] * S[1][0]
            new = [m[0] + (S[1][1] * dc[0] - S[0][1] * dc[1]) / det, m[1] + (S[0][0] * dc[1] - S[1][0] * dc[0]) / det]
        done = torch.zeros_like(p[0], dtype=torch.bool)
        for a in range(N):                   # a cell of one phase: through that phase's composition
            pure = (p[a] == 1.0) & ~done
            done = done | pure
            b = self._Mu(Ei, [c[a][k] + flux[k] for k in range(K)], a)
            new = [torch.where(pure, b[k], new[k]) for k in range(K)]
        return torch.stack([p[a] + dp[a] for a in range(N)]), torch.stack(new)

    # -- the temperature field and the moving frame of a program case
    def rows(self, t, off, offT, dlast, fresh):
        """temperature of the ring's columns -1..my in the two passes of the step after step t"""
        base, dT, dist, offset, vel = self.kw["tempgrady"]
        ry = self.my + 6
        sh, dd = (offT, dlast) if fresh else (off, 0)
        pos = offset / self.dy - sh + (vel / self.dy * (t * self.dt) if t else 0.0)
        grad = dT * self.dy / dist
        tb = base - pos * grad
        y = np.arange(ry)
        laid = tb + np.where(y <= ry - 1 - dd, y + dd, y) * grad
        src = np.array(_copy_rows(self.my, self.by, 3)) + 3
        tc = laid[src]
        tp = tc if t == 0 else laid
        f = lambda v: torch.tensor(v, dtype=_F64, device="cuda")
        return f(tp[2:-2])[None, :], f(tc[2:-2])[None, :], f(laid[3:-3]), f(tc[3:-3])


def _copy_rows(m, bc, w):
    """interior row each of the rows -w..m+w-1 is a copy of"""
    out = []
    for v in range(-w, m + w):
        if v < 0:
            v = -v if bc == 1 else v + m - 1
        elif v >= m:
            v = 2 * (m - 1) - v if bc == 1 else v - (m - 1)
        out.append(v)
    return out


def _advance(model, phi, mu, steps, smooth=False):
    """`steps` steps; long runs replay one captured step"""
    if steps < 20:
        for _ in range(steps):
            phi, mu = model.step(phi, mu, smooth=smooth)
        return phi, mu
    phi, mu = phi.clone(), mu.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        model.step(phi, mu, smooth=smooth)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a, b = model.step(phi, mu, smooth=smooth)
        phi.copy_(a)
        mu.copy_(b)
    for _ in range(steps):
        graph.replay()
    torch.cuda.synchronize()
    return phi, mu


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        return [_advance(Model(_input(m)), *_fields(m, seed * 64 + i), steps)
                for i, m in enumerate(_members(case, seed))]
    model = Model(_input(case))
    phi, mu = _fields(case, seed)
    if kind == "smooth":
        phi, mu = _advance(model, phi, mu, steps, smooth=True)
        return dict(phi=phi, mu=mu)
    if kind == "program":
        return _exact_program(model, phi, mu, steps)
    if kind == "rollout":
        return _exact_rollout(case, model, phi, mu, seed, steps)
    phi, mu = _advance(model, phi, mu, steps)
    out = dict(phi=phi, mu=mu)
    if kind == "step":
        out["stats"] = None
    return out


def _exact_program(model, phi, mu, steps):
    off = offT = dlast = 0
    fresh = False
    L, my, shiftj = model.L, model.my, model.kw["shiftj"]
    _, tc, _, _ = model.rows(0, 0, 0, 0, False)
    for _ in range(9):
        phi, mu = model.step(phi, mu, Tc=tc, smooth=True)
    for t in range(steps):
        tp, tc, _, _ = model.rows(t, off, offT, dlast, fresh)
        fresh = False
        phi, mu = model.step(phi, mu, Tp=tp, Tc=tc)
        if (t + 1) % 100 == 0:               # the frame follows the interface
            a, b = phi[L][:, :-1], phi[L][:, 1:]
            up = torch.nonzero((a < 0.5) & (b > 0.5))
            pos = int(up[:, 1].max()) + 1 + 3 if len(up) else 0
            d = pos - shiftj
            if d > 0:
                src = torch.tensor(_copy_rows(my, model.by, 3)[3 + d:], device="cuda")
                n = min(my, len(src))
                fp, fm = torch.zeros_like(phi), torch.zeros_like(mu)
                fp[L] = 1.0
                fill = model._Mu(model._E(1.0), model.c_far, L)
                for k in range(model.K):
                    fm[k] = fill[k]
                fp[:, :, :n], fm[:, :, :n] = phi[:, :, src[:n]], mu[:, :, src[:n]]
                phi, mu = fp, fm
                offT, dlast, fresh, off = off, d, True, off + d
    _, _, laid, _ = model.rows(steps, off, offT, dlast, fresh)
    return dict(phi=phi, mu=mu, T=laid[None, :].expand(model.mx, my), stats=None)


def _exact_rollout(case, model, phi, mu, seed, steps):
    from torch.utils.checkpoint import checkpoint
    phi, mu = phi.requires_grad_(), mu.requires_grad_()
    theta = torch.tensor([model.tau_ab[0, 1], model.dab[0, 1], model.eps, model.gamma[0, 1]], dtype=_F64,
                         device="cuda", requires_grad=True)

    def one(p, m, th):
        for pair in ((0, 1), (1, 0)):
            model.tau_ab[pair], model.dab[pair], model.gamma[pair] = th[0], th[1], th[3]
        model.eps = th[2]
        return model.step(p, m)

    p, m = phi, mu
    for _ in range(steps):
        p, m = checkpoint(one, p, m, theta, use_reentrant=False)
    loss = 0.5 * ((p - _fields(case, seed, grow=4.0)[0]) ** 2).sum()
    g = torch.autograd.grad(loss, (phi, mu, theta))
    return dict(phi=p.detach(), mu=m.detach(), loss=loss.detach(), g_phi=g[0], g_mu=g[1], g_theta=g[2].cpu())
