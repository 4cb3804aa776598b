"""The work that users of the propagation engine have it do, as timed cases.

Every case is one pass through the public entry points: a propagation of a
whole hierarchy over a few output intervals (single model or batch, host or
device state, every solver), one evaluation of the right-hand side for a
program with an integrator of its own, or some training steps of the learned
closure.  `exact` restates each case in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch

import libheom_gb300 as lh
from libheom_gb300 import configs
from libheom_gb300 import terminator
from libheom_gb300.noise import drude_lorentz_terms, noise_members
from libheom_gb300.params import HeomParams


def listed():
    return [
        # the smallest call: a program with its own integrator asks for one
        # right-hand side of a small hierarchy (286 ADOs of 2 x 2), host arrays
        dict(name="rhs_spin_boson", kind="rhs", model="spin_boson", depth=10, precision="fp64"),
        # the plain drop-in on the textbook two-level system, numpy state, as a Python user calls it
        dict(name="spin_boson_rk4", kind="solve", model="spin_boson", depth=10, solver="rk4", precision="fp64",
             dt=0.005, steps=200, intervals=2, host=True),
        # a two-level system whose coupling does not commute with the populations (a dense V)
        dict(name="spin_boson_x_rk4", kind="solve", model="spin_boson_x", depth=10, solver="rk4", precision="fp64",
             dt=0.005, steps=200, intervals=2, host=True),
        # the 7-site exciton aggregate with step control, the form meant for production runs
        dict(name="exciton7_rkdp_mixed", kind="solve", model="aggregate", n=7, depth=4, solver="rkdp",
             precision="mixed", dt=0.1, t_final=100.0, intervals=4),
        # the same as the plain FP64 drop-in
        dict(name="exciton7_rkdp_fp64", kind="solve", model="aggregate", n=7, depth=4, solver="rkdp",
             precision="fp64", dt=0.1, t_final=50.0, intervals=2),
        # the Liouville-space form of it
        dict(name="exciton7_liou_rk4", kind="solve", model="aggregate", form="liou", n=7, depth=3, solver="rk4",
             precision="fp64", dt=0.5, steps=20, intervals=2),
        # static disorder: 16 realisations of the 7-site aggregate stepped together
        dict(name="ensemble_rk4_mixed", kind="batch", model="ensemble", n=7, depth=4, count=16, solver="rk4",
             precision="mixed", dt=1.0, steps=20, intervals=2),
        # a parameter sweep: uneven two- and four-level instances (sizes from `mix`), a numpy state;
        # the range guard keeps some of them in FP64
        dict(name="sweep_rk4_mixed", kind="batch", model="sweep", mix=2, count=128, solver="rk4",
             precision="mixed", dt=0.005, steps=200, intervals=2, host=True),
        # the largest: 24 sites, 20825 ADOs, 192 MB of FP64 state
        dict(name="aggregate24_lsrk4_mixed", kind="solve", model="aggregate", n=24, depth=3, solver="lsrk4",
             precision="mixed", dt=0.5, steps=20, intervals=2),
        # the same as the plain FP64 drop-in
        dict(name="aggregate24_lsrk4_fp64", kind="solve", model="aggregate", n=24, depth=3, solver="lsrk4",
             precision="fp64", dt=0.5, steps=4, intervals=1),
        # the 7-site aggregate cut off at depth 3 with the learned closure
        dict(name="closure7_rk4_mixed", kind="solve", model="aggregate", n=7, depth=3, closure=True, solver="rk4",
             precision="mixed", dt=0.5, steps=20, intervals=2),
        # training that closure: eight minibatches of an epoch, then the weights are read
        dict(name="closure7_train", kind="train", n=7, batch=4096, steps=8),
    ]


def draw(rng):
    kind = rng.choice(["rhs", "two_level", "dense", "aggregate", "aggregate", "aggregate", "liou", "ensemble", "sweep",
                       "closure", "train"])
    steps = rng.randint(10, 200)
    if kind == "rhs":
        if rng.random() < 0.5:
            return dict(kind="rhs", model="spin_boson", depth=rng.randint(4, 14),
                        precision=rng.choice(["fp64", "mixed"]))
        n = rng.randint(3, 20)
        return dict(kind="rhs", model="aggregate", n=n, depth=3 if n <= 9 else 2,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "two_level":
        return dict(kind="solve", model="spin_boson", depth=rng.randint(4, 14), solver=rng.choice(["rk4", "lsrk4"]),
                    precision=rng.choice(["fp64", "mixed"]), dt=0.005, steps=steps, intervals=rng.randint(1, 3),
                    host=rng.random() < 0.5)
    if kind == "dense":
        if rng.random() < 0.5:
            return dict(kind="solve", model="spin_boson_x", depth=rng.randint(4, 14),
                        solver=rng.choice(["rk4", "lsrk4"]), precision=rng.choice(["fp64", "mixed"]), dt=0.005,
                        steps=steps, intervals=rng.randint(1, 3), host=True)
        return dict(kind="solve", model="dense", n=rng.randint(2, 9), baths=rng.randint(1, 2), depth=rng.randint(2, 5),
                    solver="rk4", precision=rng.choice(["fp64", "mixed"]), dt=0.005, steps=rng.randint(10, 60),
                    intervals=1)
    if kind == "aggregate":
        n = round(math.exp(rng.uniform(math.log(3), math.log(24))))
        depth = rng.randint(3, 5) if n <= 4 else rng.randint(2, 4) if n <= 8 else rng.randint(2, 3)
        precision = rng.choice(["fp64", "mixed", "mixed"])
        if n <= 8 and rng.random() < 0.5:
            return dict(kind="solve", model="aggregate", n=n, depth=depth, solver="rkdp", precision=precision, dt=0.1,
                        t_final=float(rng.randint(10, 50)), intervals=rng.randint(1, 4))
        return dict(kind="solve", model="aggregate", n=n, depth=depth, solver=rng.choice(["lsrk4", "rk4"]),
                    precision=precision, dt=0.5, steps=rng.randint(2, 4 if n > 12 else 20), intervals=1)
    if kind == "liou":
        return dict(kind="solve", model="aggregate", form=rng.choice(["liou", "ado"]), n=rng.randint(3, 8),
                    depth=rng.randint(2, 3), solver=rng.choice(["rk4", "lsrk4"]),
                    precision=rng.choice(["fp64", "mixed"]), dt=0.5, steps=rng.randint(5, 20), intervals=1)
    if kind == "ensemble":
        return dict(kind="batch", model="ensemble", n=rng.randint(5, 8), depth=rng.randint(2, 4),
                    count=rng.randint(2, 12), solver=rng.choice(["rk4", "lsrk4"]),
                    precision=rng.choice(["fp64", "mixed", "mixed"]), dt=1.0, steps=rng.randint(5, 20), intervals=1)
    if kind == "sweep":
        return dict(kind="batch", model="sweep", mix=rng.randint(3, 1000), count=rng.randint(12, 128), solver="rk4",
                    precision=rng.choice(["fp64", "mixed"]), dt=0.005, steps=steps, intervals=rng.randint(1, 2),
                    host=True)
    if kind == "closure":
        return dict(kind="solve", model="aggregate", n=rng.randint(3, 7), depth=rng.randint(2, 3), closure=True,
                    solver="rk4", precision=rng.choice(["fp64", "mixed"]), dt=0.5, steps=rng.randint(5, 20),
                    intervals=1)
    return dict(kind="train", n=rng.choice([2, 3, 5, 7]), batch=rng.randint(500, 6000), steps=rng.randint(2, 8))


# ---------------------------------------------------------------- inputs
def _two_level(case, seed, coupling):
    r = np.random.default_rng([seed, 11])
    return configs.spin_boson(eps=r.uniform(-1, 1), delta=r.uniform(0.8, 1.2), lam=r.uniform(0.3, 0.6),
                              depth=case["depth"], coupling=coupling)


def _dense(case, seed):
    """n levels, every bath coupled through a dense Hermitian V."""
    r = np.random.default_rng([seed, 12])
    n = case["n"]

    def herm(scale):
        m = r.standard_normal((n, n)) + 1j * r.standard_normal((n, n))
        return scale * (m + m.conj().T) / (2 * math.sqrt(n))

    g, p, s, S, A, sd = noise_members(*drude_lorentz_terms(0.3, 1.0, 1.0, 1))
    U = case["baths"]
    return HeomParams(H=herm(1.0), V=[herm(0.7) for _ in range(U)], gamma=[g] * U, phi_0=[p] * U, sigma=[s] * U,
                      S=[S] * U, A=[A] * U, s_delta=[sd] * U, max_depth=case["depth"], name="dense")


def _instances(case, seed):
    """The models of a case; their sizes depend on the case alone."""
    model = case["model"]
    if model in ("spin_boson", "spin_boson_x"):
        return [_two_level(case, seed, "x" if model == "spin_boson_x" else "z")]
    if model == "dense":
        return [_dense(case, seed)]
    if model in ("aggregate", "ensemble"):
        seeds = [seed] if model == "aggregate" else [1000 * (seed % 1000003) + i for i in range(case["count"])]
        if case["n"] == 7:
            return [configs.exciton_7site(seed=x, depth=case["depth"]) for x in seeds]
        return [configs.aggregate_24site(seed=x, depth=case["depth"], n_sites=case["n"]) for x in seeds]
    if model == "sweep":
        m, r = np.random.default_rng([case["mix"], 13]), np.random.default_rng([seed, 13])
        out = []
        for i in range(case["count"]):
            if i < 3 * case["count"] // 4:
                lam, beta = math.exp(m.uniform(math.log(0.05), math.log(5.0))), m.uniform(0.1, 10.0)
                out.append(configs.spin_boson(eps=r.uniform(-2, 2), lam=lam, beta=beta, depth=int(m.integers(4, 15))))
            else:
                out.append(configs.chain_4level(r.uniform(-1, 1, 3), r.normal(0, 1, 4), int(m.integers(4, 9))))
        return out
    raise ValueError(model)


def _start(p, r):
    """A random pure state in the system block, empty auxiliary ADOs."""
    n = p.n_level
    v = r.standard_normal(n) + 1j * r.standard_normal(n)
    rho = np.zeros((p.n_hrchy(), n, n), dtype=np.complex128)
    rho[0] = np.outer(v, v.conj()) / np.vdot(v, v).real
    return rho


def _start_states(ps, seed):
    r = np.random.default_rng([seed, 14])
    return [_start(p, r) for p in ps]


def _full_state(p, seed):
    """A state in mid-propagation: every ADO filled, smaller tier by tier."""
    r = np.random.default_rng([seed, 15])
    tier = _tables(p.n_modes, p.max_depth)[0].sum(1)
    shape = (p.n_hrchy(), p.n_level, p.n_level)
    return (r.standard_normal(shape) + 1j * r.standard_normal(shape)) * (0.3 ** tier)[:, None, None]


def _times(case):
    t_final = case["t_final"] if "t_final" in case else case["dt"] * case["steps"]
    return [t_final * i / case["intervals"] for i in range(case["intervals"] + 1)]


def _kwargs(case):
    return dict(dt=case["dt"], atol=1e-8, rtol=1e-8) if case["solver"] == "rkdp" else dict(dt=case["dt"])


HIDDEN = 256


def _net(din, dout, seed, head_bias):
    """Weights of the closure network, packed W1, b1, W2, b2, W3, b3."""
    r = np.random.default_rng([seed, 16])
    out = []
    for i, (a, b) in enumerate(((din, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, dout))):
        lim = math.sqrt(6.0 / a) * (0.1 if i == 2 else 1.0)
        out.append(r.uniform(-lim, lim, (b, a)).ravel())
        bias = np.zeros(b)
        if i == 2:
            bias[b // 2:] = head_bias  # the damping half of the head
        out.append(bias)
    return np.concatenate(out).astype(np.float32)


def _train_data(case, seed, device):
    """Feature and target rows of the closure loss: unit-scale ADOs and their
    children, the sign pattern of a bath at a random site per row."""
    n, B, S = case["n"], case["batch"], case["steps"]
    n2, K = n * n, 2 * n
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(S * B, 4 * n2 + K, generator=g) * 0.4
    k = torch.randint(0, K, (S * B,), generator=g)
    x[:, 2 * n2:2 * n2 + K] = torch.nn.functional.one_hot(k, K).float()
    r = torch.randn(S * B, 2, n2, generator=g) * 0.5
    site = torch.eye(n)[k // 2]
    sg = (site[:, :, None] - site[:, None, :]).reshape(S * B, n2)
    re, im = 0.3 + 0.1 * x[:, :n2], -0.5 * sg
    t = torch.stack([re * r[:, 0] - im * r[:, 1], re * r[:, 1] + im * r[:, 0]], 1)
    t = t + 0.05 * torch.randn(t.shape, generator=g)
    T = torch.cat([t.reshape(S * B, -1), r.reshape(S * B, -1), sg], 1)
    return [(x[i * B:(i + 1) * B].to(device).contiguous(), T[i * B:(i + 1) * B].to(device).contiguous())
            for i in range(S)]


# ---------------------------------------------------------------- the entry points
def prepare(case, seed):
    s = types.SimpleNamespace(case=case)
    if case["kind"] == "train":
        n2 = case["n"] ** 2
        din, dout = 4 * n2 + 2 * case["n"], 2 * n2
        s.mlp = terminator.MLP(din, HIDDEN, dout)
        s.mlp.set_params(_net(din, dout, seed, 0.0))
        s.mlp.set_loss(1, n2)
        s.data = _train_data(case, seed, "cuda")
        return s
    ps = _instances(case, seed)
    s.stream = torch.cuda.Stream()
    s.qmes = [lh.from_params(p, form=case.get("form", "hilb"), precision=case["precision"],
                             stream=s.stream.cuda_stream) for p in ps]
    if case["kind"] == "rhs":
        s.rho = _full_state(ps[0], seed)
        s.out = np.zeros_like(s.rho)
        return s
    if case.get("closure"):
        din, dout = terminator.dims(ps[0])
        s.mlp = terminator.MLP(din, HIDDEN, dout)
        s.mlp.set_params(_net(din, dout, seed, -5.0))
        terminator.attach(s.qmes[0], s.mlp)
    solver = lh.SOLVERS[case["solver"]]()
    s.solver = lh.batch_solver(s.qmes, solver) if case["kind"] == "batch" else lh.qme_solver(s.qmes[0], solver)
    s.rho0 = np.concatenate([x.ravel() for x in _start_states(ps, seed)])
    if not case.get("host"):
        with torch.cuda.stream(s.stream):
            s.rho0 = torch.from_numpy(s.rho0).cuda()
            s.rho = torch.empty_like(s.rho0)
        s.stream.synchronize()
    s.times, s.kw = _times(case), _kwargs(case)
    return s


def run(s):
    case = s.case
    if case["kind"] == "train":
        losses = [s.mlp.train_step(x.data_ptr(), t.data_ptr(), case["batch"], 1e-3) for x, t in s.data]
        return dict(loss=torch.tensor(losses, dtype=torch.float32), weights=s.mlp.get_params())
    if case["kind"] == "rhs":
        s.qmes[0].calc_diff_impl(s.out, s.rho)
        return s.out
    if case.get("host"):
        rho = s.rho0.copy()
        s.solver.solve(rho, s.times, None, s.kw)
        return rho
    with torch.cuda.stream(s.stream):
        s.rho.copy_(s.rho0)
    s.solver.solve_device(s.rho.data_ptr(), s.times, None, s.kw)
    return s.rho


def work(case):
    if case["kind"] == "train":
        n2, B, S = case["n"] ** 2, case["batch"], case["steps"]
        din, dout = 4 * n2 + 2 * case["n"], 2 * n2
        weights = HIDDEN * (din + HIDDEN + dout)
        # forward and weight gradients of three layers, data gradients of two
        return dict(bytes=4.0 * (S * B * (din + 5 * n2) + 2 * weights),
                    flops=2.0 * S * B * (3 * weights - HIDDEN * din))
    size = flops = 0.0
    for p in _instances(case, 0):
        n, K, nh = p.n_level, p.n_modes, p.n_hrchy()
        diag = all(np.count_nonzero(v - np.diag(np.diag(v))) == 0 for v in p.V)
        size += nh * n * n
        # commutator (real H: half), damping, and two neighbours' terms of every
        # mode that an element couples to; a dense V adds its products per bath
        per = n * (8 if np.all(p.H.imag == 0) else 16) + 8
        modes = K / p.n_noise * (2 * (1 - 1 / n) if p.n_noise == n else p.n_noise)
        per += 16 * modes if diag else 32 * n * p.n_noise + 16 * K
        if case.get("closure"):
            din, dout = 4 * n * n + K, 2 * n * n
            tier = math.comb(K + p.max_depth - 1, p.max_depth)
            flops += 2.0 * tier * K * HIDDEN * (din + HIDDEN + dout)
        flops += nh * n * n * per
    evals = 1 if case["kind"] == "rhs" else 4 * case["steps"] if "steps" in case else 7 * (8 + case["t_final"] / 3)
    return dict(bytes=32.0 * size, flops=flops * evals)


# ---------------------------------------------------------------- 64-bit restatement
def _tables(K, depth):
    """Multi-indices tier by tier, each tier in descending order, with the
    numbers of the raised and lowered neighbours (the count itself: none)."""
    rows = []

    def fill(prefix, left, total):
        if left == 1:
            rows.append(prefix + (total,))
            return
        for v in range(total, -1, -1):
            fill(prefix + (v,), left - 1, total - v)

    for d in range(depth + 1):
        fill((), K, d)
    at = {r: i for i, r in enumerate(rows)}
    nh = len(rows)
    up, down = np.full((nh, K), nh), np.full((nh, K), nh)
    for i, r in enumerate(rows):
        for k in range(K):
            if r[k]:
                j = at[r[:k] + (r[k] - 1,) + r[k + 1:]]
                down[i, k] = j
                up[j, k] = i
    return np.array(rows), up, down


class _Group:
    """Instances with the same number of levels and modes, padded to the
    deepest: D(rho) of the hierarchy with plain 64-bit products."""

    def __init__(self, ps, dev):
        K, n = ps[0].n_modes, ps[0].n_level
        self.n, self.K, self.I = n, K, len(ps)
        self.nh = [p.n_hrchy() for p in ps]
        self.M = max(self.nh)
        tab = {p.max_depth: _tables(K, p.max_depth) for p in ps}
        occ, up = np.zeros((self.I, self.M, K)), np.full((self.I, self.M, K), self.M)
        down = np.full((self.I, self.M, K), self.M)
        for i, p in enumerate(ps):
            t, u, d = tab[p.max_depth]
            h = self.nh[i]
            occ[i, :h] = t
            up[i, :h] = np.where(u == h, self.M, u)
            down[i, :h] = np.where(d == h, self.M, d)
        base = np.arange(self.I)[:, None, None] * (self.M + 1)
        self.dev = dev

        def c(a):
            return torch.as_tensor(np.asarray(a, dtype=np.complex128), device=dev)

        self.occ = torch.as_tensor(occ, device=dev)
        self.up, self.down = (torch.as_tensor((x + base).reshape(-1, K), device=dev) for x in (up, down))
        self.bath = np.concatenate([[u] * len(ps[0].sigma[u]) for u in range(ps[0].n_noise)]).astype(int)
        flat = [[(p.sigma[u][k], (p.S[u] @ p.phi_0[u])[k], (p.A[u] @ p.phi_0[u])[k], p.gamma[u][k, k])
                 for u in range(p.n_noise) for k in range(len(p.sigma[u]))] for p in ps]
        self.sig, self.s, self.a, gam = (c([[m[j] for m in f] for f in flat]) for j in range(4))
        self.gam = gam
        self.damp = (self.occ.to(torch.complex128) * gam[:, None, :]).sum(-1)
        self.H = c([p.H for p in ps])
        self.V = c([p.V for p in ps])
        off = self.V - torch.diag_embed(torch.diagonal(self.V, dim1=-2, dim2=-1))
        self.diag = not bool((off != 0).any())
        self.reach = [torch.nonzero(self.down.reshape(-1, K)[:, k] % (self.M + 1) != self.M).ravel() for k in range(K)]
        self.rise = [torch.nonzero(self.up.reshape(-1, K)[:, k] % (self.M + 1) != self.M).ravel() for k in range(K)]
        self.inst = torch.arange(self.I, device=dev).repeat_interleave(self.M)

    def pack(self, states):
        F = torch.zeros((self.I, self.M, self.n, self.n), dtype=torch.complex128, device=self.dev)
        for i, x in enumerate(states):
            F[i, :self.nh[i]] = torch.as_tensor(x, device=self.dev)
        return F

    def unpack(self, F):
        return [F[i, :self.nh[i]].cpu().numpy() for i in range(self.I)]

    def __call__(self, F, extra=None):
        n = self.n
        pad = torch.cat([F, torch.zeros_like(F[:, :1])], 1).reshape(-1, n, n)
        H = self.H[:, None]
        D = (1j * (H @ F - F @ H) + self.damp[:, :, None, None] * F).reshape(-1, n, n)
        for u in range(self.V.shape[1]):
            ph, ps = torch.zeros_like(D), torch.zeros_like(D)
            for k in np.nonzero(self.bath == u)[0]:
                rows = self.rise[k]
                if len(rows):
                    ph[rows] += self.sig[self.inst[rows], k][:, None, None] * pad[self.up[rows, k]]
                rows = self.reach[k]
                if len(rows):
                    x = pad[self.down[rows, k]] * self.occ.reshape(-1, self.K)[rows, k][:, None, None]
                    ph[rows] += self.s[self.inst[rows], k][:, None, None] * x
                    ps[rows] -= self.a[self.inst[rows], k][:, None, None] * x
            if extra is not None:
                ph += extra[u]
            if self.diag:
                v = torch.diagonal(self.V[:, u], dim1=-2, dim2=-1)[self.inst]
                D += 1j * (v[:, :, None] - v[:, None, :]) * ph + (v[:, :, None] + v[:, None, :]) * ps
            else:
                V = self.V[self.inst, u]
                D += 1j * (V @ ph - ph @ V) + V @ ps + ps @ V
        return D.reshape(F.shape)


def _closure(g, p, params):
    """The network's stand-in for the +1 neighbours of the deepest tier: per
    bath, sigma_k rho_{n+1_k} summed over its modes, for every ADO."""
    n, K, dev = g.n, g.K, g.dev
    n2 = n * n
    din, dout = 4 * n2 + K, 2 * n2
    w, i = [], 0
    for a, b in ((din, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, dout)):
        w.append(torch.as_tensor(params[i:i + a * b].reshape(b, a).astype(np.float64), device=dev))
        w.append(torch.as_tensor(params[i + a * b:i + a * b + b].astype(np.float64), device=dev))
        i += a * b + b
    tier = math.comb(K + p.max_depth - 1, p.max_depth)
    first = g.M - tier
    v = torch.diagonal(g.V[0], dim1=-2, dim2=-1)[torch.as_tensor(g.bath, device=dev)]  # (K, n)
    dv, sv = v[:, :, None] - v[:, None, :], v[:, :, None] + v[:, None, :]
    c = (-1j * g.s[0][:, None, None] * dv + g.a[0][:, None, None] * sv).reshape(K, n2)
    sg = torch.sign(dv.real).reshape(K, n2)
    rate = (g.occ[0, first:] + 1) / (g.damp[0, first:, None] + g.gam[0][None, :])
    gelu = torch.nn.functional.gelu

    def extra(F):
        R = F[0, first:].reshape(tier, n2)
        s = R.abs().amax(1).clamp_min(1e-300)
        A = rate[:, :, None] * c[None] * R[:, None] / s[:, None, None]
        Rn = (R / s[:, None])[:, None].expand(tier, K, n2)
        hot = torch.eye(K, dtype=torch.float64, device=dev).expand(tier, K, K)
        x = torch.cat([Rn.real, Rn.imag, hot, A.real, A.imag], 2)
        y = gelu(gelu(x @ w[0].T + w[1]) @ w[2].T + w[3]) @ w[4].T + w[5]
        C = torch.complex(y[..., :n2], -sg * torch.nn.functional.softplus(y[..., n2:])) * sg.abs()
        P = (C * R[:, None]).reshape(tier, K, n, n)  # sigma_k rho_{n+1_k}
        out = []
        for u in range(g.V.shape[1]):
            z = torch.zeros((g.M, n, n), dtype=torch.complex128, device=dev)
            z[first:] = P[:, np.nonzero(g.bath == u)[0]].sum(1)
            out.append(z)
        return out

    return extra


_A = ((), (1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
      (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
      (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
      (35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
_E = (-71 / 57600, 0, 71 / 16695, -71 / 1920, 17253 / 339200, -22 / 525, 1 / 40)


def _propagate(f, y, case):
    times, dt, saved = _times(case), case["dt"], case["dt"]
    eps = np.finfo(float).eps
    for t, end in zip(times[:-1], times[1:]):
        if case["solver"] == "rkdp":
            dt = min(saved, end - t) if t + saved > end else saved
            while t < end:
                k = []
                for row in _A:
                    z = y + sum((a * q for a, q in zip(row, k) if a), torch.zeros_like(y))
                    k.append(-dt * f(z))
                e = sum((a * q for a, q in zip(_E, k) if a), torch.zeros_like(y))
                scale = 1e-8 + 1e-8 * torch.maximum(z.abs(), y.abs())
                err = float(((e.abs() / scale) ** 2).mean().sqrt())
                if err < 1.0:
                    t, y, dt = t + dt, z, dt * 0.9 * min(10.0, err ** -0.2 if err else 10.0)
                else:
                    dt *= 0.9 * max(0.2, err ** -0.2)
                if t < end and t + dt > end:
                    dt = end - t
            saved = dt
            continue
        done = False
        while not done:
            h = case["dt"]
            if t + h - end > -eps:
                h, done = end - t, True
            if case["solver"] == "rk4":
                k1 = -h * f(y)
                k2 = -h * f(y + k1 / 2)
                k3 = -h * f(y + k2 / 2)
                k4 = -h * f(y + k3)
                y = y + (k1 + 2 * k2 + 2 * k3 + k4) / 6
            else:  # the low-storage form: b = k - b, y += w b
                b = torch.zeros_like(y)
                for w in (1 / 3, 3 / 4, 2 / 3, 1 / 4):
                    b = -h * f(y) - b
                    y = y + w * b
            t += h
    return y


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "train":
        return _exact_train(case, seed, dev)
    ps = _instances(case, seed)
    if case["kind"] == "rhs":
        g = _Group(ps, dev)
        return g.unpack(-g(g.pack([_full_state(ps[0], seed)])))[0]
    states, out = _start_states(ps, seed), [None] * len(ps)
    for key in sorted({(p.n_level, p.n_modes) for p in ps}):
        at = [i for i, p in enumerate(ps) if (p.n_level, p.n_modes) == key]
        g = _Group([ps[i] for i in at], dev)
        f = g
        if case.get("closure"):
            din, dout = 4 * g.n ** 2 + g.K, 2 * g.n ** 2
            extra = _closure(g, ps[0], _net(din, dout, seed, -5.0))
            f = lambda F: g(F, extra(F))  # noqa: E731
        for i, x in zip(at, g.unpack(_propagate(f, g.pack([states[i] for i in at]), case))):
            out[i] = x.ravel()
    return np.concatenate(out)


def _exact_train(case, seed, dev):
    n2 = case["n"] ** 2
    din, dout = 4 * n2 + 2 * case["n"], 2 * n2
    flat = torch.as_tensor(_net(din, dout, seed, 0.0).astype(np.float64), device=dev)
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    gelu = torch.nn.functional.gelu
    for step, (x, T) in enumerate(_train_data(case, seed, dev), 1):
        x, T = x.double(), T.double()
        flat.requires_grad_(True)
        z, i = x, 0
        for j, (a, b) in enumerate(((din, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, dout))):
            z = z @ flat[i:i + a * b].reshape(b, a).T + flat[i + a * b:i + a * b + b]
            i += a * b + b
            z = gelu(z) if j < 2 else z
        t_re, t_im, r_re, r_im, sg = T.split(n2, 1)
        c_re, c_im = z[:, :n2], -sg * torch.nn.functional.softplus(z[:, n2:])
        on = sg.abs()
        num = on * ((c_re * r_re - c_im * r_im - t_re) ** 2 + (c_re * r_im + c_im * r_re - t_im) ** 2)
        den = on * (t_re ** 2 + t_im ** 2 + 1e-2 * (r_re ** 2 + r_im ** 2))
        loss = (num.sum(1) / (den.sum(1) + 1e-6)).mean()
        grad, = torch.autograd.grad(loss, flat)
        losses.append(float(loss))
        flat = flat.detach()
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        flat = flat - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return dict(loss=torch.tensor(losses), weights=flat.float().cpu().double().numpy())
