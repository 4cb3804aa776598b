"""Fixed steps in the couplings' eigenbasis are no further from the solution than
in the caller's basis, over one interval and with a callback every ten steps.
The solution: the same steps of the scheme in extended precision (numpy's
longdouble: 64 bits of fraction or more) from the same FP64 model."""
import numpy as np
import pytest

import libheom_gb300 as lh
import oracle
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu

DT, STEPS = 2.0**-8, 200  # the sums of the step are exact: every grid of times is the same


def rhs(p):
    """-D(rho) of one bath with diagonal gamma, S and A, in extended precision."""
    C, R = np.clongdouble, np.longdouble
    occ, up, down = oracle.Oracle("port").hrchy(p.n_modes, p.max_depth)
    up, down, n = up[:-1], down[:-1], occ.astype(R)
    H, V = p.H.astype(C), p.V[0].astype(C)
    g = np.diag(np.asarray(p.gamma[0])).astype(C)
    S, A, phi = (np.asarray(x, dtype=complex).astype(C) for x in (p.S[0], p.A[0], p.phi_0[0]))
    s, a, sig, sd = S @ phi, A @ phi, np.asarray(p.sigma[0]).astype(C), C(p.s_delta[0])
    damp = (n * g).sum(1)[:, None, None]

    def f(x):
        pad = np.concatenate([x, np.zeros((1,) + x.shape[1:], C)])
        c = V @ x - x @ V
        d = C(1j) * (H @ x - x @ H) + damp * x + sd * (V @ c - c @ V)
        ph, ps = np.zeros_like(x), np.zeros_like(x)
        for k in range(p.n_modes):
            low = pad[down[:, k]] * n[:, k][:, None, None]
            ph = ph + sig[k] * pad[up[:, k]] + s[k] * low
            ps = ps - a[k] * low
        return -(d + C(1j) * (V @ ph - ph @ V) + V @ ps + ps @ V)

    return f


def steps(f, y, solver):
    R = np.longdouble
    h, y = R(DT), y.astype(np.clongdouble)
    for _ in range(STEPS):
        if solver == "rk4":
            k1 = h * f(y)
            k2 = h * f(y + k1 / R(2))
            k3 = h * f(y + k2 / R(2))
            k4 = h * f(y + k3)
            y = y + (k1 + R(2) * k2 + R(2) * k3 + k4) / R(6)
        else:
            b = np.zeros_like(y)
            for i, j in ((1, 3), (3, 4), (2, 3), (1, 4)):
                b = h * f(y) - b
                y = y + R(i) / R(j) * b
    return y


@pytest.mark.parametrize("solver", ["rk4", "lsrk4"])
def test_no_further_from_the_solution_than_the_general_kernel(solver, monkeypatch):
    err = {(basis, cb): [] for basis in ("own", "common") for cb in (False, True)}
    for seed in range(4):
        r = np.random.default_rng(seed)
        p = configs.spin_boson(eps=r.uniform(-1, 1), delta=r.uniform(0.8, 1.2), lam=r.uniform(0.3, 0.6), depth=5,
                               coupling="x")
        rho0 = p.rho0_ground()
        v = r.standard_normal(2) + 1j * r.standard_normal(2)
        rho0[0] = np.outer(v, v.conj()) / np.vdot(v, v).real
        want = steps(rhs(p), rho0, solver).astype(complex)
        for basis, cb in err:
            monkeypatch.setenv("HEOMGB_CLUSTER", "0" if basis == "own" else "1")
            s = lh.qme_solver(lh.from_params(p, precision="fp64"), lh.SOLVERS[solver]())
            assert s.tuning()["cluster"] == (basis == "common")
            rho = rho0.copy()
            ts = [DT * i for i in range(0, STEPS + 1, 10 if cb else STEPS)]
            s.solve(rho, ts, (lambda t: None) if cb else None, dict(dt=DT))
            err[basis, cb].append(np.linalg.norm(rho - want) / np.linalg.norm(want))
    for cb in (False, True):
        assert np.mean(err["common", cb]) <= np.mean(err["own", cb])
