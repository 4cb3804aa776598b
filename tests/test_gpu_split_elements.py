"""k_rhs_split element by element: the digits of a row of the operand hold 70
bits below the row's largest value, and components whose products are too small
for them take FP64 sums, so every element is as accurate as with FP64 sums
alone, whatever else its ADO holds.

Tolerances: a chain's rows have three entries, so an RK4 step is some 50
roundings of 1.1e-16 on an element's own terms, with cancellations of up to a
factor of 100: 1e-12 of the element."""
import dataclasses

import numpy as np
import pytest

import oracle
from libheom_gb300 import configs
from test_gpu_split import agg, solve, state

pytestmark = pytest.mark.gpu


def chain(n, depth=1, **kw):
    """Nearest-neighbour couplings: small elements stay small for a while."""
    p = agg(n, depth, **kw)
    H = np.diag(np.diag(p.H)) + np.diag(np.full(n - 1, 0.013 + 0j), 1) + np.diag(np.full(n - 1, 0.013 + 0j), -1)
    return dataclasses.replace(p, H=H)


def graded(p, decades):
    """Elements that fall off by `decades` per site in both directions, in every ADO."""
    n = p.n_level
    r = np.random.default_rng(n)
    g = 10.0 ** (-decades * np.arange(n))
    shape = p.rho0_ground().shape
    mag = r.uniform(0.5, 1.0, shape) * np.exp(2j * np.pi * r.uniform(size=shape))
    return mag * (g[:, None] * g[None, :])


@pytest.mark.parametrize("n", [4, 7, 12, 16, 24, 32])
@pytest.mark.parametrize("decades", [0.5, 2])
def test_small_elements_keep_their_bits(n, decades, monkeypatch):
    p, dt = chain(n), 1e-4
    rho = graded(p, decades)
    ref = oracle.Oracle("port").solve(p, rho.copy(), [0.0, dt], solver="rk4", dt=dt)[-1]
    for split in ("0", "1"):
        monkeypatch.setattr("test_gpu_split.DT", dt)
        got = solve([p], "rk4", rho.copy(), split, monkeypatch, (0.0, dt))
        assert (np.abs(got - ref) <= 1e-12 * np.abs(ref)).all()


@pytest.mark.parametrize("n", [7, 24])
@pytest.mark.parametrize("scale", [1e-262, 1e-250, 1e-241, 1e200])
def test_uniformly_scaled_states(n, scale, monkeypatch):
    """The problem is linear: a scaled state gives the scaled answer (about 100
    products a stage, 20 stages: 1e-12 of an ADO's largest element)."""
    p = agg(n, 1)
    want = solve([p], "rk4", state(p), "0", monkeypatch, (0.0, 2.5)) * scale
    got = solve([p], "rk4", state(p) * scale, "1", monkeypatch, (0.0, 2.5))
    top = np.abs(want).max(axis=(1, 2), keepdims=True)
    assert (np.abs(got - want) <= 1e-12 * top).all()


@pytest.mark.parametrize("n", [5, 24])
def test_rows_out_of_the_digits_range(n, monkeypatch):
    """One ADO from the bottom of the FP64 range to its top, row by row: the rows
    that the digits do not hold take FP64 sums and the others keep theirs."""
    p, dt = chain(n, 0), 1e-4
    rho = graded(p, 0)
    rho *= (10.0 ** np.linspace(-145, 145, n))[:, None] * (10.0 ** np.linspace(-145, 145, n))[None, :]
    ref = oracle.Oracle("port").solve(p, rho.copy(), [0.0, dt], solver="rk4", dt=dt)[-1]
    monkeypatch.setattr("test_gpu_split.DT", dt)
    got = solve([p], "rk4", rho.copy(), "1", monkeypatch, (0.0, dt))
    assert (np.abs(got - ref) <= 1e-12 * np.abs(ref) + 1e-300).all()


@pytest.mark.parametrize("n", [6, 24])
def test_energy_offset(n, monkeypatch):
    """Absolute site energies (an offset far above the couplings, which the
    commutator does not see): no further from the offset-free solve than the
    FP64 sums are.  Energies are multiples of 2^-40, so that adding the offset
    is exact."""
    p = agg(n, 1)
    H = np.round(p.H.real * 2.0**40) / 2.0**40
    p = dataclasses.replace(p, H=H.astype(complex))
    q = dataclasses.replace(p, H=(H + 4.0 * np.eye(n)).astype(complex))
    want = solve([p], "rk4", state(p), "0", monkeypatch, (0.0, 20.0))
    off = [np.linalg.norm(solve([q], "rk4", state(p), s, monkeypatch, (0.0, 20.0)) - want) for s in ("0", "1")]
    assert off[1] <= 1.25 * off[0]


@pytest.mark.parametrize("n", [8, 24])
def test_zero_columns_and_zero_parts(n, monkeypatch):
    """An H with an uncoupled site of energy 0 (a column of zeros) and one of 1e-60, and a real state."""
    p, dt = chain(n), 0.5
    H = p.H.copy()
    H[2, :] = H[:, 2] = 0.0
    H[4, :] = H[:, 4] = 0.0
    H[4, 4] = 1e-60
    p = dataclasses.replace(p, H=H)
    rho = state(p).real.astype(complex)
    ref = oracle.Oracle("port").solve(p, rho.copy(), [0.0, 3.7, 10.0], solver="rk4", dt=dt)[-1]
    got = solve([p], "rk4", rho.copy(), "1", monkeypatch)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


def _model(r):
    """A commutator alone (depth 0) with H and the state of one of several shapes."""
    n = int(r.integers(4, 33))
    p = configs.aggregate_24site(n_sites=n, depth=0, seed=int(r.integers(1000)))
    H, kind = p.H.real.copy(), int(r.integers(6))
    if kind == 1:
        H = np.diag(np.diag(H)) + np.diag(np.full(n - 1, 0.01), 1) + np.diag(np.full(n - 1, 0.01), -1)
    elif kind == 2:  # columns over 12 decades
        g = 10.0 ** r.uniform(-12, 0, n)
        H = H * (g[:, None] * g[None, :])
    elif kind == 3:  # few couplings
        m = np.triu(r.uniform(size=(n, n)) < 0.2, 1)
        H = H * (m + m.T)
    elif kind == 4:
        H = H + np.eye(n) * r.uniform(-5, 5)
    elif kind == 5:  # uncoupled sites of energy 0
        z = r.uniform(size=n) < 0.3
        H[z], H[:, z] = 0.0, 0.0
    rho, kind = r.standard_normal((n, n)) + 1j * r.standard_normal((n, n)), int(r.integers(6))
    if kind == 1:
        g = 10.0 ** r.uniform(-30, 0, n)
        rho = rho * (g[:, None] * g[None, :])
    elif kind == 2:
        rho = rho * (r.uniform(size=(n, n)) < 0.15)
    elif kind == 3:
        rho = rho.real + 0j
    elif kind == 4:
        rho = rho * (10.0 ** r.uniform(-100, 100, (n, 1)) * 10.0 ** r.uniform(-100, 100, (1, n)))
    elif kind == 5:
        rho = rho * 10.0 ** r.uniform(-8, 0, (n, n))
    return dataclasses.replace(p, H=H.astype(complex)), rho[None]


@pytest.mark.parametrize("seed", [0, 1])
def test_every_element_within_the_bound_of_fp64_sums(seed, monkeypatch):
    """One RK4 step of a batch of commutators against numpy's longdouble.  An
    element's bound: 2^-53 times the roundings of a chain of FP64 sums (2 n
    products and 10 other operations a stage, 4 stages) times the step formed
    with absolute values."""
    r, dt = np.random.default_rng(seed), 0.05
    models = [_model(r) for _ in range(30)]
    monkeypatch.setattr("test_gpu_split.DT", dt)
    flat = np.concatenate([rho.ravel() for _, rho in models])
    got, o = solve([p for p, _ in models], "rk4", flat, "1", monkeypatch, (0.0, dt)), 0
    for p, rho in models:
        n = p.n_level
        sd = np.zeros((n, n), complex)
        for u in range(p.n_noise):
            v = np.diag(p.V[u])
            sd += p.s_delta[u] * (v[:, None] - v[None, :]) ** 2

        def step(H, s, y, f):
            k1 = f(H, s, y)
            k2 = f(H, s, y + k1 / 2)
            k3 = f(H, s, y + k2 / 2)
            return y + (k1 + 2 * k2 + 2 * k3 + f(H, s, y + k3)) / 6

        C, h = np.clongdouble, np.longdouble(dt)
        want = step(p.H.astype(C), sd.astype(C), rho[0].astype(C), lambda H, s, x: -h * (C(1j) * (H @ x - x @ H) + s * x))
        bound = step(np.abs(p.H), np.abs(sd), np.abs(rho[0].real) + np.abs(rho[0].imag),
                     lambda H, s, x: dt * (H @ x + x @ H + s * x))
        err = np.abs((got[o:o + n * n].reshape(n, n) - want).astype(complex))
        assert (err <= 2.0**-53 * 4 * (2 * n + 10) * bound + 1e-300).all()
        o += n * n
