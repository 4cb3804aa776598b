"""FP64 stages with the commutator on the tensor cores (k_rhs_split) against the
port and k_rhs_diag.  The digits carry 62 bits below the largest element of an
ADO and their products are exact, so a stage differs from the FP64 sums by
their own rounding: 1e-12 of the largest element after 20 steps of about 100
products each.  Levels at the edges of the padding (4, 8, 16, 32 and odd ones),
tiles that end inside the hierarchy, sqrt normalisation, column-major states, a
filtered hierarchy, uneven batches, states over 400 decades, and infinities,
which take the FP64 sums."""
import dataclasses

import numpy as np
import pytest

import libheom_gb300 as lh
import oracle
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu


def agg(n, depth, **kw):
    return dataclasses.replace(configs.aggregate_24site(n_sites=n, depth=depth), **kw)


CASES = {
    "n4": lambda: agg(4, 4),
    "n5_sqrt": lambda: agg(5, 3, normalization="sqrt"),
    "n7_col": lambda: agg(7, 3, order="col_major"),
    "n8": lambda: agg(8, 2),
    "n12_filtered": lambda: agg(12, 2, hrchy_filter=lambda i, d: i[0] <= 1),
    "n16": lambda: agg(16, 2),
    "n17": lambda: agg(17, 1),
    "n24": lambda: agg(24, 2),
    "n32": lambda: agg(32, 1),
}
DT = 0.5


def state(p, seed=0):
    rng = np.random.default_rng(seed)
    rho = p.rho0_ground()
    return rho + 0.1 * (rng.standard_normal(rho.shape) + 1j * rng.standard_normal(rho.shape))


def solve(ps, solver, rho, split, monkeypatch, ts=(0.0, 3.7, 10.0)):
    for k, v in dict(HEOMGB_SPLIT=split, HEOMGB_RESIDENT="0", HEOMGB_CLUSTER="0", HEOMGB_LOCAL="0").items():
        monkeypatch.setenv(k, v)
    qs = [lh.from_params(p, precision="fp64") for p in ps]
    s = lh.batch_solver(qs, lh.SOLVERS[solver]()) if len(qs) > 1 else lh.qme_solver(qs[0], lh.SOLVERS[solver]())
    s.solve(rho, list(ts), None, dict(dt=DT) if solver != "rkdp" else dict(dt=DT, atol=1e-9, rtol=1e-9))
    assert all(t["split"] == (split == "1") for t in s.tuning().get("parts", [s.tuning()]))
    return rho


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("solver", ["rk4", "lsrk4", "rkdp"])
def test_split_matches_the_port(case, solver, monkeypatch):
    p = CASES[case]()
    kw = dict(dt=DT) if solver != "rkdp" else dict(dt=DT, atol=1e-9, rtol=1e-9)
    ref = oracle.Oracle("port").solve(p, state(p), [0.0, 3.7, 10.0], solver=solver, **kw)[-1]
    got = solve([p], solver, state(p), "1", monkeypatch)
    tol = 1e-12 if solver != "rkdp" else 1e-9
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


def test_split_batch(monkeypatch):
    ps = [agg(7, 3), agg(5, 2), agg(12, 1)]
    rho = np.concatenate([state(p, i).ravel() for i, p in enumerate(ps)])
    want = solve(ps, "rk4", rho.copy(), "0", monkeypatch)
    got = solve(ps, "rk4", rho.copy(), "1", monkeypatch)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("n", [5, 24])
def test_split_range(n, monkeypatch):
    """Every ADO at a scale of its own, from the bottom of the FP64 range to 1e300 (one step,
    compared ADO by ADO against its own largest element), and zero ADOs."""
    p = agg(n, 1)
    rho = state(p)
    scale = 10.0 ** np.linspace(-310, 300, rho.shape[0])
    scale[::7] = 0.0
    rho *= scale[:, None, None]
    want = solve([p], "rk4", rho.copy(), "0", monkeypatch, (0.0, DT))
    got = solve([p], "rk4", rho.copy(), "1", monkeypatch, (0.0, DT))
    assert np.isfinite(got).all() == np.isfinite(want).all()
    # depth 1: every ADO is a neighbour of ADO 0, and ADO 0 of every other
    big = max(np.abs(want[1:]).max(), np.abs(rho).max())
    assert np.abs(got[0] - want[0]).max() <= 1e-12 * big
    for l in range(1, rho.shape[0]):
        ref = max(np.abs(want[l]).max(), np.abs(rho[l]).max())
        assert np.abs(got[l] - want[l]).max() <= 1e-12 * ref + 1e-300


def test_split_infinities(monkeypatch):
    p = agg(6, 2)
    rho = state(p)
    rho[0, 2, 3] = np.inf
    rho[5, 1, 1] = np.nan
    want = solve([p], "rk4", rho.copy(), "0", monkeypatch, (0.0, DT))
    got = solve([p], "rk4", rho.copy(), "1", monkeypatch, (0.0, DT))
    ok = np.isfinite(want)
    assert np.array_equal(ok, np.isfinite(got))
    assert np.abs(got[ok] - want[ok]).max() <= 1e-12 * np.abs(want[ok]).max()
