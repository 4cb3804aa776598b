"""The row kernel (k_rhs_rows: site-local baths, mixed form) against k_rhs_diag.
The arithmetic per element is k_rhs_diag's, in its order, so fixed steps agree
bit for bit; Dormand-Prince sums the error norm in another order, which moves
the FP32 step factor by one unit at most (1e-6 of the largest element covers
the tolerance 1e-6 of the steps).  Levels around the row templates (2..8, then
four-column pieces with a remainder), hierarchies smaller than a group, uneven
batches with different levels, sqrt normalisation, column-major states, a
filtered hierarchy and a closure."""
import dataclasses

import numpy as np
import pytest

import libheom_gb300 as lh
from libheom_gb300 import configs
from libheom_gb300 import terminator as T

pytestmark = pytest.mark.gpu


def agg(n, depth, **kw):
    return dataclasses.replace(configs.aggregate_24site(n_sites=n, depth=depth), **kw)


CASES = {
    "n2": lambda: [agg(2, 5)],
    "n3_tiny": lambda: [agg(3, 1)],
    "n4_sqrt": lambda: [agg(4, 3, normalization="sqrt")],
    "n5_col": lambda: [agg(5, 3, order="col_major")],
    "n6_filtered": lambda: [agg(6, 3, hrchy_filter=lambda i, d: i[0] <= 1)],
    "n7": lambda: [agg(7, 4)],
    "n8": lambda: [agg(8, 3)],
    "n9_deep": lambda: [agg(9, 2, normalization="sqrt")],
    "n17": lambda: [agg(17, 2)],
    "n32": lambda: [agg(32, 1)],
    "batch": lambda: [agg(7, 3), agg(7, 2), agg(7, 1)],
    "mixed_levels": lambda: [agg(3, 5), agg(7, 2), agg(9, 1)],
}


def solve(ps, solver, rows, monkeypatch, closure=False):
    env = dict(HEOMGB_ROWS=rows, HEOMGB_RESIDENT="0", HEOMGB_CLUSTER="0", HEOMGB_LOCAL="0", HEOMGB_SITES="0",
               HEOMGB_TCORE="0")
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    qs = [lh.from_params(p, precision="mixed") for p in ps]
    if closure:
        mlp = T.MLP(T.dims(ps[0])[0], 64, T.dims(ps[0])[1], seed=3)
        T.attach(qs[0], mlp)
    bs = lh.batch_solver(qs, lh.SOLVERS[solver]()) if len(qs) > 1 else lh.qme_solver(qs[0], lh.SOLVERS[solver]())
    rng = np.random.default_rng(1)
    rho = np.concatenate([p.rho0_ground().ravel() for p in ps])
    rho = rho + 0.01 * (rng.standard_normal(rho.shape) + 1j * rng.standard_normal(rho.shape))
    kw = dict(dt=0.5) if solver != "rkdp" else dict(dt=0.5, atol=1e-6, rtol=1e-6)
    bs.solve(rho, [0.0, 1.7, 4.0], None, kw)
    tune = bs.tuning()
    for t in tune.get("parts", [tune]):
        assert t["rows"] == (rows == "1")
    return rho


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("solver", ["rk4", "lsrk4", "rkdp"])
def test_rows_equal_diag(case, solver, monkeypatch):
    ps = CASES[case]()
    if solver == "rkdp" and len(ps) > 1:
        pytest.skip("batches step with fixed steps")
    want = solve(ps, solver, "0", monkeypatch)
    got = solve(ps, solver, "1", monkeypatch)
    if solver == "rkdp":
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
    else:
        assert np.array_equal(got, want)


def test_rows_with_closure(monkeypatch):
    ps = [agg(5, 2)]
    assert np.array_equal(solve(ps, "rk4", "1", monkeypatch, True), solve(ps, "rk4", "0", monkeypatch, True))
