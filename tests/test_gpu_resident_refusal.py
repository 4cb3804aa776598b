"""A resident plan that the device refuses at the launch (answered on the host):
the solve goes on with the stage kernels, the next one searches their shape,
and all give the resident plan's states to rounding (Dormand-Prince: to its
tolerance, 1e-8 an attempt)."""
import numpy as np
import pytest

import libheom_gb300 as lh
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("solver", ["rk4", "rkdp"])
def test_refused_resident_plan(solver, precision, monkeypatch, capfd):
    monkeypatch.setenv("HEOMGB_CLUSTER", "0")
    monkeypatch.setenv("HEOMGB_LOCAL", "0")
    p = configs.exciton_7site(depth=3)
    kw = dict(dt=0.5) if solver == "rk4" else dict(dt=0.5, atol=1e-8, rtol=1e-8)

    def make():
        return lh.qme_solver(lh.from_params(p, precision=precision), lh.SOLVERS[solver]())

    def run(s):
        rho = p.rho0_ground()
        s.solve(rho, [0.0, 4.0, 10.0], None, kw)
        return rho

    want = run(make())
    tol = (1e-12 if precision == "fp64" else 1e-6) if solver == "rk4" else 1e-6  # of the largest element
    s = make()
    assert s.tuning()["resident"]
    monkeypatch.setenv("HEOMGB_FAULT_COOPERATIVE", "1")
    monkeypatch.setenv("HEOMGB_TUNE_LOG", "1")
    for searched in (False, True, False):  # the refused solve, the one that searches, one on its graphs
        capfd.readouterr()
        assert np.abs(run(s) - want).max() <= tol * np.abs(want).max()
        assert not s.tuning()["resident"]
        assert ("heomgb tune" in capfd.readouterr().err) == searched
    monkeypatch.delenv("HEOMGB_FAULT_COOPERATIVE")
    assert np.abs(run(s) - want).max() <= tol * np.abs(want).max()
