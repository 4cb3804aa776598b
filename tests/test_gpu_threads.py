"""Solvers on two host threads that launch the same kernel with shared memory of
different sizes: neither launch fails and neither state changes."""
import threading

import numpy as np
import pytest

import libheom_gb300 as lh
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("env", [dict(HEOMGB_CLUSTER="1", HEOMGB_CLUSTER_SIZE="1"),
                                 dict(HEOMGB_CLUSTER="0", HEOMGB_LOCAL="1"),
                                 dict(HEOMGB_CLUSTER="0", HEOMGB_LOCAL="0")], ids=["cluster", "local", "resident"])
def test_solvers_of_one_kernel_on_two_threads(env, precision, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    jobs = []
    for depth in (8, 7) if precision == "fp64" else (11, 10):  # both above the default limit of 48 KB
        p = configs.spin_boson(depth=depth)
        s = lh.qme_solver(lh.from_params(p, precision=precision), lh.rk4())
        want = p.rho0_ground()
        s.solve(want, [0.0, 0.005], None, dict(dt=0.005))
        jobs.append((s, p.rho0_ground(), want))
    failed = []
    go = threading.Barrier(2)

    def work(s, rho0, want):
        try:
            go.wait(60)
            for _ in range(15000):
                rho = rho0.copy()
                s.solve(rho, [0.0, 0.005], None, dict(dt=0.005))
                assert np.array_equal(rho, want)
        except BaseException as e:  # noqa: BLE001  (a failed assertion too)
            failed.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
