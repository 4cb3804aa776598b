"""Cluster-resident fixed-step intervals (k_cluster: the ADOs of a bin of
instances dealt out to the CTAs of a thread-block cluster, neighbours read from
the owners' shared memory) against the per-stage kernels, for every cluster
size.  The arithmetic per element is the stage kernels', in their order, so the
states agree bit for bit: uneven instances with two and four levels, complex H
and sqrt normalisation, hierarchies smaller than the cluster, odd numbers of
levels, a clamped last step and two intervals without a callback between."""
import dataclasses

import numpy as np
import pytest

import libheom_gb300 as lh
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu


def complex_sqrt(depth):
    X = np.random.default_rng(5).uniform(-0.2, 0.2, (2, 2))
    p = configs.spin_boson(depth=depth)
    return dataclasses.replace(p, H=p.H + 1j * (X - X.T), normalization="sqrt")


CASES = {
    "two_level": lambda: ([configs.spin_boson(depth=7)], 0.005),
    "depth0_and_1": lambda: ([configs.spin_boson(depth=0), configs.spin_boson(depth=1)], 0.005),
    "sweep": lambda: (configs.batched_sweep()[:6] + configs.batched_sweep()[768:771], 0.005),
    "complex_sqrt_col": lambda: ([dataclasses.replace(complex_sqrt(d), order="col_major") for d in (4, 6)], 0.005),
    "filtered": lambda: ([dataclasses.replace(configs.spin_boson(depth=6), hrchy_filter=lambda i, d: i[0] <= 2)], 0.005),
    "five_sites": lambda: ([configs.aggregate_24site(n_sites=5, depth=2)], 0.5),
    "seven_sites": lambda: ([configs.exciton_7site(depth=2)], 0.5),
}


def solve(ps, solver, precision, dt, env, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    bs = lh.batch_solver([lh.from_params(p, precision=precision) for p in ps], lh.SOLVERS[solver]())
    tune = bs.tuning()
    for k in env:
        monkeypatch.delenv(k)
    rho = np.concatenate([p.rho0_ground().ravel() for p in ps])
    bs.solve(rho, [0.0, 17 * dt + 0.3 * dt, 30 * dt], None, {"dt": dt})
    return rho, tune.get("parts", [tune])


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("solver", ["rk4", "lsrk4"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_bit_identical_to_stage_kernels(case, solver, precision, monkeypatch):
    ps, dt = CASES[case]()
    off = dict(HEOMGB_CLUSTER="0", HEOMGB_LOCAL="0", HEOMGB_RESIDENT="0")
    ref, tune = solve(ps, solver, precision, dt, off, monkeypatch)
    assert not any(t["cluster"] for t in tune)
    ran = 0
    for size in (1, 2, 4, 8, 16):
        got, tune = solve(ps, solver, precision, dt, dict(HEOMGB_CLUSTER="1", HEOMGB_CLUSTER_SIZE=str(size)), monkeypatch)
        if all(t["cluster"] and t["cluster_size"] == size for t in tune):
            ran += 1
        assert np.all(np.isfinite(got))
        assert np.array_equal(got, ref)
    assert ran >= 2
