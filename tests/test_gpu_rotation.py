"""FP64 models whose couplings are dense but share an eigenbasis: fixed-step
solves run there on the diagonal-coupling kernels, and their states equal the
port's to FP64 rounding (1e-12 of the largest element after 20 steps: about
100 products of n terms), with callbacks between intervals, every form, both
orders, and blocks of 1 to 13 levels; Dormand-Prince and couplings without a
common basis keep the general kernel."""
import dataclasses

import numpy as np
import pytest

import libheom_gb300 as lh
import oracle
from _cases import _herm, generic_case
from libheom_gb300 import configs

pytestmark = pytest.mark.gpu


def _commuting(n, depth, seed, **kw):
    """Two baths, dense Hermitian V of one eigenbasis (repeated eigenvalues
    among them), complex H, nonzero s_delta, dense S and A."""
    rng = np.random.default_rng(seed)
    W = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    V0 = (W * np.round(rng.standard_normal(n))) @ W.conj().T
    V1 = (W * (rng.standard_normal(n) + 0.1)) @ W.conj().T
    V = [(v + v.conj().T) / 2 for v in (V0 + V1, V1)]
    return dataclasses.replace(generic_case(), H=_herm(rng, n), V=V, s_delta=[0.05, 0.02], max_depth=depth, **kw)


def _case(name):
    if name == "spin_boson_x":
        return configs.spin_boson(depth=6, coupling="x")
    if name == "not_commuting":
        rng = np.random.default_rng(3)
        return dataclasses.replace(generic_case(), V=[_herm(rng, 3), _herm(rng, 3)])
    n, depth = {"n1": (1, 2), "n3": (3, 3), "n5_sqrt_col": (5, 3), "n13": (13, 2)}[name]
    kw = dict(normalization="sqrt", order="col_major") if name == "n5_sqrt_col" else {}
    return _commuting(n, depth, 11 + n, **kw)


@pytest.mark.parametrize("form", ["hilb", "liou", "ado"])
@pytest.mark.parametrize("name", ["spin_boson_x", "n1", "n3", "n5_sqrt_col", "n13", "not_commuting"])
@pytest.mark.parametrize("scheme", ["rk4", "lsrk4", "rkdp"])
def test_dense_couplings_match_the_port(form, name, scheme):
    p = _case(name)
    if scheme == "rkdp" and form != "hilb":
        pytest.skip("the forms share the adaptive solve's kernel")
    rng = np.random.default_rng(2)
    shape = p.rho0_ground().shape
    rho0 = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    rho0[1:] *= 0.01
    kw = dict(dt=0.01) if scheme != "rkdp" else dict(dt=0.01, atol=1e-9, rtol=1e-9)
    ts = [0.0, 0.05, 0.2]
    ref = oracle.Oracle("port").solve(p, rho0.copy(), ts, solver=scheme, **kw)
    make = {"rk4": lh.rk4, "lsrk4": lh.lsrk4, "rkdp": lh.rkdp}[scheme]
    qs = lh.qme_solver(lh.from_params(p, form=form, precision="fp64"), make())
    seen, rho = [], rho0.copy()
    qs.solve(rho, ts, lambda t: seen.append(rho.copy()), kw)
    tol = 1e-12 if scheme != "rkdp" else 1e-9
    for got, want in zip(seen, ref):
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
    again = rho0.copy()  # without a callback the state stays on the device between intervals
    qs.solve(again, ts, None, kw)
    assert np.abs(again - ref[-1]).max() <= tol * np.abs(ref[-1]).max()
