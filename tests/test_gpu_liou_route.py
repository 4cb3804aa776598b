"""FP64 Liouville-space models on the Hilbert-space kernels: the states of
heom_liou and heom_ado equal those of the block-sparse products to FP64
rounding (1e-12 of the largest element after 20 steps; the mixed form, which
keeps the block-sparse kernel, checks the same propagation to 1e-6), and what
only heom_hilb offered is still refused."""
import dataclasses

import numpy as np
import pytest

import libheom_gb300 as lh
import oracle
from _cases import generic_case, projector_case
from libheom_gb300 import configs
from libheom_gb300 import terminator as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["liou", "ado"])
@pytest.mark.parametrize("case", ["projector", "generic", "generic_sqrt_col", "one_level_baths"])
def test_liouville_forms_match_the_port(form, case):
    p = {"projector": lambda: projector_case(depth=2),
         "generic": lambda: generic_case(),
         "generic_sqrt_col": lambda: dataclasses.replace(generic_case(), normalization="sqrt", order="col_major"),
         "one_level_baths": lambda: configs.aggregate_24site(n_sites=3, depth=1)}[case]()
    ref = oracle.Oracle("port").solve(p, p.rho0_ground(), [0.0, 0.2], solver="rk4", dt=0.01)[-1]
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-6)):
        qs = lh.qme_solver(lh.from_params(p, form=form, precision=precision), lh.rk4())
        rho = p.rho0_ground()
        qs.solve(rho, [0.0, 0.2], None, {"dt": 0.01})
        assert np.abs(rho - ref).max() <= tol * np.abs(ref).max()


def test_hilbert_only_features_stay_refused():
    p = configs.aggregate_24site(n_sites=3, depth=1)
    q = lh.from_params(p, form="liou")
    with pytest.raises(lh.HeomError):
        T.attach(q, T.MLP(T.dims(p)[0], 64, T.dims(p)[1]))
    with pytest.raises(lh.HeomError):
        lh.batch_solver([q], lh.rk4())
