"""The FP64 stages on the tensor cores are taken by a rule on sizes, so that a
model has the same bits in every run, and not by the tile search's timing."""
import pytest

import libheom_gb300 as lh
from test_gpu_split import agg

pytestmark = pytest.mark.gpu

CASES = [(4, 5, False), (8, 4, False), (10, 2, False), (10, 3, True), (12, 2, False), (15, 2, True), (16, 1, False),
         (16, 2, True), (24, 1, True), (32, 1, True)]


@pytest.mark.parametrize("n,depth,taken", CASES)
@pytest.mark.parametrize("solver", ["rk4", "lsrk4", "rkdp"])
def test_rule(n, depth, taken, solver, monkeypatch, capfd):
    for k, v in dict(HEOMGB_RESIDENT="0", HEOMGB_CLUSTER="0", HEOMGB_LOCAL="0", HEOMGB_TUNE_LOG="1").items():
        monkeypatch.setenv(k, v)
    s = lh.qme_solver(lh.from_params(agg(n, depth), precision="fp64"), lh.SOLVERS[solver]())
    assert s.tuning()["split"] == taken
    log = capfd.readouterr().err
    assert ("split" in log) == taken and ("heomgb tune: diag" in log) == (not taken)


@pytest.mark.parametrize("pair,taken", [(((12, 2), (12, 2), (12, 2)), True), (((12, 2), (8, 2), (24, 1)), False)])
def test_rule_counts_a_batch_together(pair, taken, monkeypatch):
    for k in ("HEOMGB_CLUSTER", "HEOMGB_LOCAL"):
        monkeypatch.setenv(k, "0")
    s = lh.batch_solver([lh.from_params(agg(n, d), precision="fp64") for n, d in pair], lh.rk4())
    assert s.tuning()["split"] == taken
