"""A batch of two sub-batches of which one fails: rho is left with every instance
at the last output time that all of them reached, and the error is raised.
The sub-batch solvers are stand-ins on the host (adding 1 per interval)."""
import numpy as np
import pytest

import libheom_gb300 as lh


class Part:
    def __init__(self, base, fails_at=None):
        self.base, self.fails_at, self.rho = base, fails_at, None

    def _advance(self, rho, t_list):
        for t0, t1 in zip(t_list[:-1], t_list[1:]):
            if self.fails_at is not None and t1 > self.fails_at:
                raise RuntimeError("no further")
            rho += 1

    def solve(self, rho, t_list, callback, kwargs):
        assert callback is None
        self._advance(rho, t_list)

    def solve_device(self, ptr, t_list, callback, kwargs):
        self._advance(self.rho, t_list)

    def stats(self):
        return dict(rhs=1, attempts=1, accepted=1)


class Solver:
    pass


def batch(parts, solver):
    bs = lh.batch_solver.__new__(lh.batch_solver)
    bs.solver = solver
    bs._off = np.array([0, 2, 4])
    bs._parts = [(p, [i], [(2 * i, 2 * i + 2)], True) for i, p in enumerate(parts)]
    return bs


TIMES = [0.0, 1.0, 2.0, 3.0, 4.0]


@pytest.mark.parametrize("kind", [Solver, lh.rkdp])
@pytest.mark.parametrize("with_callback", [False, True])
@pytest.mark.parametrize("failing", [0, 1])
def test_a_failed_sub_batch_leaves_the_last_common_time(kind, with_callback, failing):
    solver = kind.__new__(kind)
    parts = [Part(0), Part(0)]
    parts[failing].fails_at = 2.5
    rho, seen = np.zeros(4, dtype=np.complex128), []
    with pytest.raises(RuntimeError, match="no further"):
        batch(parts, solver).solve(rho, TIMES, seen.append if with_callback else None, None)
    assert np.array_equal(rho, np.full(4, 2.0))
    assert seen == (TIMES[:3] if with_callback else [])


@pytest.mark.parametrize("kind", [Solver, lh.rkdp])
def test_a_good_solve_reaches_the_end(kind):
    bs = batch([Part(0), Part(0)], kind.__new__(kind))
    rho = np.zeros(4, dtype=np.complex128)
    bs.solve(rho, TIMES, None, None)
    assert np.array_equal(rho, np.full(4, 4.0))
    assert bs._counts[0]["rhs"] == (1 if kind is Solver else 4)


@pytest.mark.parametrize("failing", [0, 1])
def test_device_states_are_at_most_one_interval_apart(failing):
    parts = [Part(0), Part(0)]
    for p in parts:
        p.rho = np.zeros(2)
    parts[failing].fails_at = 2.5
    with pytest.raises(RuntimeError, match="no further"):
        batch(parts, Solver()).solve_device(0, TIMES, None, None)
    assert parts[failing].rho[0] == 2.0 and parts[1 - failing].rho[0] in (2.0, 3.0)
