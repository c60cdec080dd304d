"""The backward over the tape the forward kept, against the one that computes
the checkpoint segments again: the same bits, with segments that divide the
horizon or not, one step, several flocks, obstacles, a horizon that grows or
shrinks between calls, and state changed between forward and backward."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _workload(name):
    if name == "one":
        return workloads.adjoint(n=3001, L=48.0)
    return workloads.fitting(num_flocks=5, lo=200, hi=900, obstacles=7)


def _run(w, checkpoints, horizons, every, disturb=False):
    rng = np.random.default_rng(1)
    target = w.pos.copy()
    target[:, :3] += rng.normal(0, 1, (w.num_agents, 3)).astype(np.float32)
    out = []
    with Engine(w.params) as eng:
        eng.set_option("adjoint_checkpoints", checkpoints)
        for T in horizons:
            eng.set_state(w.pos, w.fwd, w.acc)
            loss = eng.adjoint_forward(target, T, every, w.dt)
            final = eng.get_state(features=False)[:3]
            if disturb:
                eng.set_state(w.fwd, w.fwd, w.acc)
                eng.step(w.dt, 2)
            for _ in range(2):
                g = eng.adjoint_backward()
                out += [loss, *final, *(g[k] for k in sorted(g)), *eng.get_state(features=False)[:3]]
    return out


@pytest.mark.parametrize("name", ["one", "fitting"])
@pytest.mark.parametrize("horizons,every", [((1,), 1), ((10,), 5), ((7,), 3), ((4, 9, 6), 4)])
def test_whole_tape_equals_recompute(name, horizons, every):
    w = _workload(name)
    for a, b in zip(_run(w, 0, horizons, every), _run(w, 1, horizons, every)):
        assert np.array_equal(a, b, equal_nan=True)


def test_state_changed_before_the_backward():
    w = _workload("one")
    for a, b in zip(_run(w, 0, (6,), 2, disturb=True), _run(w, 1, (6,), 2)):
        assert np.array_equal(a, b, equal_nan=True)


def test_mode_switched_between_calls():
    w = _workload("one")
    with Engine(w.params) as eng:
        got = []
        for mode in (0, 1, 0, 1):
            eng.set_option("adjoint_checkpoints", mode)
            eng.set_state(w.pos, w.fwd, w.acc)
            eng.adjoint_forward(w.pos, 8, 3, w.dt)
            got.append(eng.adjoint_backward())
    for g in got[1:]:
        for k in g:
            assert np.array_equal(g[k], got[0][k], equal_nan=True)
