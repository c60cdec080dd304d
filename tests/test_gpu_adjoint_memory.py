"""The adjoint's storage: a forward whose storage does not fit fails as a whole."""
import numpy as np
import pytest

from behavert_b200 import BrtError, workloads
from behavert_b200 import _abi
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu

HORIZON = 200_000_000  # a tape of 28 TB for the 1,001 agents here


def test_backward_after_a_forward_that_did_not_fit():
    w = workloads.adjoint(n=1001, L=32.0)
    with Engine(w.params) as eng:
        eng.set_state(w.pos, w.fwd, w.acc)
        loss = eng.adjoint_forward(w.pos, 6, 3, w.dt)
        g = eng.adjoint_backward()
        eng.set_state(w.pos, w.fwd, w.acc)
        with pytest.raises(BrtError) as ei:
            eng.adjoint_forward(w.pos, HORIZON, HORIZON, w.dt)
        assert ei.value.status == _abi.BRT_ERR_CUDA
        # the first forward's tape may be gone: nothing is left to go back through
        with pytest.raises(BrtError) as ei:
            eng.adjoint_backward()
        assert ei.value.status == _abi.BRT_ERR_STATE
        # and the error is not reported a second time by what runs next
        eng.set_state(w.pos, w.fwd, w.acc)
        eng.step(w.dt, 1)
        eng.sync()
        eng.set_state(w.pos, w.fwd, w.acc)
        assert np.array_equal(eng.adjoint_forward(w.pos, 6, 3, w.dt), loss)
        again = eng.adjoint_backward()
        for k in g:
            assert np.array_equal(g[k], again[k])


def _grown(eng, w, T, every):
    """Device bytes that a forward takes for good."""
    import torch
    eng.set_state(w.pos, w.fwd, w.acc)
    eng.sync()
    before = torch.cuda.mem_get_info()[0]
    eng.adjoint_forward(w.pos, T, every, w.dt)
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("T,every", [(400, 10), (300, 3), (50, 5)])
def test_storage_follows_the_checkpoint_distance(T, every):
    w = workloads.adjoint(n=40_000, L=80.0)
    grown = []
    for checkpoints in (1, 0):
        with Engine(w.params) as eng:
            eng.step(w.dt, 1)
            eng.set_option("adjoint_checkpoints", checkpoints)
            grown.append(_grown(eng, w, T, every))
            eng.adjoint_backward()
    slack = 64 << 20  # allocation granularity, the graphs
    assert grown[1] <= 3 * grown[0] + slack


def test_all_engines_share_the_bound():
    import torch
    w = workloads.adjoint(n=1_000_000, L=252.0)
    tape = 50 * w.num_agents * (72 + 4 * (w.params[0].maxNeighbors + 1))
    bound = torch.cuda.mem_get_info()[1] // 8
    assert 2 * tape < bound < 6 * tape
    engines = [Engine(w.params) for _ in range(6)]
    try:
        grown = [_grown(eng, w, 50, 10) for eng in engines]
        whole = [x > grown[-1] + tape // 4 for x in grown]
        assert whole == [True] * (bound // tape) + [False] * (6 - bound // tape)
        # one given back makes room for another
        free = torch.cuda.mem_get_info()[0]
        engines[0].set_option("adjoint_checkpoints", 1)
        assert torch.cuda.mem_get_info()[0] - free >= tape * 9 // 10
        with pytest.raises(BrtError):
            engines[0].adjoint_backward()
        assert _grown(engines[-1], w, 50, 10) > tape // 4
    finally:
        for eng in engines:
            eng.close()
