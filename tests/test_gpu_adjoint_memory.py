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
