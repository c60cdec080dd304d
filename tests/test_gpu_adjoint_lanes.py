"""The lanes an agent of the reverse kernels follow the engine's size (4, 2 or 1
a thread group in the emit kernel) and maxNeighbors (4 or 8 in the gather):
gradients at the sizes around each change, with a remainder in the last group,
against the FP64 reverse linearised at the GPU's own trajectory.  The tolerance
is the adjoint's 1e-4 bar."""
import numpy as np
import pytest

from behavert_b200 import workloads
from tests.test_gpu_adjoint import DT, REL, _counts_per_agent, _L_per_agent, _min_image, _oracle, _run, _vel_grad

pytestmark = pytest.mark.gpu

# 148 SMs x 6 blocks of 128 threads: 28,416 agents of 4 lanes, 56,832 of 2
SIZES = [3, 28416, 28417, 56833]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("M", [16, 17, 32])
def test_gradients_at_the_edges(n, M):
    o = _oracle()
    T = 3
    wl = workloads.adjoint(n=n, L=workloads.cube_for(n), M=M)
    rng = np.random.default_rng(n + M)
    target = wl.pos.copy()
    target[:, :3] += rng.normal(0, 1, (n, 3)).astype(np.float32)
    eng, loss, g, (lists, flags) = _run(wl, target, T, 2)
    states = eng.adjoint_tape_states(T)
    final = eng.get_state(features=False)[0]
    eng.close()
    d = _min_image(final[:, :3].astype(np.float64) - target[:, :3], _L_per_agent(wl.params)[:, None])
    gT = np.zeros((n, 4))
    gT[:, :3] = 2.0 * d / _counts_per_agent(wl.params)[:, None]
    p = wl.params[0]
    w = np.array([[p.separationParams[0], p.alignmentParams[0], p.cohesionParams[0]]])
    ref = o.frozen_reverse_at(wl.params, states, lists, gT, weights=w, flags=flags, dt=DT)
    ref["vel"] = _vel_grad(ref, wl.fwd.astype(np.float64))
    assert abs(loss[0] - np.mean(np.sum(d * d, axis=1))) <= 1e-9 * loss[0]
    for got, want in ((g["pos"], ref["pos"]), (g["vel"], ref["vel"]), (g["weights"], ref["weights"])):
        got, want = np.asarray(got)[:, :3], np.asarray(want, np.float64)[:, :3]
        assert np.linalg.norm(got - want) <= REL * np.linalg.norm(want)
