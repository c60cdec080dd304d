"""The number of agents a warp of the cooperative scans takes follows the
engine's size (32, or fewer when that many warps would leave the GPU part
empty): one step at the sizes around each change, with a remainder in the last
warp, against the FP32 oracle, bit for bit."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu

# 148 SMs x 32 resident warps = 4736 warps of 4, 8, 16 agents; other residencies
# change at other sizes of the same list
SIZES = [1, 5, 131, 9472, 9473, 18944, 18945, 37889, 75777]


def _same(a, b):
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)])


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kernel", ["flock", "two_pass", "school"])
def test_step_at_the_edges(n, kernel):
    from oracle import oracle as o
    L = workloads.cube_for(n)
    if kernel == "school":
        w = workloads.schooling(n=n, L=L)
    else:
        w = workloads.plain(n=n, L=L, M=12)
    with Engine(w.params) as eng:
        eng.set_option("two_pass", int(kernel == "two_pass"))
        eng.record_lists(True)
        eng.set_state(w.pos, w.fwd, w.acc)
        eng.step(w.dt)
        pos, fwd, acc, _ = eng.get_state(features=False)
        fused = eng.getNeighborLists()
        eng.set_state(w.pos, w.fwd, w.acc)
        eng.reorderSimData()
        eng.computeNeighborhoods()
        staged = eng.getNeighborLists()
    r = o.step(w.params, w.pos, w.fwd, w.acc, dt=w.dt, mode=0, random_step=1)
    for got, want in ((pos, r["pos"]), (fwd, r["fwd"]), (acc, r["acc"])):
        _same(got, want)
    used = np.arange(fused.shape[1])[None, :] <= r["lists"][:, :1]
    for lists in (fused, staged):
        assert np.array_equal(lists[used], r["lists"][used])
