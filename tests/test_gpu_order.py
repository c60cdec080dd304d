"""The order by counting (cells counted, scanned and ranked by id) against the
radix sort, at the sizes where it changes: cells around the size above which
members are sorted instead of ranked, several such cells, cells that only the
last slots reach, one agent."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu

RANK_LIMIT = 4096


def _order(w, pos, by_count):
    with Engine(w.params) as eng:
        eng.set_option("incremental_sort", int(by_count))
        # one step first: the slot order is then not the id order
        eng.set_state(w.pos, w.fwd, w.acc)
        eng.step(w.dt)
        eng.set_state(pos, w.fwd, w.acc)
        eng.reorderSimData()
        out = eng.getHash() + eng.getCellRanges()
        eng.reorderSimData()  # the counters are clean for the next order
        again = eng.getHash() + eng.getCellRanges()
        assert eng.device_error() == 0
    for a, b in zip(out, again):
        assert np.array_equal(a, b)
    return out


@pytest.mark.parametrize("crowds", [(), (RANK_LIMIT,), (RANK_LIMIT + 1,), (5003, 4999), (11999,)])
@pytest.mark.parametrize("n", [12000, 12289])
def test_crowded_cells(crowds, n):
    w = workloads.plain(n=n, L=32.0)
    rng = np.random.default_rng(len(crowds) + n)
    pos = w.pos.copy()
    members = rng.permutation(n)
    for k, size in enumerate(crowds):
        who, members = members[:size], members[size:]
        pos[who, :3] = np.float32([4.0 * (7 - 3 * k), 28.0 - 8.0 * k, 28.0]) + 4 * rng.random((size, 3)).astype(np.float32) * 0.99
    for a, b in zip(_order(w, pos, True), _order(w, pos, False)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("sizes", [(1,), (2, 1, 31), (33, 1, 700), (5000, 3, 9000)])
def test_flocks_and_single_agents(sizes):
    params, P, W = [], [], []
    for k, n in enumerate(sizes):
        w = workloads.plain(n=n, L=workloads.cube_for(n), seed=k)
        params += w.params
        P.append(w.pos)
        W.append(w.fwd)
    w.params, w.pos, w.fwd = params, np.concatenate(P), np.concatenate(W)
    w.acc = np.zeros_like(w.pos)
    for a, b in zip(_order(w, w.pos, True), _order(w, w.pos, False)):
        assert np.array_equal(a, b)
