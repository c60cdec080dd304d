"""Crowded cells in the order by counting: the cells that are sorted instead of
ranked, alone and by all blocks, against the radix sort; their time; and a wait of
theirs that runs out."""
import time

import numpy as np
import pytest

from behavert_b200 import BrtError, Engine, workloads
from behavert_b200 import _abi

pytestmark = pytest.mark.gpu

RANK_LIMIT = 512


def _giant_limit(n):
    return max(RANK_LIMIT, n // 256)


def _crowded(n, crowds, L=64.0, seed=0):
    """n agents in a cube of 16 x 16 x 16 cells, crowds[k] of them in cell k of a
    scattered sequence, the rest spread over all cells."""
    w = workloads.plain(n=n, L=L)
    rng = np.random.default_rng(seed)
    pos = w.pos.copy()
    members = rng.permutation(n)
    cells = rng.permutation(int(L / 4.0) ** 3)
    G = int(L / 4.0)
    for k, size in enumerate(crowds):
        who, members = members[:size], members[size:]
        c = int(cells[k])
        corner = np.float32([4.0 * (c % G), 4.0 * (c // G % G), 4.0 * (c // (G * G))])
        pos[who, :3] = corner + np.float32(3.9) * rng.random((size, 3)).astype(np.float32)
    return w, pos


def _order(w, pos, by_count, warm):
    with Engine(w.params) as eng:
        eng.set_option("incremental_sort", int(by_count))
        if warm:  # a slot order that is not the id order
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


CASES = [
    (513, (513,)), (2048, (RANK_LIMIT + 1, RANK_LIMIT - 1, RANK_LIMIT)), (2049, (2049,)),
    (6000, (RANK_LIMIT + 1,) * 11), (40001, (40001,)), (40001, (20000, 19000)),
    # cells sorted by a block each beside cells sorted by all blocks
    (200_000, (_giant_limit(200_000),) * 40 + (_giant_limit(200_000) + 1,) * 40 + (RANK_LIMIT + 1,) * 40 + (30_000,)),
    # as many giant cells as there can be
    (200_000, (_giant_limit(200_000) + 1,) * 255),
    (140_000, (RANK_LIMIT + 1,) * 30 + (_giant_limit(140_000),) * 30),
]


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("n,crowds", CASES)
def test_order_of_crowds(n, crowds, warm):
    w, pos = _crowded(n, crowds, seed=n)
    for a, b in zip(_order(w, pos, True, warm), _order(w, pos, False, warm)):
        assert np.array_equal(a, b)


def test_steps_through_a_crowd():
    """A graph of steps in which agents leave and enter crowded cells."""
    w, pos = _crowded(30_000, (700, 9000, 513, 2000), seed=1)
    got = []
    for by_count in (1, 0):
        with Engine(w.params) as eng:
            eng.set_option("incremental_sort", by_count)
            eng.set_state(pos, w.fwd, w.acc)
            for _ in range(3):
                eng.step(0.7, 4)
            eng.sync()
            got.append(eng.get_state(features=False)[:3])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [513, 128 * 27, 128 * 27 + 1, 20_000])
def test_few_cells(n):
    """Worlds of 27 cells, on both sides of the mean above which the radix sort orders."""
    w = workloads.plain(n=n, L=12.0)
    for a, b in zip(_order(w, w.pos, True, True), _order(w, w.pos, False, True)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,crowds", [(1_000_000, (1_000_000,)), (1_000_000, (250_000, 4000, 4000, 700_000))])
def test_crowds_cost_no_cliff(n, crowds):
    """An order with crowds takes a few times the radix sort's time (it took 330 times)."""
    w, pos = _crowded(n, crowds, L=128.0)
    best = []
    for by_count in (1, 0):
        with Engine(w.params) as eng:
            eng.set_option("incremental_sort", by_count)
            eng.set_state(pos, w.fwd, w.acc)
            eng.reorderSimData()
            eng.sync()
            times = []
            for _ in range(5):
                t = time.perf_counter()
                for _ in range(3):
                    eng.reorderSimData()
                eng.sync()
                times.append(time.perf_counter() - t)
            best.append(min(times))
    assert best[0] < 20 * best[1], best


def test_a_wait_that_runs_out_is_reported():
    w, pos = _crowded(30_000, (12_000, 13_000), seed=2)
    with Engine(w.params) as eng:
        eng.set_state(pos, w.fwd, w.acc)
        eng.set_option("lookback_spin_limit", 2000)
        eng.set_option("lookback_stall_tile", 3)
        eng.reorderSimData()
        with pytest.raises(BrtError) as ei:
            eng.sync()
        assert ei.value.status == _abi.BRT_ERR_TIMEOUT
        eng.set_option("lookback_stall_tile", -1)
        eng.set_option("lookback_spin_limit", 1 << 21)
        eng.set_state(pos, w.fwd, w.acc)
        eng.reorderSimData()
        got = eng.getHash() + eng.getCellRanges()
        assert eng.device_error() == 0
    for a, b in zip(got, _order(w, pos, False, False)):
        assert np.array_equal(a, b)
