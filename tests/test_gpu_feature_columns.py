"""Flocks of one engine with different featuresCount: a flock computes with its
own columns, and the others (which state I/O carries too) move with their agents.
Against the FP32 oracle, bit for bit."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine
from oracle import oracle as o

pytestmark = pytest.mark.gpu


def _workload(counts, clustering, relax, seed=0):
    rng = np.random.default_rng(seed)
    params, P, W = [], [], []
    for k, F in enumerate(counts):
        n = (2500, 2100, 1300, 90)[k % 4]
        w = workloads.plain(n=n, L=24.0, M=11, seed=seed + k)
        p = w.params[0]
        p.featuresCount, p.featureRelaxRate = F, relax
        if clustering:
            p.clusteringForceParams[0], p.alignmentClusteringForceParams[0] = 1.0, 0.5
        params.append(p)
        P.append(w.pos)
        W.append(w.fwd)
    w.params, w.pos, w.fwd = params, np.concatenate(P), np.concatenate(W)
    w.acc = np.zeros_like(w.pos)
    w.feat = rng.random((len(w.pos), max(counts))).astype(np.float32) + np.float32(0.5)
    stats = np.tile(np.float32([0.2, 0.5, 0.8, 0.0]), (len(w.pos), 1))
    return w, stats


def _oracle(w, stats, steps):
    state = (w.pos, w.fwd, w.acc, w.feat, stats)
    for _ in range(steps):
        r = o.step(w.params, *state, dt=w.dt, mode=0)
        state = (r["pos"], r["fwd"], r["acc"], r["feat"], r["stats"])
    return state


def _check(eng, want):
    got = list(eng.get_state()) + [eng.get_similarity_stats()]
    for name, g, r in zip(("pos", "fwd", "acc", "feat", "stats"), got, want):
        assert np.array_equal(g, r, equal_nan=True), name


def _start(eng, w, stats):
    eng.set_state(w.pos, w.fwd, w.acc, w.feat)
    eng.set_similarity_stats(stats)


@pytest.mark.parametrize("counts", [(8, 0, 8), (3, 8, 5), (5,)])
def test_list_first_kernel(counts):
    w, stats = _workload(counts, True, 0.05)
    with Engine(w.params) as eng:
        eng.set_option("two_pass", 1)
        _start(eng, w, stats)
        eng.step(w.dt, 3)
        _check(eng, _oracle(w, stats, 3))


@pytest.mark.parametrize("counts", [(8, 0, 8), (3, 8, 5)])
def test_stages(counts):
    w, stats = _workload(counts, False, 0.05)
    with Engine(w.params) as eng:
        _start(eng, w, stats)
        for _ in range(3):
            eng.update_stagewise(w.dt)
        _check(eng, _oracle(w, stats, 3))


@pytest.mark.parametrize("counts", [(8, 0, 8), (3, 8), (3, 8, 5, 8), (9, 32, 16, 0), (1, 2, 1)])
@pytest.mark.parametrize("clustering,relax", [(False, 0.05), (True, 0.05), (True, 0.0)])
def test_single_pass_kernel(counts, clustering, relax):
    w, stats = _workload(counts, clustering, relax, seed=3)
    with Engine(w.params) as eng:
        _start(eng, w, stats)
        eng.step(w.dt, 3)
        _check(eng, _oracle(w, stats, 3))


@pytest.mark.parametrize("scan,walk,order", [(0, 0, 1), (0, 1, 1), (4, 0, 0), (5, 2, 0), (6, 0, 1), (6, 2, 1), (7, 2, 1)])
def test_other_scans_and_walks(scan, walk, order):
    w, stats = _workload((3, 8, 5, 0), False, 0.05, seed=4)
    with Engine(w.params) as eng:
        for key, value in (("scan_variant", scan), ("phase2_variant", walk), ("incremental_sort", order)):
            eng.set_option(key, value)
        _start(eng, w, stats)
        eng.step(w.dt, 3)
        _check(eng, _oracle(w, stats, 3))


def test_values_that_are_no_numbers_in_columns_of_no_flock():
    w, stats = _workload((3, 8, 5), True, 0.05, seed=5)
    w.feat[:2500, 3:] = np.float32(np.nan)
    w.feat[4600:, 5:] = np.float32(np.inf)
    for n_knn in (0, 1):
        for p in w.params:
            p.useKnn = n_knn
            if n_knn:
                p.clusteringForceParams[0] = p.alignmentClusteringForceParams[0] = 0.0
        with Engine(w.params) as eng:
            _start(eng, w, stats)
            eng.step(w.dt, 3)
            _check(eng, _oracle(w, stats, 3))
