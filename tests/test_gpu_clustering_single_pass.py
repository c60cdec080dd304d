"""Clustering steering in the single-pass kernel against the list-first kernel
(option two_pass) and the FP32 oracle, bit for bit: feature counts around the
register widths, one of the two forces, with and without relaxation, flocks
without clustering or without features beside it, agents without neighbours,
coincident agents, obstacles."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _workload(F, coh, ali, relax, seed=0):
    rng = np.random.default_rng(seed)
    params, P, W = [], [], []
    for k, (n, L) in enumerate([(700, 24.0), (90, 40.0), (1500, 24.0), (33, 12.0)]):
        w = workloads.plain(n=n, L=L, M=11, seed=seed + k)
        p = w.params[0]
        p.featuresCount = F if k != 3 else 0
        p.featureRelaxRate = relax
        if k != 2:
            p.clusteringForceParams[0] = coh
            p.alignmentClusteringForceParams[0] = ali
        if k == 0:
            p.set_obstacles([[3.0, 4.0, 5.0, 3.0]])
            p.obstacleAvoidanceWeight = 2.0
            w.pos[5, :3] = w.pos[6, :3]
        params.append(p)
        P.append(w.pos)
        W.append(w.fwd)
    w.params, w.pos, w.fwd = params, np.concatenate(P), np.concatenate(W)
    w.acc = np.zeros_like(w.pos)
    w.feat = rng.random((len(w.pos), F)).astype(np.float32)
    stats = np.tile(np.float32([0.2, 0.5, 0.8, 0.0]), (len(w.pos), 1))
    return w, stats


def _run(w, stats, two_pass, steps):
    with Engine(w.params) as eng:
        eng.set_option("two_pass", two_pass)
        eng.record_lists(True)
        eng.set_state(w.pos, w.fwd, w.acc, w.feat)
        eng.set_similarity_stats(stats)
        eng.step(w.dt, steps)
        lists = eng.getNeighborLists()
        lists = np.where(np.arange(lists.shape[1])[None, :] <= lists[:, :1], lists, 0)
        return list(eng.get_state()) + [eng.get_similarity_stats(), lists]


@pytest.mark.parametrize("F", [1, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("coh,ali,relax", [(1.0, 0.5, 0.05), (0.7, 0.0, 0.0), (0.0, 1.2, 0.05)])
def test_single_pass_equals_two_pass(F, coh, ali, relax):
    w, stats = _workload(F, coh, ali, relax, seed=F)
    own = slice(0, len(w.pos) - 33)  # the last flock has no features: the list-first kernel does not move them
    for steps in (1, 4):
        a, b = _run(w, stats, 0, steps), _run(w, stats, 1, steps)
        a[3], b[3] = a[3][own], b[3][own]
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)


def test_against_the_oracle():
    from oracle import oracle as o
    w, stats = _workload(8, 1.0, 0.5, 0.05)
    pos, fwd, acc, feat, st, _ = _run(w, stats, 0, 1)
    r = o.step(w.params, w.pos, w.fwd, w.acc, w.feat, stats, dt=w.dt, mode=0)
    for got, want in ((pos, r["pos"]), (fwd, r["fwd"]), (acc, r["acc"]), (feat, r["feat"]), (st, r["stats"])):
        assert np.array_equal(got, want, equal_nan=True)
