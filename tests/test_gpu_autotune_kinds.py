"""The autotuner tries the options that the engine's kernel has, and only those:
clustering and kNN engines run the flock kernel, mixed ones the list-first kernel."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _workload(kind):
    w = workloads.plain(n=6000, L=48.0, M=40 if kind == "long_knn" else 16)
    p = w.params[0]
    if kind in ("clustering", "mixed"):
        p.featuresCount = 5
        p.clusteringForceParams[0] = 1.0
        w.feat = np.random.default_rng(0).random((6000, 5)).astype(np.float32)
    p.useKnn = int(kind in ("knn", "long_knn", "mixed", "knn_features"))
    if kind == "knn_features":
        p.featuresCount, p.featureRelaxRate = 5, 0.05
        w.feat = np.random.default_rng(0).random((6000, 5)).astype(np.float32)
    if kind == "school":
        p.schooling.mode = 1
    return w


@pytest.mark.parametrize("kind,tried", [
    ("plain", {"block_size/scan0/walk0", "block_size/scan5/walk0", "scan6/walk0", "registers"}),
    ("clustering", {"block_size"}),
    ("knn", {"block_size/walk0", "registers"}),
    ("knn_features", {"block_size/walk0", "block_size/walk2", "registers"}),
    ("long_knn", set()), ("mixed", set()), ("school", set()),
])
def test_options_tried(kind, tried):
    w = _workload(kind)
    with Engine(w.params) as eng:
        eng.set_state(w.pos, w.fwd, w.acc, w.feat)
        before = eng.get_state()
        report = eng.autotune(w.dt, steps=2)
        for a, b in zip(before, eng.get_state()):
            assert a is None or np.array_equal(a, b)
        names = {k for t in report["trials"] for k in t if k != "ms_per_step"} - {"sort_digit_bits", "incremental_sort"}
        if kind == "plain":
            assert tried <= names
        else:
            assert names == tried
        eng.step(w.dt, 3)
        tuned = eng.get_state()
    with Engine(w.params) as eng:
        eng.set_state(w.pos, w.fwd, w.acc, w.feat)
        eng.step(w.dt, 3)
        for a, b in zip(tuned, eng.get_state()):
            assert a is None or np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n,orders", [(27 * 128, 2), (27 * 128 + 1, 1)])
def test_orders_tried(n, orders):
    w = workloads.plain(n=n, L=12.0)
    with Engine(w.params) as eng:
        eng.set_state(w.pos, w.fwd, w.acc)
        report = eng.autotune(w.dt, steps=2)
        assert sum("incremental_sort" in t for t in report["trials"]) == orders
        assert report["ms_per_step"] > 0
