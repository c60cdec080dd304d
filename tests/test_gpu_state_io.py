"""set_state / get_state through one launch: features whose count is or is not a
multiple of four, device pointers that are not 16-byte aligned, arrays left
out, and a permuted slot order, against the host path and the inputs."""
import numpy as np
import pytest

from behavert_b200 import workloads
from behavert_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features", [0, 1, 4, 6, 8, 32])
@pytest.mark.parametrize("n", [1, 33, 5000, (1 << 18) + 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_round_trip(features, n, offset):
    import torch
    w = workloads.large(n=n, L=workloads.cube_for(n), F=features, blobs=1)
    rng = np.random.default_rng(n + features)
    acc = rng.random((n, 4)).astype(np.float32)
    with Engine(w.params) as eng:
        eng.set_state(w.pos, w.fwd, acc, w.feat)
        eng.step(w.dt, 2)  # slots now in cell order
        dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (w.pos, w.fwd, acc)]
        feat = None
        if features:
            buf = torch.empty(n * features + offset, device="cuda")
            buf[offset:] = torch.from_numpy(w.feat).cuda().flatten()
            feat = buf[offset:].view(n, features)
        eng.set_state(*dev, feat)
        got = eng.get_state()
        want = [w.pos, w.fwd, acc] + ([w.feat] if features else [])
        out = [torch.full((n, 4), -1.0, device="cuda") for _ in range(3)]
        fout = torch.full((n * features + offset,), -1.0, device="cuda") if features else None
        torch.cuda.synchronize()
        eng.get_state_into(*out, fout[offset:].view(n, features) if features else None)
        eng.sync()
        dev_got = [x.cpu().numpy() for x in out] + ([fout[offset:].view(n, features).cpu().numpy()] if features else [])
        for a, b, c in zip(want, got, dev_got):
            ref = a.copy()
            if a is w.pos:
                ref[:, 3] = 1.0
            assert np.array_equal(ref, b) and np.array_equal(ref, c)
        # one array alone, the others untouched
        eng.set_state(fwd4=dev[2])
        pos2, fwd2, acc2, _ = eng.get_state(features=False)
        assert np.array_equal(fwd2, acc) and np.array_equal(acc2, acc) and np.array_equal(pos2[:, :3], w.pos[:, :3])
