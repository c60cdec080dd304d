"""The standalone sort's input loads: 16-byte aligned or only 8, odd counts, and
counts around the histogram's unrolled stride (4 * 592 blocks * 256 threads, two
pairs a load), against a stable host sort."""
import numpy as np
import pytest

from behavert_b200 import radix_sort_pairs, radix_sort_scratch_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4097, 303105, 1212416, 1212419])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("bits", [7, 18])
def test_alignment_and_tails(n, offset, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    pairs = np.stack([rng.integers(0, 1 << bits, n), np.arange(n)], axis=1).astype(np.int32)
    buf = torch.empty((n + 1, 2), dtype=torch.int32, device="cuda")
    src = buf[offset:offset + n]
    src.copy_(torch.from_numpy(pairs))
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    scratch = torch.full((radix_sort_scratch_bytes(n, bits),), 0xAB, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    radix_sort_pairs(src, out, n, bits, scratch)
    assert np.array_equal(out.cpu().numpy(), pairs[np.argsort(pairs[:, 0], kind="stable")])
