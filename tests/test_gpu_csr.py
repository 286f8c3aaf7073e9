"""Edge sort at the edges of its branches: buckets of 31 to 130 edges (register sorts of 32, 64 and
128 keys, and beyond), with the destinations rising from edge to edge and not, against the host
statement of the order."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["sorted", "dst_only", "src_first", "random", "last_pair_swapped"])
@pytest.mark.parametrize("degree", [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130])
def test_bucket_sizes_and_input_orders(degree, order):
    from zippel_b200.graph import EdgeGraph, csr_reference
    rng = np.random.default_rng(degree)
    n = 150
    # node i receives from and sends to the `degree` nodes around it, some pairs twice; ragged at the end
    dst = np.repeat(np.arange(n), degree)
    src = (dst + np.tile(np.arange(degree) // 2 * 2, n)) % n
    keep = (dst < n - 7) | (rng.random(dst.size) < 0.7)
    src, dst = src[keep], dst[keep]
    perm = {"sorted": lambda: np.lexsort((src, dst)),
            "dst_only": lambda: np.lexsort((rng.random(src.size), dst)),
            "src_first": lambda: np.lexsort((dst, src)),
            "random": lambda: rng.permutation(src.size),
            "last_pair_swapped": lambda: np.concatenate(
                [np.lexsort((src, dst))[1:], np.lexsort((src, dst))[:1]])}[order]()
    ei = np.stack([src[perm], dst[perm]]).astype(np.int64)
    want = csr_reference(ei, n)
    g = EdgeGraph.build(torch.from_numpy(ei).cuda(), n)
    for key, value in want.items():
        assert np.array_equal(getattr(g, key).cpu().numpy(), value), key


@pytest.mark.parametrize("n,degree", [(64, 64), (65, 63), (128, 32)])
def test_recorded_sorts_on_either_side_of_the_one_block_line(n, degree):
    from zippel_b200.graph import EdgeGraph, csr_reference
    rng = np.random.default_rng(n)
    edges = [rng.integers(0, n, (2, n * degree)) for _ in range(2)]
    ei = torch.from_numpy(edges[0]).cuda()
    EdgeGraph.build(ei, n)
    recorded = torch.cuda.CUDAGraph()
    with torch.cuda.graph(recorded):
        g = EdgeGraph.build(ei, n, validate=False)
    for e in edges:
        ei.copy_(torch.from_numpy(e))
        recorded.replay()
        for key, value in csr_reference(e, n).items():
            assert np.array_equal(getattr(g, key).cpu().numpy(), value), key
