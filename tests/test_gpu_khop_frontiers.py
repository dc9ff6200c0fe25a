"""k-hop with frontiers on both sides of the 64 vertices that a warp keeps in
shared memory, fanouts around a warp's 32 lanes and a random window's 128 draws,
and seeds without neighbors, standalone and in a batch with a seed's expansion
split over warps, against the oracle."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu

FANOUTS = [(1,), (1, 1, 1), (31, 2), (32, 3), (33, 2), (64, 2), (65, 2), (8, 8, 2), (13, 5, 3), (128, 1), (129, 2),
           (2, 200, 3), (4, 4, 4, 4), (1, 64, 2, 1)]


@pytest.mark.parametrize("mode", ["GT", "LE"])
@pytest.mark.parametrize("fanouts", FANOUTS)
def test_frontiers(oracle_mod, mode, fanouts):
    import torch
    d, _, _, _ = golden_graph("edge_cases")  # (has vertices without neighbors)
    prefix = os.path.join(d, mode)
    g, og = G.Graph(prefix, mode), oracle_mod.OracleGraph(prefix)
    seeds = np.random.default_rng(3).integers(0, g.n + 1, 77, dtype=np.uint32)
    refs, total = og.khop(mode, seeds, fanouts, 6)
    outs, e = g.khop(seeds, fanouts, 6)
    assert e == total
    for a, b in zip(outs, refs):
        np.testing.assert_array_equal(a, b)
    dev = torch.from_numpy(seeds.view(np.int32)).cuda()
    for obj in (g, g.csr()):
        for parts in (1, 2, 4):
            b = G.Batch(obj)
            hops = [torch.zeros(len(seeds), w, dtype=torch.int32, device="cuda") for w in G.hop_widths(fanouts)]
            count = torch.zeros(1, dtype=torch.int64, device="cuda")
            b.add_khop(dev, len(seeds), fanouts, 6, hops)
            b.set_config(warps_per_vertex=parts)
            b.run(total=count)
            torch.cuda.synchronize()
            assert int(count) == total
            for h, r in zip(hops, refs):
                np.testing.assert_array_equal(h.cpu().numpy().view(np.uint32), r)
