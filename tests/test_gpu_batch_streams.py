"""Batches of both levels: plain runs on several streams, under capture and beside
one; the count of their kernels."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


def _mixed(oracle_mod):
    """A batch of a multi-RW job (block-level) and a walk job (warp-level), its outputs and what they should be."""
    import torch
    prefix = os.path.join(golden_graph("rmat_s10_e8")[0], "LE")
    g, og = G.Graph(prefix, "LE"), oracle_mod.OracleGraph(prefix)
    rng = np.random.default_rng(5)
    roots, starts = rng.integers(0, g.n, (5, 40), dtype=np.uint32), rng.integers(0, g.n, 300, dtype=np.uint32)
    dev = [torch.from_numpy(x.view(np.int32)).cuda() for x in (roots, starts)]
    src, dst = (torch.zeros(5, 600, dtype=torch.int32, device="cuda") for _ in range(2))
    paths = torch.zeros(300, 21, dtype=torch.int32, device="cuda")
    b = G.Batch(g)
    b.add_mrw(dev[0], 5, 40, 600, 1, src, dst)
    b.add_rw(dev[1], 300, 20, 2, paths)
    b.keep = dev
    rs, rd, re, _ = og.mrw("LE", roots, 600, 1)
    return b, [(src, rs), (dst, rd), (dev[0], re), (paths, og.rw("LE", starts, 20, 2)[0])]


def _check(outs):
    import torch
    torch.cuda.synchronize()
    for got, ref in outs:
        np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), ref)
        got.fill_(-7)
    torch.cuda.synchronize()


def test_plain_run_beside_its_own_capture(oracle_mod):
    import torch
    b, outs = _mixed(oracle_mod)
    b.set_config(use_graph=2)
    b.run()  # builds
    _check(outs)
    graph, stream, other = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        b.run(stream=stream)
        b.run(stream=other)  # not captured: runs now
    _check(outs)
    graph.replay()
    _check(outs)
    b.set_config(use_graph=1)
    b.run(stream=other)
    _check(outs)


@pytest.mark.parametrize("use_graph", [1, 2])
def test_every_kernel_of_a_run_is_counted(oracle_mod, use_graph):
    import torch
    b, _ = _mixed(oracle_mod)
    one = G.Batch(b._g)
    paths = torch.zeros(300, 21, dtype=torch.int32, device="cuda")
    one.add_rw(b.keep[1], 300, 20, 2, paths)
    for batch, kernels in ((b, 2), (one, 1), (G.Batch(b._g), 0)):
        batch.set_config(use_graph=use_graph)
        batch.run()
        before = G.launch_count()
        for _ in range(3):
            batch.run()
        assert G.launch_count() - before == 3 * kernels
    torch.cuda.synchronize()
