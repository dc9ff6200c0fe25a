"""Multi-RW at the edges of its kernels, against the oracle: one walker, walker
counts around the 8 lanes of a group and the 256 up to which groups are used,
sample counts that leave groups of a warp without a sample, step counts around a
warp's 32 and a group's 8, and chains on both sides of the block-per-sample
rule."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("select", [G.SELECT_UNIFORM, G.SELECT_DEGREE])
@pytest.mark.parametrize("samples,walkers,steps", [
    (1, 1, 1), (3, 1, 70), (5, 7, 33), (4, 8, 8), (33, 9, 31), (7, 255, 40), (6, 256, 41), (6, 257, 41),
    (2, 2000, 65), (1, 13000, 50), (2, 80, 511), (2, 80, 512), (700, 80, 513)])
def test_multi_rw_shapes(oracle_mod, select, samples, walkers, steps):
    d, _, _, _ = golden_graph("edge_cases")  # (has vertices without neighbors)
    prefix = os.path.join(d, "LE")
    g, og = G.Graph(prefix, "LE"), oracle_mod.OracleGraph(prefix)
    roots = np.random.default_rng(walkers).integers(0, g.n + 1, (samples, walkers), dtype=np.uint32)
    src, dst, end, e = g.mrw(roots, steps, 9, select)
    ref = og.mrw("LE", roots, steps, 9, select)
    for a, b in zip((src, dst, end, e), ref):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("samples,walkers,steps", [
    (3, 1, 40), (300, 80, 100), (2, 512, 600), (3, 513, 601), (1, 2000, 10000), (1, 50, 33000), (2, 7, 70000)])
def test_continuous_time_shapes(oracle_mod, samples, walkers, steps):
    """Continuous time on both sides of 512 walkers (the wide kernel) and of the
    event count from which the radix sort replaces the buckets."""
    d, _, _, _ = golden_graph("rmat_s10_e8")
    prefix = os.path.join(d, "GT")
    g, og = G.Graph(prefix, "GT"), oracle_mod.OracleGraph(prefix)
    roots = np.random.default_rng(steps).integers(0, g.n, (samples, walkers), dtype=np.uint32)
    got = g.mrw(roots, steps, 4, G.SELECT_DEGREE_CT)
    for a, b in zip(got, og.mrw("GT", roots, steps, 4, G.SELECT_DEGREE_CT)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("obj", ["LE", "csr"])
@pytest.mark.parametrize("use_graph", [1, 2])
def test_batch_of_both_levels(oracle_mod, obj, use_graph):
    """Block-level and warp-level items of one batch, run twice, replayed and launched plainly."""
    import torch
    d, _, _, _ = golden_graph("rmat_s10_e8")
    prefix = os.path.join(d, "LE")
    g, og = G.Graph(prefix, "LE"), oracle_mod.OracleGraph(prefix)
    b = G.Batch(g if obj == "LE" else g.csr())
    rng, checks = np.random.default_rng(2), []

    def dev(x):
        return torch.from_numpy(x.view(np.int32)).cuda()

    for i in range(12):
        if i % 3 == 0:
            select = (2, 1, 0)[i // 3 % 3]
            roots = rng.integers(0, g.n, (3, 40), dtype=np.uint32)
            outs = [dev(roots), *(torch.zeros(3, 300, dtype=torch.int32, device="cuda") for _ in range(2))]
            b.add_mrw(outs[0], 3, 40, 300, i, outs[1], outs[2], select=select)
            src, dst, end, _ = og.mrw("LE", roots, 300, i, select)
            checks += zip(outs, (end, src, dst))
        elif i % 3 == 1:
            starts = rng.integers(0, g.n, 200, dtype=np.uint32)
            paths, inp = torch.zeros(200, 31, dtype=torch.int32, device="cuda"), dev(starts)
            b.add_rw(inp, 200, 30, i, paths)
            checks += [(paths, og.rw("LE", starts, 30, i)[0]), (inp, starts)]
        else:
            seeds = rng.integers(0, g.n, 90, dtype=np.uint32)
            hops, inp = [torch.zeros(90, w, dtype=torch.int32, device="cuda") for w in (5, 35)], dev(seeds)
            b.add_khop(inp, 90, (5, 7), i, hops)
            checks += [*zip(hops, og.khop("LE", seeds, (5, 7), i)[0]), (inp, seeds)]
    b.set_config(use_graph=use_graph)
    for _ in range(2):
        b.run()
        torch.cuda.synchronize()
        for got, ref in checks:
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), ref)
