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
