"""Walk-major paths are collected 16 / depth columns at a time and written by
rows: lengths around that, walker counts around a warp and a block, walks that
stop, for every depth, against the oracle."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 2, 4])
@pytest.mark.parametrize("walkers,length", [(1, 1), (31, 2), (32, 3), (33, 4), (63, 14), (65, 15), (129, 16), (500, 17), (777, 33)])
def test_walk_major_rows(oracle_mod, depth, walkers, length):
    d, _, _, _ = golden_graph("edge_cases")  # (has vertices without neighbors)
    prefix = os.path.join(d, "GT")
    g, og = G.Graph(prefix, "GT"), oracle_mod.OracleGraph(prefix)
    g.set_tuning(rw_depth=depth, rw_blocks_per_sm=1)
    starts = np.random.default_rng(length).integers(0, g.n + 1, walkers, dtype=np.uint32)
    paths, e = g.rw(starts, length, 5)
    ref, re_ = og.rw("GT", starts, length, 5)
    np.testing.assert_array_equal(paths, ref)
    assert e == re_
    steps, e = g.rw(starts, length, 5, G.LAYOUT_STEP_MAJOR)
    np.testing.assert_array_equal(steps, ref.T)
    assert e == re_
