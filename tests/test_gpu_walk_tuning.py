"""Launch shapes of the walk that a caller sets in part."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning,threads", [
    (dict(), 64), (dict(rw_blocks_per_sm=2), 256), (dict(rw_depth=2, rw_blocks_per_sm=1), 256),
    (dict(rw_threads=32, rw_blocks_per_sm=2), 32), (dict(rw_threads=512), 512)])
def test_threads_of_a_walk(oracle_mod, tuning, threads):
    """Blocks per SM bound blocks of 256 threads where the caller says no number of them."""
    prefix = os.path.join(golden_graph("rmat_s10_e8")[0], "GT")
    g = G.Graph(prefix, "GT")
    g.set_tuning(**tuning)
    assert g.tuning()["rw_threads"] == threads
    starts = np.arange(3000, dtype=np.uint32) % g.n
    ref, edges = oracle_mod.OracleGraph(prefix).rw("GT", starts, 9, 3)
    paths, e = g.rw(starts, 9, 3)
    np.testing.assert_array_equal(paths, ref)
    assert e == edges
