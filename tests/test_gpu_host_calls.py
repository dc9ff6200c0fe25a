"""Small walks on host buffers (one pinned buffer, a running edge counter) when
something around them fails."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


def _graphs(oracle_mod):
    prefix = os.path.join(golden_graph("rmat_s10_e8")[0], "LE")
    g = G.Graph(prefix, "LE")
    return g, oracle_mod.OracleGraph(prefix), np.arange(100, dtype=np.uint32) % g.n


def _leave_an_error(g):
    """A refused allocation (2^62 bytes), whose error the CUDA runtime keeps for the next query."""
    with pytest.raises(G.GrassError):
        G.Batch(g).add_mrw(1 << 12, (1 << 30) - 1, (1 << 30) - 1, 1, 0, 1 << 12, 1 << 12)


def test_edges_after_a_failed_small_call(oracle_mod):
    """A call that fails after its walk was launched leaves nothing to the next one's edge count."""
    g, og, starts = _graphs(oracle_mod)
    ref, edges = og.rw("LE", starts, 20, 3)
    assert g.rw(starts, 20, 3)[1] == edges
    _leave_an_error(g)
    with pytest.raises(G.GrassError):
        g.rw(starts[:50], 30, 4)
    for _ in range(2):
        paths, e = g.rw(starts, 20, 3)
        np.testing.assert_array_equal(paths, ref)
        assert e == edges
