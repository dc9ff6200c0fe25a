"""Small walks on host buffers (one pinned buffer, a running edge counter) when
something around them fails."""
import contextlib
import ctypes as C
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


def test_a_call_too_large_for_64_bits_is_refused(oracle_mod):
    """Sizes whose product in bytes is a multiple of 2^64: no memory, not a small call."""
    g, og, starts = _graphs(oracle_mod)
    many = np.zeros(1 << 31, np.uint32)  # (never written: takes no memory)
    p, e = G.RwParams((1 << 31) - 2, G.LAYOUT_WALK_MAJOR, 3), C.c_uint64()
    assert len(many) * (p.length + 2) * 4 == 1 << 64
    assert G.lib.grass_rw_host(g.handle, C.byref(p), G._p(many), len(many), G._p(many), C.byref(e)) == G.E_OOM
    with contextlib.suppress(G.GrassError):  # (takes the refused allocation's error)
        g.rw(starts, 20, 3)
    np.testing.assert_array_equal(g.rw(starts, 20, 3)[0], og.rw("LE", starts, 20, 3)[0])


def test_small_call_without_pinned_memory(oracle_mod):
    """The test build of the library, where pinned memory cannot be had: the same walks."""
    lib, P = C.CDLL(os.path.join(os.path.dirname(G.LIB_PATH), "libgrass_b200_stagetest.so")), C.c_void_p
    lib.grass_open.argtypes = [C.c_char_p, C.c_int, C.c_int, C.POINTER(P)]
    lib.grass_rw_host.argtypes = [P, P, P, C.c_uint64, P, C.POINTER(C.c_uint64)]
    lib.grass_close.argtypes = [P]
    prefix, h, e = os.path.join(golden_graph("rmat_s10_e8")[0], "LE"), P(), C.c_uint64()
    assert lib.grass_open(prefix.encode(), G.MODE_LE, 0, C.byref(h)) == G.OK
    starts = np.arange(100, dtype=np.uint32)
    ref, edges = oracle_mod.OracleGraph(prefix).rw("LE", starts, 20, 3)
    for _ in range(2):
        paths, p = np.zeros((100, 21), np.uint32), G.RwParams(20, G.LAYOUT_WALK_MAJOR, 3)
        assert lib.grass_rw_host(h, C.byref(p), G._p(starts), 100, G._p(paths), C.byref(e)) == G.OK
        np.testing.assert_array_equal(paths, ref)
        assert e.value == edges
    assert lib.grass_close(h) == G.OK
