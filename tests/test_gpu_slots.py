"""The device slot layout at its edges, against the input lists and the oracle.

A vertex's slots depend on its degree and on how its neighbors spread: dense
lists put more than 64 neighbors in a sector, sparse ones 8; a list of up to 32
neighbors can be one slot without a head; a vertex of degree 1 has no slot.  The
decode sweep treats degrees below and from 128 differently, stages 32 sectors at
a time, and splits vertices from 2048 neighbors.  Every value is compared
exactly."""
import numpy as np
import pytest

import grass_b200 as G

pytestmark = pytest.mark.gpu

N = 3_000_000  # ids of up to 22 bits
DEGREES = (1, 2, 3, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 2047, 2048, 2049, 4097)


def _csr(gap):
    """Vertices 0, 2, 4, ... have DEGREES[k] neighbors whose gaps are at most
    `gap` (0: spread over all ids); the others have none, but for the last."""
    rng = np.random.default_rng(gap)
    rows = []
    for k, d in enumerate(DEGREES):
        if gap:
            nb = 2 * k + 1 + np.cumsum(rng.integers(1, gap + 1, d))
        else:
            nb = np.unique(rng.integers(0, N, 3 * d + 9))
            nb = rng.permutation(nb[nb != 2 * k])[:d]
        rows.append(np.sort(nb).astype(np.uint32))
    rp = np.zeros(N + 1, np.uint64)
    rp[1:2 * len(rows):2] = [len(r) for r in rows]
    rp[N] = 1  # (trailing vertices with no neighbors would be trimmed)
    return np.cumsum(rp, dtype=np.uint64), np.concatenate(rows + [np.array([7], np.uint32)])


@pytest.mark.parametrize("mode", ["GT", "LE"])
@pytest.mark.parametrize("gap", [1, 2, 9, 700, 0])
def test_slots_hold_the_lists(oracle_mod, tmp_path, mode, gap):
    rp, cols = _csr(gap)
    G.compress_to_files(rp, cols, mode, str(tmp_path / mode))
    g = G.Graph(str(tmp_path / mode), mode)
    r, c = g.decode_all()
    np.testing.assert_array_equal(r, rp)
    np.testing.assert_array_equal(c, cols)
    g.check_device_error()
    # one draw from every neighbor index in reach, by the walk, k-hop and node2vec kernels
    og = oracle_mod.OracleGraph(str(tmp_path / mode))
    starts = np.repeat(np.arange(0, 2 * len(DEGREES), 2, dtype=np.uint32), 800)
    paths, e = g.rw(starts, 2, 3)
    ref, re_ = og.rw(mode, starts, 2, 3)
    np.testing.assert_array_equal(paths, ref)
    assert e == re_
    hops, e = g.khop(starts[::7], (33, 2), 4)
    refs, re_ = og.khop(mode, starts[::7], (33, 2), 4)
    for a, b in zip(hops, refs):
        np.testing.assert_array_equal(a, b)
    assert e == re_


@pytest.mark.parametrize("depth", [1, 2, 4])
@pytest.mark.parametrize("gap", [1, 9, 0])
def test_staged_sectors_hold_the_lists(tmp_path, depth, gap):
    rp, cols = _csr(gap)
    G.compress_to_files(rp, cols, "LE", str(tmp_path / "LE"))
    g = G.Graph(str(tmp_path / "LE"), "LE")
    g.set_tuning(decode_stage_depth=depth)
    r, c = g.decode_all()
    np.testing.assert_array_equal(r, rp)
    np.testing.assert_array_equal(c, cols)
    g.check_device_error()
