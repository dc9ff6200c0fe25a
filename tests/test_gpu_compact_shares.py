"""Compaction at the edges of its tiles (4096 slots) and of the blocks' shares of
them, with parents of few and of many slots, against a mask of the input."""
import pytest

import grass_b200 as G

pytestmark = pytest.mark.gpu
TILE = 4096


def _children(torch, shape, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    x = torch.randint(0, 1 << 30, shape, generator=gen, device="cuda", dtype=torch.int32)
    return x.masked_fill_(torch.rand(shape, generator=gen, device="cuda") < 0.3, -1)


def _check(torch, call, src, dst):
    keep = dst != -1
    src, dst, n = src[keep], dst[keep], int(keep.sum())
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    for cap in (n + 3, n // 2):
        out = torch.full((2, n + 3), -7, dtype=torch.int32, device="cuda")
        call(out[0], out[1], cap, count)
        torch.cuda.synchronize()
        m = min(n, cap)
        assert int(count) == n
        assert torch.equal(out[0, :m], src[:m]) and torch.equal(out[1, :m], dst[:m])
        assert bool((out[:, m:] == -7).all())


@pytest.mark.parametrize("slots", [1, 31, TILE, TILE + 1, 2368 * TILE, 2368 * TILE + 1, 5000 * TILE - 1])
def test_shares(slots):
    import torch
    src = torch.arange(slots, dtype=torch.int32, device="cuda")
    dst = _children(torch, (slots,), slots)
    dst[TILE:3 * TILE] = -1  # tiles without an edge
    _check(torch, lambda s, d, cap, n: G.mrw_edges_device(src, dst, slots, 1, s, d, cap, n), src, dst)


@pytest.mark.parametrize("seeds,fanouts", [(1, (1,)), (700, (3, 7)), (3, (4096, 2)), (2, (4097, 3)), (1, (9000,)), (41, (5, 5, 5, 33))])
def test_fanouts(seeds, fanouts):
    import torch
    roots = torch.arange(seeds, dtype=torch.int32, device="cuda")
    hops = [_children(torch, (seeds, w), w) for w in G.hop_widths(fanouts)]
    src = torch.cat([p.reshape(-1).repeat_interleave(f) for p, f in zip([roots, *hops], fanouts)])
    dst = torch.cat([h.reshape(-1) for h in hops])
    _check(torch, lambda s, d, cap, n: G.khop_edges_device(roots, seeds, fanouts, hops, s, d, cap, n), src, dst)


@pytest.mark.parametrize("layout", [G.LAYOUT_WALK_MAJOR, G.LAYOUT_STEP_MAJOR])
@pytest.mark.parametrize("walks,length", [(1, 1), (5000, 1), (130, 31), (129, 32), (260, 33), (2, 4097), (1, 9001)])
def test_paths(layout, walks, length):
    import torch
    shape = (walks, length + 1) if layout == G.LAYOUT_WALK_MAJOR else (length + 1, walks)
    paths = _children(torch, shape, length)
    if layout == G.LAYOUT_WALK_MAJOR:
        src, dst = paths[:, :-1].reshape(-1), paths[:, 1:].reshape(-1)
    else:
        src, dst = paths[:-1].reshape(-1), paths[1:].reshape(-1)
    _check(torch, lambda s, d, cap, n: G.rw_edges_device(paths, walks, length, s, d, cap, n, layout), src, dst)
