"""The membership search of the second-order walk: lists of one sector, one line
and many lines (their fences are built by the first call that is not captured;
a captured first call searches without them), against the oracle."""
import numpy as np
import pytest

import grass_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["GT", "LE"])
@pytest.mark.parametrize("spread", [1, 40, 700])
def test_search_with_and_without_fences(oracle_mod, tmp_path, mode, spread):
    import torch
    # a ring of hubs with lists of 1 to 5000 neighbors, each of them a neighbor of the hubs around it,
    # so that candidates are often neighbors of the vertex before
    rng = np.random.default_rng(spread)
    degrees = [1, 2, 5, 12, 13, 40, 100, 101, 160, 400, 1000, 5000]
    n = 5100 * spread + 50
    rows = []
    for k, d in enumerate(degrees):
        near = [(k + j) % len(degrees) for j in range(1, 6)][:d]
        far = 12 + np.cumsum(rng.integers(1, spread + 1, max(d - len(near), 0)))
        rows.append(np.unique(np.concatenate([near, far])))
    rows += [rng.choice(12, 3, replace=False) for _ in range(n - len(rows))]
    rows = [np.sort(r).astype(np.uint32) for r in rows]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    G.compress_to_files(rp, np.concatenate(rows), mode, str(tmp_path / mode))
    g, og = G.Graph(str(tmp_path / mode), mode), oracle_mod.OracleGraph(str(tmp_path / mode))
    W, L = 3001, 24
    starts = rng.integers(0, 12, W, dtype=np.uint32)
    ref, total = og.node2vec(mode, starts, L, 5, 1.0, 0.5)
    dev = torch.from_numpy(starts.view(np.int32)).cuda()
    paths = torch.zeros(W, L + 1, dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        g.node2vec_device(dev, W, L, 5, 1.0, 0.5, paths, edge_count=count, stream=stream)
    for call in (graph.replay, lambda: g.node2vec_device(dev, W, L, 5, 1.0, 0.5, paths, edge_count=count)):
        paths.fill_(-7)
        count.zero_()
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(paths.cpu().numpy().view(np.uint32), ref)
        assert int(count) == total


def test_first_call_beside_a_capture(oracle_mod, tmp_path):
    """The first call builds the fences; another stream's capture goes on."""
    import torch
    n, d = 400, 150
    rows = [np.sort(np.random.default_rng(v).choice(n, d, replace=False)).astype(np.uint32) for v in range(n)]
    rp = (np.arange(n + 1) * d).astype(np.uint64)
    G.compress_to_files(rp, np.concatenate(rows), "LE", str(tmp_path / "g"))
    g, og = G.Graph(str(tmp_path / "g"), "LE"), oracle_mod.OracleGraph(str(tmp_path / "g"))
    W, L = 500, 10
    starts = np.arange(W, dtype=np.uint32) % n
    ref, _ = og.node2vec("LE", starts, L, 5, 1.0, 0.5)
    dev = torch.from_numpy(starts.view(np.int32)).cuda()
    captured, beside = (torch.zeros(W, L + 1, dtype=torch.int32, device="cuda") for _ in range(2))
    graph, stream, other = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        g.node2vec_device(dev, W, L, 5, 1.0, 0.5, captured, stream=stream)
        g.node2vec_device(dev, W, L, 5, 1.0, 0.5, beside, stream=other)
    graph.replay()
    torch.cuda.synchronize()
    for paths in (captured, beside):
        np.testing.assert_array_equal(paths.cpu().numpy().view(np.uint32), ref)
