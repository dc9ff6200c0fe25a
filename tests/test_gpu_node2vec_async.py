"""The first second-order walk on a graph starts the build of its index and
returns: it waits for no work of the caller's stream."""
import numpy as np
import pytest

import grass_b200 as G

pytestmark = pytest.mark.gpu


def _graph(tmp_path, name, seed):
    n, d = 400, 150  # (lists of several lines: they have fences)
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(n, d, replace=False)).astype(np.uint32) for _ in range(n)]
    G.compress_to_files((np.arange(n + 1) * d).astype(np.uint64), np.concatenate(rows), "LE", str(tmp_path / name))
    return G.Graph(str(tmp_path / name), "LE")


def test_first_call_behind_pending_work(oracle_mod, tmp_path):
    import torch
    warm, g = _graph(tmp_path, "warm", 1), _graph(tmp_path, "g", 2)
    og = oracle_mod.OracleGraph(str(tmp_path / "g"))
    W, L = 500, 10
    starts = np.arange(W, dtype=np.uint32) % g.n
    ref, _ = og.node2vec("LE", starts, L, 5, 1.0, 0.5)
    dev = torch.from_numpy(starts.view(np.int32)).cuda()
    first, beside, later = (torch.zeros(W, L + 1, dtype=torch.int32, device="cuda") for _ in range(3))
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    warm.node2vec_device(dev, W, L, 5, 1.0, 0.5, first, stream=stream)  # (loads the kernels)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(2_000_000_000)  # about a second
        slept = stream.record_event()
    g.node2vec_device(dev, W, L, 5, 1.0, 0.5, first, stream=stream)
    g.node2vec_device(dev, W, L, 5, 1.0, 0.5, beside, stream=other)
    other.synchronize()
    assert not slept.query(), "the first call waited for its stream's earlier work"
    stream.synchronize()
    g.node2vec_device(dev, W, L, 5, 1.0, 0.5, later, stream=other)
    torch.cuda.synchronize()
    for paths in (first, beside, later):
        np.testing.assert_array_equal(paths.cpu().numpy().view(np.uint32), ref)
