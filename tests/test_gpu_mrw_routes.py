"""Multi-RW on both sides of the rules that pick its kernels and their shapes,
against the oracle."""
import os

import numpy as np
import pytest

from conftest import golden_graph
import grass_b200 as G

pytestmark = pytest.mark.gpu


def _compare(oracle_mod, name, mode, samples, walkers, steps, select, roots=None):
    prefix = os.path.join(golden_graph(name)[0], mode)
    g, og = G.Graph(prefix, mode), oracle_mod.OracleGraph(prefix)
    if roots is None:
        roots = np.random.default_rng(steps).integers(0, g.n + 1, (samples, walkers), dtype=np.uint32)
    got = g.mrw(roots, steps, 4, select)
    for a, b in zip(got, og.mrw(mode, roots, steps, 4, select)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("walkers,steps", [
    (5, 1), (300, 2), (40, 15), (40, 16), (33, 31), (33, 32), (33, 33), (600, 64), (20, 500), (300, 4095), (600, 4097)])
def test_few_events_to_order(oracle_mod, walkers, steps):
    """Continuous time with event counts around the numbers of buckets."""
    _compare(oracle_mod, "rmat_s10_e8", "LE", 3, walkers, steps, G.SELECT_DEGREE_CT)


def test_no_events(oracle_mod):
    """Continuous time from no vertex at all (ids past the last): nothing moves."""
    _compare(oracle_mod, "edge_cases", "GT", 2, 5, 9, G.SELECT_DEGREE_CT, np.full((2, 5), G.INVALID, np.uint32))


@pytest.mark.parametrize("samples,walkers,steps", [(148, 257, 40), (149, 257, 40), (200, 512, 33), (150, 161, 20), (149, 200, 500)])
def test_more_continuous_time_samples_than_sms(oracle_mod, samples, walkers, steps):
    """Blocks of fewer threads than walkers."""
    _compare(oracle_mod, "rmat_s10_e8", "GT", samples, walkers, steps, G.SELECT_DEGREE_CT)


@pytest.mark.parametrize("samples,walkers,steps", [
    (2, 40, 319), (2, 40, 320), (148, 80, 300), (593, 80, 300), (2, 11, 4000), (2, 12, 4000), (1, 1, 600),
    (149, 1000, 300), (297, 2000, 600), (2, 5000, 400)])
def test_uniform_samples_as_blocks_or_warps(oracle_mod, samples, walkers, steps):
    _compare(oracle_mod, "edge_cases", "LE", samples, walkers, steps, G.SELECT_UNIFORM)


@pytest.mark.parametrize("samples,walkers,steps", [
    (3, 178, 40), (3, 181, 40), (5, 256, 9), (8000, 208, 30), (5000, 208, 30), (9000, 20, 5), (9000, 160, 5)])
def test_degree_samples_as_groups_or_warps(oracle_mod, samples, walkers, steps):
    _compare(oracle_mod, "edge_cases", "GT", samples, walkers, steps, G.SELECT_DEGREE)


@pytest.mark.parametrize("select", [G.SELECT_UNIFORM, G.SELECT_DEGREE_CT])
@pytest.mark.parametrize("shapes", [[(296, 40, 20)], [(297, 40, 20)], [(3, 600, 30), (400, 20, 9)], [(100, 300, 40)] * 3])
def test_block_level_samples_of_a_batch(oracle_mod, shapes, select):
    """Few and many samples, of one job and of several sizes: blocks of 128 to 512 threads."""
    import torch
    prefix = os.path.join(golden_graph("rmat_s10_e8")[0], "LE")
    g, og = G.Graph(prefix, "LE"), oracle_mod.OracleGraph(prefix)
    b, checks, rng = G.Batch(g), [], np.random.default_rng(3)
    for i, (samples, walkers, steps) in enumerate(shapes):
        roots = rng.integers(0, g.n, (samples, walkers), dtype=np.uint32)
        outs = [torch.from_numpy(roots.view(np.int32)).cuda(),
                *(torch.zeros(samples, steps, dtype=torch.int32, device="cuda") for _ in range(2))]
        b.add_mrw(outs[0], samples, walkers, steps, i, outs[1], outs[2], select=select)
        src, dst, end, _ = og.mrw("LE", roots, steps, i, select)
        checks += zip(outs, (end, src, dst))
    for _ in range(2):
        b.run()
        torch.cuda.synchronize()
        for got, ref in checks:
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), ref)


def test_scratch_for_fewer_blocks(oracle_mod):
    """Block-level samples where the scratch of all resident blocks does not fit (some 4 GB): the same chains."""
    import torch
    g = G.Graph(os.path.join(golden_graph("rmat_s10_e8")[0], "LE"), "LE")
    S, R, T = 500, 400, 100_000
    roots = torch.randint(0, g.n, (S, R), dtype=torch.int32, device="cuda")
    calls = [[roots.clone(), *(torch.zeros(S, T, dtype=torch.int32, device="cuda") for _ in range(2))] for _ in range(2)]
    hog = []
    for walkers, src, dst in calls:
        g.mrw_device(walkers, S, R, T, 3, src, dst, select=G.SELECT_DEGREE_CT)
        g.check_device_error()
        torch.cuda.empty_cache()
        if not hog:  # (the library's pool gives back what it freed when the device is idle)
            hog.append(torch.empty(torch.cuda.mem_get_info()[0] - (2 << 30), dtype=torch.uint8, device="cuda"))
    del hog
    torch.cuda.empty_cache()
    for a, b in zip(*calls):
        assert torch.equal(a, b)
