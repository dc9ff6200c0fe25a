"""Workloads of the sampling library, for measuring it: what its users run, over the range they run it in.

A program opens a compressed graph once, keeps it on the GPU and calls the samplers on it again and again, each time
with other start vertices and another random seed.  So a state holds the resident graph (shared by all states of one
graph), the start vertices, the output buffers and the seed; only the decode workload has a graph of its own per seed,
because there the graph is the input.  Graphs are R-MAT graphs in the shapes the repository benchmarks: scale 16, edge
factor 16 (fits L2) and scale 22, edge factor 32 (250 M neighbors, far larger than L2), with scale 20 between them.
"""
import functools
import math

import numpy as np
import torch

import grass_b200 as G

DEV = "cuda"
STEP, WALK = G.LAYOUT_STEP_MAJOR, G.LAYOUT_WALK_MAJOR
GRAPHS = ((16, 16), (20, 16), (22, 32))
FANOUTS = ("25,10", "15,10", "10,5", "5,5,5")
BIASES = ((1.0, 0.5), (4.0, 0.25), (0.5, 2.0))


def listed():
    return [
        # The plain host call of a script or a test: a few walks on a small graph, arrays in and out.
        dict(name="rw host small", kind="rw_host", mode="GT", scale=16, ef=16, walkers=1000, length=20, layout=WALK),
        # One mini-batch of walks for an embedding trainer, small graph: latency of the 80-step chain.
        dict(name="rw small", kind="rw", mode="LE", scale=16, ef=16, walkers=4096, length=80, layout=STEP),
        # The repository's headline: 1M uniform walkers x 80 steps, step-major paths.
        dict(name="rw large", kind="rw", mode="LE", scale=22, ef=32, walkers=1 << 20, length=80, layout=STEP),
        # Shorter walks of a ragged number of walkers in the default (walk-major) layout, the other format.
        dict(name="rw walk-major", kind="rw", mode="GT", scale=22, ef=32, walkers=200_003, length=40, layout=WALK),
        # The benchmarked 2-hop neighborhood sampling, a large batch of seeds.
        dict(name="khop large", kind="khop", mode="LE", scale=22, ef=32, seeds=65_536, fanouts="25,10"),
        # 3-hop sampling for a mini-batch of an odd size.
        dict(name="khop 3-hop", kind="khop", mode="GT", scale=22, ef=32, seeds=2_999, fanouts="5,5,5"),
        # What feeds a GNN layer: a neighborhood sample and its compaction to an edge list.
        dict(name="khop to edges", kind="khop_edges", mode="LE", scale=20, ef=16, seeds=16_384, fanouts="15,10"),
        # The multi-RW app's shape, 80 walkers x 100 steps a sample, walkers picked uniformly.
        dict(name="mrw uniform", kind="mrw", mode="LE", scale=22, ef=32, samples=65_536, walkers=80, steps=100, select=0),
        # Frontier sampling: the same shape, the walker of each step picked in proportion to its degree.
        dict(name="mrw degree", kind="mrw", mode="GT", scale=22, ef=32, samples=8_192, walkers=80, steps=100, select=1),
        # Second-order walks with the usual in-out bias.
        dict(name="node2vec", kind="n2v", mode="LE", scale=22, ef=32, walkers=262_144, length=80, p=1.0, q=0.5),
        # Decompression of a whole graph to CSR.
        dict(name="decode", kind="decode", mode="LE", scale=21, ef=16),
        # Many uneven requests in one launch: 40 % walks, 40 % k-hops, 20 % long degree-proportional multi-RW chains.
        dict(name="batch mix", kind="batch", mode="LE", scale=22, ef=32, jobs=256, mix=3),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("rw", "rw", "rw_host", "khop", "khop", "khop_edges", "mrw", "mrw", "n2v", "decode", "batch"))
    scale, ef = rng.choice(GRAPHS)
    c = dict(kind=kind, mode=rng.choice(("LE", "GT")), scale=scale, ef=ef)
    if kind in ("rw", "rw_host"):
        c.update(walkers=_log(rng, 100, 1_000_000 if kind == "rw" else 20_000), length=rng.randint(5, 80),
                 layout=rng.choice((STEP, WALK)))
    elif kind in ("khop", "khop_edges"):
        c.update(seeds=_log(rng, 20, 65_000), fanouts=rng.choice(FANOUTS))
    elif kind == "mrw":
        c.update(select=rng.choice((0, 0, 1, 2)), walkers=rng.choice((80, rng.randint(8, 250))), steps=rng.randint(30, 150))
        most = (5_000_000, 500_000, 200_000)[c["select"]] // c["steps"]
        c.update(samples=_log(rng, 8, most))
        if c["select"] == 2 and rng.random() < 0.5:  # a few long chains
            c.update(walkers=rng.randint(500, 2000), steps=rng.randint(2_000, 10_000), samples=rng.randint(1, 50))
    elif kind == "n2v":
        p, q = rng.choice(BIASES)
        c.update(walkers=_log(rng, 100, 250_000), length=rng.randint(10, 80), p=p, q=q)
    elif kind == "decode":
        c.update(scale=rng.randint(14, 21), ef=rng.randint(8, 16))
    else:
        c.update(jobs=_log(rng, 8, 250), mix=rng.randint(10, 1_000_000))
    return c


# ---- inputs ----

def _rmat(scale, ef, seed):
    """An undirected R-MAT graph as CSR (rowptr, cols) on the GPU: vertices numbered by first appearance in the edge
    list, self-loops and duplicates dropped, rows sorted."""
    gen = torch.Generator(DEV).manual_seed(seed)
    m = ef << scale
    s = torch.zeros(m, dtype=torch.int64, device=DEV)
    d = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device=DEV)
        down = r >= 0.76
        right = ((r >= 0.57) & ~down) | (r >= 0.95)
        s.mul_(2).add_(down)
        d.mul_(2).add_(right)
    keep = s != d
    s, d = s[keep], d[keep]
    at = torch.arange(s.numel(), device=DEV)
    first = torch.full((1 << scale,), 1 << 62, dtype=torch.int64, device=DEV)
    first.scatter_reduce_(0, s, 2 * at, "amin").scatter_reduce_(0, d, 2 * at + 1, "amin")
    order = torch.argsort(first)
    n = int((first < 1 << 62).sum())
    name = torch.empty_like(order)
    name[order] = torch.arange(1 << scale, device=DEV)
    s, d = name[s], name[d]
    key = torch.cat((s * n + d, d * n + s)).sort().values
    key = key[torch.cat((torch.ones(1, dtype=torch.bool, device=DEV), key[1:] != key[:-1]))]
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
    return rowptr, (key % n).to(torch.int32)


@functools.lru_cache(None)
def _csr(scale, ef):
    return _rmat(scale, ef, 42)


def _open(rowptr, cols, mode):
    graph, offset = G.compress(rowptr.cpu().numpy().view(np.uint64), cols.cpu().numpy().view(np.uint32), mode)
    torch.cuda.empty_cache()  # the library allocates outside torch's pool
    return G.Graph.from_bytes(graph, offset, mode)


@functools.lru_cache(None)
def _graph(scale, ef, mode):
    return _open(*_csr(scale, ef), mode)


def _gen(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _vertices(n, shape, gen):
    return torch.randint(0, n, shape, generator=gen, device=DEV, dtype=torch.int32)


def _out(*shape):
    return torch.full(shape, -1, dtype=torch.int32, device=DEV)


def _fanouts(c):
    return tuple(int(f) for f in c["fanouts"].split(","))


def _paths_shape(c):
    w, l1 = c["walkers"], c["length"] + 1
    return (w, l1) if c.get("layout", WALK) == WALK else (l1, w)


def _mix(c):
    """The batched-jobs workload: 40 % walks, 40 % k-hops, 20 % multi-RW samples of 2000 walkers x 10,000 steps; the
    numbers of walkers and seeds are lognormal around 1024."""
    rng = np.random.default_rng(c["mix"])
    jobs = []
    for i in range(c["jobs"]):
        size = int(np.clip(np.rint(rng.lognormal(np.log(1024), 1.5)), 1, 65_536))
        kind = ("rw", "rw", "khop", "khop", "mrw")[i % 5]
        jobs.append((kind, size, int(rng.integers(10, 101)), G.MIX_FANOUTS[int(rng.integers(0, 4))]))
    return jobs


def _room(c, x):
    """x in a buffer with room for any graph of this shape."""
    most = (1 << c["scale"]) + 1 if x.dtype == torch.int64 else 2 * c["ef"] << c["scale"]
    return torch.nn.functional.pad(x, (0, most - x.numel()), value=-1)


class _Arena:
    """One buffer for the outputs of a batch's jobs, each of them on a 512-byte boundary."""

    def __init__(self, words):
        self.all, self.used = _out(sum(_round(w) for w in words)), 0

    def take(self, words):
        self.used += _round(words)
        return self.all[self.used - _round(words):][:words]


def _round(words):
    return (words + 127) // 128 * 128


def _batch_words(jobs):
    for job, size, length, fanouts in jobs:
        if job == "mrw":
            yield from (10_000, 10_000)
        elif job == "rw":
            yield size * (length + 1)
        else:
            yield from (size * w for w in G.hop_widths(fanouts))


def prepare(case, seed):
    c, kind, gen = case, case["kind"], _gen(seed)
    st = dict(case=c, seed=seed)
    if kind == "decode":
        rowptr, cols = _rmat(c["scale"], c["ef"], seed)
        st["g"] = _open(rowptr, cols, c["mode"])
        st["rowptr"], st["cols"] = (torch.full_like(_room(c, x), -1) for x in (rowptr, cols))
        return st
    g = st["g"] = _graph(c["scale"], c["ef"], c["mode"])
    n = g.n
    st["count"] = torch.zeros(1, dtype=torch.int64, device=DEV)
    if kind == "rw_host":
        st["starts"] = np.random.default_rng(seed).integers(0, n, c["walkers"], dtype=np.uint32)
    elif kind in ("rw", "n2v"):
        st.update(starts=_vertices(n, (c["walkers"],), gen), paths=_out(*_paths_shape(c)))
    elif kind in ("khop", "khop_edges"):
        st["starts"] = _vertices(n, (c["seeds"],), gen)
        st["hops"] = [_out(c["seeds"], w) for w in G.hop_widths(_fanouts(c))]
        if kind == "khop_edges":
            st["slots"] = c["seeds"] * sum(G.hop_widths(_fanouts(c)))
            st["edges"] = [_out(st["slots"]) for _ in range(2)]
    elif kind == "mrw":
        st.update(roots=_vertices(n, (c["samples"], c["walkers"]), gen), walkers=_out(c["samples"], c["walkers"]))
        st["edges"] = [_out(c["samples"], c["steps"]) for _ in range(2)]
    else:
        jobs = _mix(c)
        walks, chains = _Arena(_batch_words(jobs)), sum(job == "mrw" for job, *_ in jobs)
        st.update(out=walks.all, roots=_vertices(n, (chains, 2000), gen), keep=[])
        b, roots = G.Batch(g), iter(st["roots"])
        for i, (job, size, length, fanouts) in enumerate(jobs):
            if job == "mrw":
                b.add_mrw(next(roots), 1, 2000, 10_000, seed + i, walks.take(10_000), walks.take(10_000),
                          select=G.SELECT_DEGREE_CT)
                continue
            starts = _vertices(n, (size,), gen)
            st["keep"].append(starts)
            if job == "rw":
                b.add_rw(starts, size, length, seed + i, walks.take(size * (length + 1)))
            else:
                b.add_khop(starts, size, fanouts, seed + i, [walks.take(size * w) for w in G.hop_widths(fanouts)])
        st["batch"] = b
    return st


def run(st):
    c, g, seed = st["case"], st["g"], st["seed"]
    kind = c["kind"]
    if kind == "decode":
        g.decode_all_device(st["rowptr"], st["cols"])
        return [st["rowptr"], st["cols"]]
    if kind == "rw_host":
        return g.rw(st["starts"], c["length"], seed, layout=c["layout"])
    count = st["count"].zero_()
    if kind == "rw":
        g.rw_device(st["starts"], c["walkers"], c["length"], seed, st["paths"], edge_count=count, layout=c["layout"])
        return [st["paths"], count]
    if kind == "n2v":
        g.node2vec_device(st["starts"], c["walkers"], c["length"], seed, c["p"], c["q"], st["paths"], edge_count=count)
        return [st["paths"], count]
    if kind == "khop":
        g.khop_device(st["starts"], c["seeds"], _fanouts(c), seed, st["hops"], edge_count=count)
        return [*st["hops"], count]
    if kind == "khop_edges":
        g.khop_device(st["starts"], c["seeds"], _fanouts(c), seed, st["hops"])
        G.khop_edges_device(st["starts"], c["seeds"], _fanouts(c), st["hops"], *st["edges"], st["slots"], count)
        return [*st["hops"], *st["edges"], count]
    if kind == "mrw":  # the walkers move in place: they start from the roots again
        st["walkers"].copy_(st["roots"])
        g.mrw_device(st["walkers"], c["samples"], c["walkers"], c["steps"], seed, *st["edges"], select=c["select"],
                     edge_count=count)
        return [st["walkers"], *st["edges"], count]
    st["batch"].run(total=count)
    return [st["out"], st["roots"], count]


def work(case):
    """Bytes one pass cannot do without: its starts, its outputs, and the part of the graph that it visits, at most the
    whole compressed graph once (a draw needs its vertex's 16 bytes and about 4 bytes of payload)."""
    c, kind = case, case["kind"]
    neighbors = 1.9 * (c["ef"] << c["scale"])
    graph = neighbors * c["scale"] / 8
    if kind == "decode":
        return dict(bytes=graph + 4 * neighbors + 8 * (1 << c["scale"]), flops=0)
    if kind in ("rw", "rw_host", "n2v"):
        draws, other = c["walkers"] * c["length"], 2 * c["walkers"]
    elif kind in ("khop", "khop_edges"):
        draws, other = c["seeds"] * sum(G.hop_widths(_fanouts(c))), c["seeds"]
        if kind == "khop_edges":
            other += 2 * draws
    elif kind == "mrw":
        draws = c["samples"] * c["steps"]
        other = draws + 2 * c["samples"] * c["walkers"]
    else:
        draws = other = 0
        for job, size, length, fanouts in _mix(c):
            draws += size * length if job == "rw" else size * sum(G.hop_widths(fanouts)) if job == "khop" else 10_000
            other += 2 * size if job != "mrw" else 10_000 + 4_000
    return dict(bytes=4 * (draws + other) + min(20 * draws, graph), flops=0)


# ---- the same samples from the uncompressed rows, in 64-bit integers ----

def _mul(a, b):
    """High and low word of the 64-bit product of 32-bit words (int64 tensors)."""
    p, q = a * (b & 0xFFFF), a * (b >> 16)
    return (q + (p >> 16)) >> 16, (((q & 0xFFFF) << 16) + p) & 0xFFFFFFFF


def _philox(seed, x0, x1, tag):
    """Philox4x32-10 of key `seed` and counter (x0, x1, 0, tag)."""
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    x2 = torch.zeros_like(x1)
    x3 = torch.full_like(x1, tag)
    for _ in range(10):
        h0, l0 = _mul(x0, 0xD2511F53)
        h1, l1 = _mul(x2, 0xCD9E8D57)
        x0, x1, x2, x3 = h1 ^ x1 ^ k0, l1, h0 ^ x3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return torch.stack((x0, x1, x2, x3))


def _neighbor(rowptr, cols, v, word):
    """The neighbor of v that a random word picks (every vertex of these graphs has one)."""
    return cols[rowptr[v] + _mul(word, rowptr[v + 1] - rowptr[v])[0]].long()


def exact(case, seed):
    c, kind, gen = case, case["kind"], _gen(seed)
    if kind == "decode":
        return [_room(c, x) for x in _rmat(c["scale"], c["ef"], seed)]
    if kind in ("n2v", "batch") or kind == "mrw" and c["select"] != G.SELECT_UNIFORM:
        return None
    rowptr, cols = _csr(c["scale"], c["ef"])
    n = rowptr.numel() - 1
    if kind in ("rw", "rw_host"):
        w = c["walkers"]
        v = (_vertices(n, (w,), gen) if kind == "rw" else
             torch.from_numpy(np.random.default_rng(seed).integers(0, n, w, dtype=np.uint32)).to(DEV)).long()
        ids, path = torch.arange(w, device=DEV), [v]
        for s in range(c["length"]):
            if s % 4 == 0:
                words = _philox(seed, torch.full_like(ids, s >> 2), ids, 0x52570001)
            path.append(_neighbor(rowptr, cols, path[-1], words[s % 4]))
        paths = torch.stack(path).to(torch.int32)
        paths = paths.T.contiguous() if c["layout"] == WALK else paths
        return [paths, torch.tensor([w * c["length"]])] if kind == "rw" else (paths, w * c["length"])
    if kind in ("khop", "khop_edges"):
        s = c["seeds"]
        v = _vertices(n, (s,), gen)[:, None].long()
        hops, src = [], []
        for h, f in enumerate(_fanouts(c)):
            v = v.repeat_interleave(f, 1)
            src.append(v.to(torch.int32).reshape(-1))
            slot = torch.arange(v.shape[1], device=DEV).repeat(s)
            ids = torch.arange(s, device=DEV).repeat_interleave(v.shape[1])
            word = _philox(seed, slot >> 2, ids, 0x4B480000 | h).gather(0, (slot & 3)[None])[0]
            v = _neighbor(rowptr, cols, v.reshape(-1), word).reshape(v.shape)
            hops.append(v.to(torch.int32))
        edges = [torch.cat(src), torch.cat([h.reshape(-1) for h in hops])] if kind == "khop_edges" else []
        return [*hops, *edges, torch.tensor([sum(h.numel() for h in hops)])]
    s, r = c["samples"], c["walkers"]
    v = _vertices(n, (s, r), gen).long()
    ids, src, dst = torch.arange(s, device=DEV), [], []
    for t in range(c["steps"]):
        words = _philox(seed, torch.full_like(ids, t), ids, 0x4D520001)
        x = _mul(words[0], torch.tensor(r, device=DEV))[0]
        src.append(v[ids, x])
        dst.append(_neighbor(rowptr, cols, src[-1], words[1]))
        v[ids, x] = dst[-1]
    return [v.to(torch.int32), *(torch.stack(e, 1).to(torch.int32) for e in (src, dst)),
            torch.tensor([s * c["steps"]])]
