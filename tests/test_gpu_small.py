"""The one-cluster kernel of small graphs (small.cuh) at its edges: the largest
size and one beyond, words and CTA ranges that end early, lists read by a lane,
a warp and a CTA, queues that overflow, searches that push and pull, nothing
and something left after the peel, batches; exact labels against the oracle's
Tarjan and the stage kernels' counts (runs with exact statistics take those)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = ("scc_count", "giant_size", "n_trim1", "n_trim2", "n_trim3", "n_mice_scc", "n_mice_vertices", "residual",
          "fw_size")


def _rand(V, E, seed):
    rng = np.random.default_rng(seed)
    return V, rng.integers(0, max(V, 1), E), rng.integers(0, max(V, 1), E)


def _ring(V, seed=None):
    p = np.arange(V) if seed is None else np.random.default_rng(seed).permutation(V)
    return V, p, np.roll(p, -1)


def _path(V):
    return V, np.arange(V - 1), np.arange(1, V)


def _hubs(sizes, back):
    """Stars of the given sizes, centres on a ring; back: leaves lead back."""
    c = np.concatenate([[0], np.cumsum(np.array(sizes) + 1)])
    S, D = [c[:-1]], [np.roll(c[:-1], -1)]
    for a, n in zip(c, sizes):
        leaf = a + 1 + np.arange(n)
        S.append(np.full(n, a))
        D.append(leaf)
        S.append(leaf if back else leaf[:1])
        D.append(np.full(n if back else 1, a))
    return int(c[-1]), np.concatenate(S), np.concatenate(D)


def _islands(n, size, seed):
    """A hub ring, then rings of `size` in a line: left after the peel."""
    V, s, d = _ring(n * size, None)
    nxt = np.arange(1, V + 1)
    nxt[size - 1::size] -= size
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, V, n), rng.integers(0, V, n)
    h = V + np.arange(50)
    return V + 50, np.concatenate([np.arange(V), np.minimum(a, b), h, h, h[1:]]), \
        np.concatenate([nxt, np.maximum(a, b), np.roll(h, -1), np.roll(h, 1), h[:-1]])


GRAPHS = {
    **{f"random {V}": _rand(V, 3 * V, V) for V in (1, 2, 31, 32, 33, 511, 512, 513, 1000, 65535, 65536, 65537)},
    "no edges": (100, np.zeros(0, int), np.zeros(0, int)),
    "no vertices": (0, np.zeros(0, int), np.zeros(0, int)),
    "loops only": (70, np.arange(70), np.arange(70)),
    "dense": _rand(2000, 400000, 3),
    "ring": _ring(65536),
    "mixed ring": _ring(30000, 5),
    "path": _path(65536),
    "lists": _hubs([15, 16, 17, 4095, 4096, 4097, 20000], True),
    "leaves": _hubs([16, 17, 4097, 50000], False),
    "islands": _islands(3000, 20, 1),
    "few islands": _islands(3, 5, 2),
}


def _csr(V, s, d, dtype=np.int32):
    from ispan_b200.graphs import CSR
    s, d = np.asarray(s, np.int64), np.asarray(d, np.int64)
    fb = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=V))]).astype(dtype)
    bb = np.concatenate([[0], np.cumsum(np.bincount(d, minlength=V))]).astype(dtype)
    return CSR(V, len(s), fb, d[np.argsort(s, kind="stable")].astype(np.int32), bb,
               s[np.argsort(d, kind="stable")].astype(np.int32))


def _check(ctx, csr, exact, **kw):
    import oracle
    got = []
    for run in (dict(), dict(), dict(use_graph=False), dict(exact_stats=True)):
        labels, st = ctx.run_csr(csr, histogram=True, **run, **kw)
        assert np.array_equal(labels, exact)
        assert st["histogram"] == oracle.histogram(exact)
        got.append({k: st[k] for k in COUNTS})
    assert got[0] == got[1] == got[2] == got[3]


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_one_graph(name, dtype):
    import oracle
    from ispan_b200 import Context
    csr = _csr(*GRAPHS[name], dtype=dtype)
    with Context(max(csr.V, 1), max(csr.E, 1)) as ctx:
        _check(ctx, csr, oracle.tarjan(csr))


BATCHES = {
    "mixed": ["random 33", "no edges", "lists", "random 1000", "random 1", "few islands", "loops only"],
    "many": ["random 31", "random 2", "random 33"] * 500,
    "rings": ["few islands"] * 200,
    "one": ["random 1000"],
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_batch(name):
    import oracle
    from ispan_b200 import Context
    from ispan_b200 import graphs as G
    u, vb = G.disjoint_union([_csr(*GRAPHS[n]) for n in BATCHES[name]])
    with Context(u.V, max(u.E, 1)) as ctx:
        _check(ctx, u, oracle.tarjan(u), vbase=vb)
