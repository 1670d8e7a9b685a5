"""The contraction of cycles along near ids (cycles.cuh) on graphs large enough
to reach it (32,768 residual vertices in WCCs above the tiles' size): labels,
the size histogram and the SCC count against the oracle's Tarjan.  A node's
size is read from the histogram, and by the peel of the nodes as the length of
its slice of the node order."""
import numpy as np
import pytest

from test_gpu_resolve import _csr

pytestmark = pytest.mark.gpu

CYC_MIN = 32768  # residual vertices from which cycles are looked for


def _gadgets(count, size, edges, dag, seed, order):
    """`count` copies of a gadget (edges among ids [0, size)), joined into one
    WCC by a line and `dag` random edges from earlier to later copies, beside a
    hub graph (the pivot's SCC).  The copies' ids: in the order of the DAG
    ("up"), against it ("down"), or at random ("blocks", where no span of
    descending edges ends a node and the peel runs)."""
    rng = np.random.default_rng(seed)
    e = np.array(edges)
    place = {"up": np.arange(count), "down": np.arange(count)[::-1], "blocks": rng.permutation(count)}[order]
    base = place * size
    x, y = rng.integers(0, count, dag), rng.integers(0, count, dag)
    x, y = np.minimum(x, y), np.maximum(x, y)
    keep = x < y
    x, y = x[keep], y[keep]
    S = [(base[:, None] + e[None, :, 0]).ravel(), base[:-1], base[x] + rng.integers(0, size, len(x))]
    D = [(base[:, None] + e[None, :, 1]).ravel(), base[1:], base[y] + rng.integers(0, size, len(y))]
    n, h = count * size, 1200
    S += [np.full(h, n), n + 1 + np.arange(h)]
    D += [n + 1 + np.arange(h), np.full(h, n)]
    return _csr(n + h + 1, np.concatenate(S), np.concatenate(D))


def _check(csr, runs=3):
    import oracle
    from ispan_b200 import Context
    exact = oracle.tarjan(csr)
    hist = oracle.histogram(exact)
    with Context(csr.V, csr.E) as ctx:
        for k in range(runs):
            labels, st = ctx.run_csr(csr, histogram=True, use_graph=k % 3 != 2)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == hist
            assert st["scc_count"] == len(np.unique(exact))
            assert st["n_mice_vertices"] >= CYC_MIN  # cycles were looked for


def _ring_down(lo, hi):
    """A ring whose edges lead to the id before: its minimum's nearest
    in-neighbour is the id after it."""
    return [(i + 1, i) for i in range(lo, hi)] + [(lo, hi)]


# a descending ring whose minimum lies on a way of single vertices back to the
# ring (they are joined to it, and its size counts), and two such rings joined
# both ways through their minima
ASCENDING = {
    "way": (56, _ring_down(5, 55) + [(i, i + 1) for i in range(4)] + [(4, 7), (6, 0)]),
    "minima": (80, _ring_down(0, 39) + _ring_down(40, 79) + [(0, 40), (40, 0)]),
    "two": (60, _ring_down(2, 57) + [(0, 1), (1, 0), (1, 2), (2, 58), (58, 59), (59, 2)]),
}


@pytest.mark.parametrize("name", list(ASCENDING))
@pytest.mark.parametrize("order", ["up", "down", "blocks"])
def test_minimum_that_leads_up(name, order):
    size, edges = ASCENDING[name]
    _check(_gadgets(1500, size, edges, dag=9000, seed=len(name), order=order))


# a ring of several vertices with the lowest ids, from which a way of two (or
# more) single vertices leads back to it: the cycle of nodes has its lowest id
# in the ring and several single vertices that could each walk it.  Their ids
# follow the way, run against it, or lie apart (rings between them)
_RING = [(i, i + 1) for i in range(7)] + [(7, 0)]
WAYS = {
    "along": (10, _RING + [(7, 8), (8, 9), (9, 0)]),
    "against": (10, _RING + [(7, 9), (9, 8), (8, 0)]),
    "apart": (19, _RING + [(7, 8), (8, 18), (18, 0)] + [(i, i + 1) for i in range(9, 17)] + [(17, 9)]),
}


@pytest.mark.parametrize("name", list(WAYS))
@pytest.mark.parametrize("order", ["up", "blocks"])
def test_ways_back_to_the_lowest_ring(name, order):
    """More single vertices (above 200,000) than threads, so that walks begin
    at different times, over and over in one context."""
    size, edges = WAYS[name]
    _check(_gadgets(101_000, size, edges, dag=300_000, seed=len(name), order=order), runs=50)


@pytest.mark.parametrize("order", ["up", "down", "blocks"])
@pytest.mark.parametrize("copies", [1, 40])
def test_spans_of_many_edges(order, copies):
    """Vertices with many edges against the order, near and far, each `copies`
    times: a vertex has one span, to the farthest."""
    rng = np.random.default_rng(copies)
    csr = _gadgets(900, 40, [(i, (i + 1) % 40) for i in range(40)], dag=4000, seed=5, order=order)
    src = np.repeat(np.arange(csr.V), np.diff(csr.fw_beg))
    n = 900 * 40
    # back edges over spans of up to 60 rings, from few vertices
    v = rng.integers(0, n, 150).repeat(12)
    w = np.maximum(0, v - rng.integers(0, 2400, len(v)))
    csr = _csr(csr.V, np.concatenate([src, np.tile(v, copies)]), np.concatenate([csr.fw_adj, np.tile(w, copies)]))
    _check(csr)


@pytest.mark.parametrize("ring", ["up", "down"])
@pytest.mark.parametrize("order", ["up", "down"])
def test_line_of_rings_either_way(ring, order):
    """A line of 20,000 rings, its ids along it or against it, whatever way the
    rings' own edges lead: ended by the spans (about 1 ms), not by a peel of
    10,000 rounds (430 ms)."""
    import time
    from ispan_b200 import Context
    L = 30
    edges = [(i, (i + 1) % L) for i in range(L)]
    csr = _gadgets(20_000, L, edges if ring == "up" else [(b, a) for a, b in edges], dag=0, seed=1, order=order)
    _check(csr)
    with Context(csr.V, csr.E) as ctx:
        ctx.run_csr(csr)
        t = time.perf_counter()
        ctx.run_csr(csr)
        assert time.perf_counter() - t < 0.05


# walks that lead into cycles they are not on, or up a long way: gadgets of a ring
# and a vertex below it, alone and in a line whose ids ascend
@pytest.mark.parametrize("line", [False, True])
@pytest.mark.parametrize("step", [1, 7])
def test_walks_beside_rings(line, step):
    import time
    from ispan_b200 import Context
    L, k = 20, 50_000
    edges = [(1 + i, 1 + (i + step) % L) for i in range(L)] + [(5, 0)] + ([] if line else [(0, 7)])
    size = L + 1
    if line:  # the vertex below leads to the ring of the copy before
        e = np.array(edges)
        base = np.arange(k) * size
        S = [(base[:, None] + e[None, :, 0]).ravel(), base[1:], [0], [k * size]]
        D = [(base[:, None] + e[None, :, 1]).ravel(), base[:-1] + 3, [3], [k * size]]
        h = 1200
        n = k * size
        S += [np.full(h, n), n + 1 + np.arange(h)]
        D += [n + 1 + np.arange(h), np.full(h, n)]
        csr = _csr(n + h + 1, np.concatenate(S), np.concatenate(D))
    else:
        e = np.array(edges)
        base = np.arange(k) * size
        n, h = k * size, 1200
        csr = _csr(n + h + 1, np.concatenate([(base[:, None] + e[None, :, 0]).ravel(), np.full(h, n), n + 1 + np.arange(h)]),
                   np.concatenate([(base[:, None] + e[None, :, 1]).ravel(), n + 1 + np.arange(h), np.full(h, n)]))
    _check(csr)
    with Context(csr.V, csr.E) as ctx:
        ctx.run_csr(csr)
        t = time.perf_counter()
        ctx.run_csr(csr)
        assert time.perf_counter() - t < 0.1  # (the line with ids as priorities: 0.3 s and more)


# rings of about kCycMax runs of consecutive ids (every second id, two rings
# interleaved), and cycles of about kCycMax nodes (rings of four and single
# vertices in turn), just below, at and above the longest walk; edges up and down
@pytest.mark.parametrize("length", [4095, 4096, 4097, 4098])
@pytest.mark.parametrize("down", [False, True])
def test_longest_walks_of_runs(length, down):
    i = np.arange(length)
    edges = [(int(2 * a + p), int(2 * ((a + 1) % length) + p)) for p in (0, 1) for a in i] + [(0, 1)]
    if down:
        edges = [(b, a) for a, b in edges]
    _check(_gadgets(6, 2 * length, edges, dag=20, seed=length, order="blocks"))


@pytest.mark.parametrize("pairs", [2046, 2047, 2048, 2049])
@pytest.mark.parametrize("down", [False, True])
@pytest.mark.parametrize("order", ["up", "blocks"])
def test_longest_walks_of_nodes(pairs, down, order):
    edges = []
    for k in range(pairs):
        b, nxt = 5 * k, 5 * ((k + 1) % pairs)
        edges += [(b, b + 1), (b + 1, b + 2), (b + 2, b + 3), (b + 3, b), (b + 3, b + 4), (b + 4, nxt)]
    if down:
        edges = [(b, a) for a, b in edges]
    _check(_gadgets(5, 5 * pairs, edges, dag=20, seed=pairs, order=order))
