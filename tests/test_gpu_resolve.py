"""The splitting, tile and labelling kernels of the large WCCs (resolve.cuh) on
graphs whose residual is built to reach their edges, and the cycles along near
ids (cycles.cuh): components one vertex
below, at and above the tile sizes, lists longer than a lane reads alone, a
component too dense for a tile, duplicate edges and self-loops; exact labels
against the oracle's Tarjan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst):
    from ispan_b200.graphs import CSR
    o = np.lexsort((dst, src))
    s, d = src[o], dst[o]
    fb = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=V))]).astype(np.int64)
    o = np.lexsort((src, dst))
    bb = np.concatenate([[0], np.cumsum(np.bincount(dst, minlength=V))]).astype(np.int64)
    return CSR(V, len(src), fb, d.astype(np.int32), bb, src[o].astype(np.int32))


def _blocks(sizes, dag, seed, scramble, chords=0.5, dense=0, join=True):
    """SCCs of the given sizes (ring and chords) in a line, joined by random
    edges from earlier to later ones into one WCC, beside a strongly connected
    hub graph (the pivot's SCC) and isolated vertices (four times the rest)."""
    rng = np.random.default_rng(seed)
    sizes = np.array(sizes)
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    of = np.repeat(np.arange(len(sizes)), sizes)
    nxt = np.arange(1, n + 1)
    nxt[off[1:] - 1] = off[:-1]
    S, D = [np.arange(n)], [nxt]
    c = rng.integers(0, n, int(n * chords))
    S.append(c)
    D.append(off[of[c]] + rng.integers(0, sizes[of[c]]))
    x, y = rng.integers(0, n, dag), rng.integers(0, n, dag)
    swap = of[x] > of[y]
    S += [np.where(swap, y, x), np.arange(0, n, 97)]  # (the last: self-loops)
    D += [np.where(swap, x, y), np.arange(0, n, 97)]
    if join:  # one WCC
        S.append(off[:-2])
        D.append(off[1:-1])
    if dense:  # the first block is dense, and a hub with long lists both ways
        S += [rng.integers(0, sizes[0], dense), np.zeros(300, int), rng.integers(0, sizes[0], 300)]
        D += [rng.integers(0, sizes[0], dense), rng.integers(0, n if join else sizes[0], 300), np.zeros(300, int)]
    S.append(S[2][:500])  # duplicates
    D.append(D[2][:500])
    h = 1200  # the hub graph: one vertex to and from all others
    S += [np.full(h, n), n + 1 + np.arange(h)]
    D += [n + 1 + np.arange(h), np.full(h, n)]
    V = 5 * (n + h + 1)
    S, D = np.concatenate(S), np.concatenate(D)
    if scramble:
        p = rng.permutation(V)
        S, D = p[S], p[D]
    return _csr(V, S, D)


# WCCs below, at and above the limit of the shared-memory path, tiles whose
# edges overflow (solved WCC by WCC) and a WCC whose own do (spilled)
SMALL = {
    "limits": dict(sizes=[4095, 4096, 4097, 8192, 8193, 2, 3, 1] + [4] * 700, dag=0),
    "one tile": dict(sizes=[9, 5, 4], dag=0),
    "dense": dict(sizes=[100] * 12, dag=0, chords=400.0),
    "overflow": dict(sizes=[100] * 12, dag=0, chords=500.0),
    "chords": dict(sizes=[1000] * 30, dag=0, chords=9.0),
}

CASES = {
    "tile edges": dict(sizes=[2, 3, 1, 4095, 4096, 4097, 8191, 8192, 8193, 10000, 33] + [40] * 500, dag=60000),
    "small": dict(sizes=[10] * 8000 + [700, 900], dag=160000),
    "dense and hub": dict(sizes=[600] + [25] * 3000, dag=120000, dense=30000),
    "rings": dict(sizes=[1000] * 90 + [7] * 100, dag=150000, chords=0.0),
    "long ring": dict(sizes=[70000, 5, 5], dag=30, chords=0.0),
    "nothing joins": dict(sizes=[3000] * 30, dag=0),
}


def _renumber(csr, order):
    """csr with vertex order[i] renamed i."""
    to = np.empty(csr.V, np.int64)
    to[order] = np.arange(csr.V)
    src = np.repeat(np.arange(csr.V), np.diff(csr.fw_beg))
    return _csr(csr.V, to[src], to[csr.fw_adj])


# ids along the rings: rings in topological order, in the reverse of it and in
# random order (where only the peel of the contracted rings ends them), rings
# with chords, one longer than the longest walk, a closing edge that is not
# the nearest in-edge, and ids without locality inside some blocks
NEAR = {
    "order": dict(sizes=[300] * 60 + [2, 3, 900, 1], dag=30000, chords=0.0),
    "chords": dict(sizes=[40] * 300, dag=20000, chords=0.3),
    "pairs": dict(sizes=[2] * 4000, dag=12000, chords=0.0),
    "long": dict(sizes=[20000, 30, 16384, 16385, 500], dag=40000, chords=0.0),
    "few": dict(sizes=[900] * 6, dag=11000, chords=0.02),
}


@pytest.mark.parametrize("name", list(NEAR))
@pytest.mark.parametrize("ids", ["up", "down", "blocks", "mixed"])
def test_cycles_along_ids(name, ids):
    import oracle
    from ispan_b200 import Context
    c = NEAR[name]
    csr = _blocks(seed=len(name), scramble=False, **c)
    rng = np.random.default_rng(7)
    n = sum(c["sizes"])
    order = np.arange(csr.V)
    if ids == "down":
        order[:n] = order[:n][::-1]
    elif ids == "blocks":
        off = np.concatenate([[0], np.cumsum(c["sizes"])])
        perm = rng.permutation(len(c["sizes"]))
        order[:n] = np.concatenate([np.arange(off[k], off[k + 1]) for k in perm])
    elif ids == "mixed":
        order[:n // 3] = rng.permutation(n // 3)
    csr = _renumber(csr, order)
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for graph in (True, False):
            labels, st = ctx.run_csr(csr, histogram=True, use_graph=graph)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == oracle.histogram(exact)
            assert st["scc_count"] == len(np.unique(exact))


@pytest.mark.parametrize("name", list(SMALL))
@pytest.mark.parametrize("graph", [False, True])
def test_small_wccs(name, graph):
    import oracle
    from ispan_b200 import Context
    csr = _blocks(seed=len(name), scramble=True, join=False, **SMALL[name])
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        labels, st = ctx.run_csr(csr, histogram=True, use_graph=graph)
    assert np.array_equal(labels, exact)
    assert st["histogram"] == oracle.histogram(exact)
    assert st["local_wcc"] == st["n_wcc"] - {"limits": 1, "overflow": 12}.get(name, 0)


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("scramble", [False, True])
def test_exact_labels(name, scramble):
    import oracle
    from ispan_b200 import Context
    csr = _blocks(seed=len(name), scramble=scramble, **CASES[name])
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for _ in range(2):
            labels, st = ctx.run_csr(csr, histogram=True)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == oracle.histogram(exact)
            assert st["scc_count"] == len(np.unique(exact))
            assert st["n_mice_vertices"] >= 65536  # the large-WCC path ran


# a component left to splitting and labelling just at and just above the size
# up to which values spread over links, with ids along its ring (chords make
# it several rings), against them and at random
@pytest.mark.parametrize("size", [262144, 262145])
@pytest.mark.parametrize("ids", ["up", "down", "mixed"])
def test_links(size, ids):
    import oracle
    from ispan_b200 import Context
    csr = _blocks([size, 3, 500], dag=200, seed=3, scramble=ids == "mixed", chords=0.02)
    if ids == "down":
        csr = _renumber(csr, np.arange(csr.V)[::-1])
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for graph in (True, False):
            labels, st = ctx.run_csr(csr, histogram=True, use_graph=graph)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == oracle.histogram(exact)
