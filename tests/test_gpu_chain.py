"""Searches along rings and paths of consecutive ids (the look-ahead of the
asynchronous mode, bfs.cuh): stretches one id shorter than, as long as and
longer than a warp looks ahead, up and down, past hubs and to both ends of the
id range; exact labels against the oracle's Tarjan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stretches(length, down, hubs, V=80000, tail=3000, seed=1):
    """One ring over stretches of `length` consecutive ids in random order, two
    paths hanging off it (one in, one out), short side edges; hubs: every 97th
    vertex of the ring has 40 more edges ahead of its own stretch."""
    rng = np.random.default_rng(seed)
    n = V - 2 * tail
    ids = np.arange(tail, tail + n)
    starts = np.arange(0, n, length)
    order = rng.permutation(len(starts))
    ring = np.concatenate([ids[starts[k]:starts[k] + length] for k in order])
    if down:
        ring = ring[::-1]
    S, D = [ring], [np.roll(ring, -1)]
    out, into = np.arange(tail), np.arange(V - tail, V)  # both ends of the id range
    for p in (out, into):
        S.append(p[:-1])
        D.append(p[1:])
    S += [ring[5:6], into[-1:]]
    D += [out[:1], ring[9:10]]
    if hubs:
        h = np.repeat(ring[::97], 40)
        S.append(h)
        D.append(out[rng.integers(0, tail, len(h))])
    S, D = np.concatenate(S), np.concatenate(D)
    o = rng.permutation(len(S))
    return V, S[o], D[o]


@pytest.mark.parametrize("length", [1, 2, 14, 15, 16, 17, 31, 33, 74000])
@pytest.mark.parametrize("down", [False, True])
@pytest.mark.parametrize("hubs", [False, True])
def test_stretches(length, down, hubs):
    import oracle
    from ispan_b200 import Context
    from ispan_b200.graphs import from_edges
    V, s, d = _stretches(length, down, hubs)
    csr = from_edges(V, np.stack([s, d], 1))
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for pair in (1, -1):
            ctx.set_tuning(pair_searches=pair)
            for graph in (True, False):
                labels, st = ctx.run_csr(csr, use_graph=graph)
                assert np.array_equal(labels, exact)
                assert st["giant_size"] == 74000
                assert st["fw_size"] == 74000 + 2999  # (the last of the path out is trimmed)


@pytest.mark.parametrize("second", [1400, 3000, 14999])
def test_ebbing_search(second):
    """A bottom-up level that found few beside what stays unreached hands them
    to the top-down queue (from both dense and sparse words of the visit map)."""
    import oracle
    from ispan_b200 import Context
    from ispan_b200.graphs import from_edges
    leaves, third, pairs = 60000, 200, 100000
    leaf = 1 + np.arange(leaves)
    two = 1 + leaves + np.arange(second)
    three = 1 + leaves + second + np.arange(third)
    rest = 1 + leaves + second + third + np.arange(2 * pairs)
    V = 1 + leaves + second + third + 2 * pairs
    up = [(np.zeros(leaves, int), leaf), (leaf[::4][:second], two), (two[:third], three), (rest[::2], rest[1::2])]
    S = np.concatenate([x for a, b in up for x in (a, b)])
    D = np.concatenate([x for a, b in up for x in (b, a)])
    p = np.arange(V)
    p[leaves:] = leaves + np.random.default_rng(2).permutation(V - leaves)
    csr = from_edges(V, np.stack([p[S], p[D]], 1))
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for pair in (1, -1):
            ctx.set_tuning(pair_searches=pair)
            for graph in (True, False):
                labels, st = ctx.run_csr(csr, use_graph=graph)
                assert np.array_equal(labels, exact)
                assert st["giant_size"] == st["fw_size"] == 1 + leaves + second + third


@pytest.mark.parametrize("mixed,run", [(7, 100), (8, 100), (9, 64), (31, 33), (32, 200), (33, 100), (300, 700)])
def test_stretches_after_shuffled_ids(mixed, run):
    """Stretches of consecutive ids with `mixed` vertices of shuffled ids between
    them: levels that look ahead in vain, then seldom, and find links again."""
    import oracle
    from ispan_b200 import Context
    from ispan_b200.graphs import from_edges
    V = 90_000
    rng = np.random.default_rng(mixed)
    k = V // (mixed + run)
    near = np.arange(k * run).reshape(k, run)
    far = rng.permutation(np.arange(k * run, k * (run + mixed))).reshape(k, mixed)
    ring = np.concatenate([np.concatenate([near[i], far[i]]) for i in rng.permutation(k)])
    csr = from_edges(V, np.stack([ring, np.roll(ring, -1)], 1))
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for graph in (False, True, True):
            labels, st = ctx.run_csr(csr, use_graph=graph)
            assert np.array_equal(labels, exact)
            assert st["giant_size"] == len(ring)
