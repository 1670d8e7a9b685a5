"""Labelling rounds of tiles and of k_resolve: lines of SCCs whose low ids lie
at both ends, where the ranks of the ids as labels end one SCC a round.  The
model of the rule in test_rounds_of_a_line (CPU) counts the rounds; on the
GPU every label is checked, and the time is held to what that many rounds of a
tile take (a round of 2,000 rings: about 1.7 ms with ranks alone, 3.4 s in all)."""
import time

import numpy as np
import pytest


def _ends(k):
    """Place in the line -> id: even ids from the left end, odd ones from the right."""
    j = np.arange(k)
    ids = np.empty(k, int)
    ids[np.where(j % 2 == 0, j // 2, k - 1 - j // 2)] = j
    return ids


def _mix(rnd, bits):
    """LabelMix (tile.cuh): labels of the numbers below 2^bits in a round."""
    word, mask = 0xffffffff, (1 << bits) - 1
    a = (0x9e3779b1 * (2 * rnd + 1)) & word | 1
    b = ((0x9e3779b1 * (2 * rnd + 2)) & word) >> 5 | 1
    x = np.arange(1 << min(bits, 17), dtype=np.uint64)
    y = x if rnd < 3 else (x * np.uint64(a)) & np.uint64(mask)
    return x if rnd < 3 else (((y ^ (y >> np.uint64((bits + 1) // 2))) * np.uint64(b)) & np.uint64(mask))


def _rounds(ids, bits):
    """Rounds until every SCC of a line is found: in each class the lowest label
    upstream (f) and downstream (b), found where they are equal."""
    left, n = [np.arange(len(ids))], 0
    while left:
        lab, nxt = _mix(n, bits)[ids].astype(np.int64), []
        for s in left:
            f = np.minimum.accumulate(lab[s])
            b = np.minimum.accumulate(lab[s][::-1])[::-1]
            keep = f != b
            cut = np.flatnonzero((f[1:] != f[:-1]) | (b[1:] != b[:-1]) | ~keep[1:] | ~keep[:-1]) + 1
            nxt += [p for p, k in zip(np.split(s, cut), np.split(keep, cut)) if k[0]]
        left, n = nxt, n + 1
    return n


def test_rounds_of_a_line():
    for bits in (13, 32):
        for rnd in range(3, 40):
            x = _mix(rnd, bits)
            assert len(np.unique(x)) == len(x)
        for k in (10, 100, 500, 2000):
            assert _rounds(_ends(k), bits) <= 25
            assert _rounds(np.arange(k), bits) <= 3  # ids along the line: as with ranks


# in tiles (components up to 8,192 vertices), alone and as one of several; and
# above them (the line is then split first)
@pytest.mark.gpu
@pytest.mark.parametrize("k,copies", [(10, 40), (500, 1), (500, 9), (2000, 1), (2048, 3), (2500, 1), (20000, 1)])
def test_low_ids_at_both_ends(k, copies):
    import oracle
    from ispan_b200 import Context
    from test_gpu_resolve import _csr
    base = (4 * (_ends(k)[None, :] + k * np.arange(copies)[:, None]))
    n, h = 4 * k * copies, 1200
    first = base.ravel()
    S = [first, first + 1, first + 2, first + 3, base[:, :-1].ravel(), np.full(h, n), n + 1 + np.arange(h)]
    D = [first + 1, first + 2, first + 3, first, base[:, 1:].ravel(), n + 1 + np.arange(h), np.full(h, n)]
    csr = _csr(5 * (n + h + 1), np.concatenate(S), np.concatenate(D))
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for graph in (True, False):
            labels, st = ctx.run_csr(csr, histogram=True, use_graph=graph)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == oracle.histogram(exact)
        t = time.perf_counter()
        ctx.run_csr(csr)
        if copies == 1 and k <= 2000:  # one tile: 25 rounds of at most 2 ms
            assert time.perf_counter() - t < 0.1


# one SCC outside the pivot's whose diameter is hundreds of edges, below and
# above the size up to which values spread over links: masks of pivots say
# nothing on it, and are given up within the first round
@pytest.mark.gpu
@pytest.mark.parametrize("k", [400, 600])
@pytest.mark.parametrize("ids", ["rows", "mixed"])
def test_masks_given_up(k, ids):
    import oracle
    from ispan_b200 import Context
    from test_gpu_resolve import _csr
    i = np.arange(k * k)
    r, d = i[i % k < k - 1], i[:-k]
    n, h = k * k, 1200
    S, D = np.concatenate([r, d, r + 1, d + k]), np.concatenate([r + 1, d + k, r, d])
    if ids == "mixed":
        p = np.random.default_rng(k).permutation(n)
        S, D = p[S], p[D]
    csr = _csr(5 * (n + h + 1), np.concatenate([S, np.full(h, n), n + 1 + np.arange(h)]),
               np.concatenate([D, n + 1 + np.arange(h), np.full(h, n)]))
    exact = oracle.tarjan(csr)
    with Context(csr.V, csr.E) as ctx:
        for graph in (True, False):
            labels, st = ctx.run_csr(csr, histogram=True, use_graph=graph)
            assert np.array_equal(labels, exact)
            assert st["histogram"] == oracle.histogram(exact)
            assert st["color_rounds"] <= 2  # (4 to 8 before)
