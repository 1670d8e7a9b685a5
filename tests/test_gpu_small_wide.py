"""Frontiers of the one-cluster kernel (small.cuh) that widen at once, stay
narrow, or do both: exact labels; on graphs whose frontier widens at once, not
slower than the stage kernels (whose route runs with stage times take)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(V, E):
    rng = np.random.default_rng(V + E)
    return V, rng.integers(0, V, E), rng.integers(0, V, E)


def _grid(k, seed):
    i = np.arange(k * k)
    r, d = i[i % k < k - 1], i[:-k]
    p = np.random.default_rng(seed).permutation(k * k) if seed else i
    return k * k, p[np.concatenate([r, d, r + 1, d + k])], p[np.concatenate([r + 1, d + k, r, d])]


def _broom(n, m, width):
    """A ring of n, at one place of which m paths of two lead around an edge of it,
    `width` of them for each of the next places."""
    S, D = [np.arange(n)], [(np.arange(n) + 1) % n]
    at = np.repeat(np.arange(m // width) % n, width)
    mid = n + np.arange(len(at))
    S += [at, mid]
    D += [mid, (at + 1) % n]
    return n + len(at), np.concatenate(S), np.concatenate(D)


GRAPHS = {
    "uniform 8k": _uniform(8000, 500_000), "uniform 30k": _uniform(30_000, 1_000_000),
    "uniform 65k": _uniform(65_000, 1_000_000), "dense 65k": _uniform(65_000, 4_000_000),
    "grid": _grid(250, 0), "grid at random": _grid(250, 3),
    # as wide as the limit (1,024) and one to each side of it
    **{f"broom {w}": _broom(2000, 40_000, w) for w in (64, 1023, 1024, 1025, 4000)},
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_wide_and_narrow(name):
    import oracle
    import torch
    from ispan_b200 import Context
    from test_gpu_resolve import _csr
    csr = _csr(*GRAPHS[name])
    exact = oracle.tarjan(csr)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = [t(a) for a in (csr.fw_beg, csr.fw_adj, csr.bw_beg, csr.bw_adj)]
    lab = torch.empty(csr.V, dtype=torch.int32, device="cuda")
    ms = {}
    with Context(csr.V, csr.E) as ctx:
        for stages in (False, True):
            ts = []
            for _ in range(12):
                lab.fill_(-1)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                ctx.run(*g, labels_out=lab, stage_times=stages)
                ts.append(time.perf_counter() - t0)
                assert np.array_equal(lab.cpu().numpy(), exact)
            ms[stages] = sorted(ts)[len(ts) // 2] * 1e3
    # (uniform graphs took 1.5 to 4 times the stage kernels' time while each CTA went on by itself)
    if "uniform" in name or "dense" in name:
        assert ms[False] < 1.2 * ms[True], ms
