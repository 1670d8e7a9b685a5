"""Host graphs in ordinary memory, copied through pinned pieces by several
threads: totals just below and above the size where that starts, last pieces
of every array cut short, the same context for one graph after another; exact
labels against the oracle's Tarjan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("over", [-8, 0, 8, 9_000_008])
def test_ordinary_memory(dtype, over):
    import oracle
    from ispan_b200 import Context, graphs as G
    V = 200_001
    E = ((16 << 20) + over - 2 * (V + 1) * np.dtype(dtype).itemsize) // 8
    with Context(V, E) as ctx:
        for seed in (1, 2, 3):
            csr = G.random_graph(V, E, seed)
            if csr.fw_beg.dtype != dtype:
                csr = G.CSR(csr.V, csr.E, csr.fw_beg.astype(dtype), csr.fw_adj, csr.bw_beg.astype(dtype), csr.bw_adj)
            exact = oracle.tarjan(csr)
            labels, _ = ctx.run_csr(csr)
            for a in (csr.fw_beg, csr.fw_adj, csr.bw_beg, csr.bw_adj):
                a[:] = 0  # read by now
            assert np.array_equal(labels, exact)
