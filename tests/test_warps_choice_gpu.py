"""The launch rule's choice of warps per query against every choice a caller can
make: no call takes half as long again as with the best one. (Residents counted as
the launch takes them; a rule that counted more ran such batches in two waves, 1.7 and
1.8 times the best.) Kernel times, the shortest of five."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,deg,M,calls", [(128, 45, 8, [(2047, 1480), (1600, 1000), (100, 1000), (384, 3000)]),
                                           (96, 19, 8, [(1900, 1000), (2047, 1480), (384, 300), (608, 3000)]),
                                           (96, 19, 1, [(384, 500), (384, 2500)])])
def test_choice_is_near_the_best(d, deg, M, calls):
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.formats import NSGGraph
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(d)
    n = 100_000
    nb = rng.integers(0, n, size=(n, deg), dtype=np.int64)
    g = NSGGraph(deg, 0, np.arange(n + 1, dtype=np.int64) * deg, nb.reshape(-1).astype(np.uint32))
    with Index(0) as ix:
        ix.set_base(rng.random((n, d), dtype=np.float32))
        ix.set_graph(g)
        for L, nq in calls:
            q = rng.random((nq, d), dtype=np.float32)
            ms = {w: min(ix.search(q, K=10, L=L, mode=N.MODE_TOP_M, M=M, warps_per_query=w)[1]["kernel_ms"]
                         for _ in range(5)) for w in (0, 1, 2, 4, 8)}
            assert ms[0] <= 1.5 * min(ms.values()), (L, nq, ms)
