"""The out-edge estimate that picks the kind of a round depends on the snapshot alone: on small
graphs it holds every listed word whichever kernel lists them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_graph_scans_the_same_edges_profiled(cg):
    """2^15 pairs (v, v + 1), then 10,000 edges that lower one end of a pair each: the active
    vertices hold more than an eighth of the edges but few of them lie in any 129 words."""
    n = 1 << 16
    even = np.arange(0, n, 2, dtype=np.uint32)
    rng = np.random.default_rng(5)
    low = rng.permutation(even[100:])[:10000].astype(np.uint32)
    got = []
    for profiled in (False, True):
        with cg.Engine(n, 1024) as eng:
            eng.insert_edges(even, even + 1)
            cc = cg.CC(eng, max_iterations=1000)
            cc.execute_algorithm()
            eng.insert_edges(np.zeros(len(low), np.uint32), low)
            eng.set_profiling(profiled)
            x = cc.execute_algorithm()
            eng.set_profiling(False)
            got.append((x["iterations"], x["count_edges"], x["edges_scanned"], cc.result().tobytes()))
    assert got[0] == got[1]
