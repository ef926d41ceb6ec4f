"""Allocations of the PageRank family's shared structures (renumbering, CSC, its merge): each in
turn fails once during a run. The run reports that it is out of memory and the same call, repeated,
gives the ranks of an undisturbed context; results may be asked for in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = ["PageRank", "PageRankDelta", "WeightedPageRank"]


def program(cg, eng, form):
    if form == "PageRankDelta":
        return cg.PageRankDelta(eng, delta=0.0, max_iterations=1000, tolerance=1e-9)
    return getattr(cg, form)(eng, max_iterations=1000, tolerance=1e-10, kahan=True)


def disturbed(cg, eng, p, k):
    """Runs p with its k-th allocation failing; True once the run has fewer than k."""
    eng.set_fault_injection(fail_alloc_after=k)
    try:
        p.execute_algorithm()
    except cg.CytomError as e:
        assert e.code == -2
        p.result()  # whatever it holds: it must not reach for what is not there
        p.execute_algorithm()
        return False
    finally:
        eng.set_fault_injection()
    return True


@pytest.mark.parametrize("form", FORMS)
def test_first_build(cg, form):
    n = 1 << 14  # sorts of the vertices take scratch of their own
    rng = np.random.default_rng(1)
    s, t = rng.integers(0, n - 99, 60000, dtype=np.uint32), rng.integers(0, n, 60000, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s)).astype(np.float32).view(np.uint32) if form == "WeightedPageRank" else None
    ref, quiet = None, 0
    for k in range(0, 60):
        with cg.Engine(n, 4096, weight_type=cg.WEIGHT_F32 if w is not None else cg.UNWEIGHTED) as eng:
            eng.insert_edges(s, t, w)
            eng.do_global_compaction()
            p = program(cg, eng, form)
            done = disturbed(cg, eng, p, k)
            r = np.asarray(p.result(), np.float64)
        if ref is None:
            ref = r
        assert np.abs(r - ref).sum() <= 1e-6 * np.abs(ref).sum(), k
        quiet = quiet + 1 if done and k else 0
        if quiet == 2:
            break
    assert quiet == 2 and k > 10


@pytest.mark.parametrize("form", FORMS[:2])
def test_merge_of_a_second_batch(cg, form):
    """2^21 edges and more: the CSC of the second snapshot is merged from the first one's."""
    n = 1 << 16
    rng = np.random.default_rng(2)
    m = 2300000
    s, t = rng.integers(0, n - 99, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32)
    s2, t2 = rng.integers(0, n - 99, 50000, dtype=np.uint32), rng.integers(0, n, 50000, dtype=np.uint32)
    ref, quiet = None, 0
    for k in range(0, 40):
        with cg.Engine(n, 65536) as eng:
            eng.insert_edges(s, t)
            eng.do_global_compaction()
            p = program(cg, eng, form)
            p.execute_algorithm()
            eng.insert_edges(s2, t2)
            eng.do_global_compaction()
            done = disturbed(cg, eng, p, k)
            r = np.asarray(p.result(), np.float64)
        if ref is None:
            ref = r
        assert np.abs(r - ref).sum() <= 1e-6 * np.abs(ref).sum(), k
        quiet = quiet + 1 if done and k else 0
        if quiet == 2:
            break
    assert quiet == 2 and k > 3
