"""Allocations of the store's updates, each in turn failing once: the call reports that it is out of
memory, leaves the graph as it was, and succeeds when repeated. Against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, VPT = 1 << 13, 1024


def batch(rng, m):
    return (rng.integers(0, N, m, dtype=np.uint32), rng.integers(0, N, m, dtype=np.uint32),
            rng.integers(1, 1000, m, dtype=np.uint32))


def disturbed(cg, eng, k, call, between=lambda: None):
    """call() with its k-th allocation failing; if it reports that, between() and call() again. False
    once the call has fewer allocations."""
    eng.set_fault_injection(fail_alloc_after=k)
    try:
        call()
    except cg.CytomError as e:
        assert e.code == -2
        between()
        call()
        return True
    try:
        cg.Engine(16, 16).close()
    except cg.CytomError:  # the failure was still to come
        return False
    finally:
        eng.set_fault_injection()
    return True


def test_compaction(cg, orc):
    rng = np.random.default_rng(1)
    parts = [batch(rng, m) for m in (70000, 150000, 20000, 400000)]  # the second and fourth grow the store
    st = orc.Store(N, VPT, True)
    for p in parts:
        st.insert(*p)
        st.compact()
    want = st.dump()
    ref, _ = st.run_minprop(orc.SSSP, start=0, max_iter=1000)
    for step in (0, 1, 3):
        for k in range(1, 30):
            with cg.Engine(N, VPT, weight_type=cg.WEIGHT_U32) as eng:
                done = False
                sssp = cg.SSSP(eng, start_vertex=0, max_iterations=1000)
                for j, p in enumerate(parts):
                    eng.insert_edges(*p)
                    if j == step:
                        done = not disturbed(cg, eng, k, eng.do_global_compaction)
                    eng.do_global_compaction()
                    sssp.execute_algorithm()
                got = eng.dump_tiles(weights=True)
                assert all(np.array_equal(a, b) for a, b in zip(got, want)), (step, k)
                assert np.array_equal(sssp.result(), ref), (step, k)
            if done:
                break
        assert done, step


def test_deletion(cg, orc):
    """A deletion that runs out of memory has not lowered any degree."""
    rng = np.random.default_rng(2)
    s, t, w = batch(rng, 300000)  # its scan takes scratch of its own
    gone = slice(1000, 90000)
    for k in range(1, 20):
        with cg.Engine(N, VPT, weight_type=cg.WEIGHT_U32) as eng:
            eng.insert_edges(s, t, w)
            eng.do_global_compaction()
            before = eng.degrees()

            def same():
                assert all(np.array_equal(a, b) for a, b in zip(eng.degrees(), before))

            more = disturbed(cg, eng, k, lambda: eng.delete_edges(s[gone], t[gone]), same)
            pairs = lambda a, b: np.unique(a.astype(np.uint64) << np.uint64(32) | b)  # noqa: E731
            left = np.setdiff1d(pairs(s, t), pairs(s[gone], t[gone]))
            assert eng.count_edges()[0] == len(left)
            killed = np.intersect1d(pairs(s, t), pairs(s[gone], t[gone]))
            out, inn = eng.degrees()
            assert np.array_equal(out, before[0] - np.bincount((killed >> np.uint64(32)).astype(np.int64), minlength=N))
            assert np.array_equal(inn, before[1] - np.bincount((killed & np.uint64(0xFFFFFFFF)).astype(np.int64), minlength=N))
        if not more:
            break
    assert not more


def test_dynamic_compaction_counters(cg, orc):
    """An insert whose counters found no room has inserted nothing."""
    rng = np.random.default_rng(3)
    parts = [batch(rng, 3000), batch(rng, 9000)]
    st = orc.Store(N, VPT, True)
    for p in parts:
        st.insert(*p)
    st.compact()
    want = st.dump()
    for k in range(1, 20):
        with cg.Engine(N, VPT, weight_type=cg.WEIGHT_U32, dynamic_compaction=True) as eng:
            more = False
            for j, p in enumerate(parts):
                if j == 0:
                    empty = lambda: [x.sum() for x in eng.degrees()] == [0, 0] and eng.count_edges() == (0, 0)  # noqa: E731

                    def nothing():
                        assert empty()

                    more = disturbed(cg, eng, k, lambda: eng.insert_edges(*p), nothing)
                else:
                    eng.insert_edges(*p)
            out, _ = eng.degrees()
            assert np.array_equal(out, np.bincount(np.concatenate([p[0] for p in parts]), minlength=N))
            eng.do_global_compaction()
            got = eng.dump_tiles(weights=True)
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), k
        if not more:
            break
    assert not more


def test_failed_compactions_give_their_memory_back(cg):
    """A compaction that fails again and again, at each of its allocations, holds no more memory than
    one that succeeds."""
    import torch
    n, m = 1 << 16, 1 << 21  # some 100 MB of temporaries each
    rng = np.random.default_rng(4)
    s, t = rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    with cg.Engine(n, 65536) as eng:
        eng.insert_edges(s, t)
        eng.do_global_compaction()
        eng.insert_edges(s, t)  # the same edges: every buffer has its size
        eng.do_global_compaction()
        eng.sync()
        before = free()
        for k in range(1, 9):
            for _ in range(4):
                eng.insert_edges(s, t)
                disturbed(cg, eng, k, eng.do_global_compaction)
        eng.sync()
        assert before - free() < 64 << 20
