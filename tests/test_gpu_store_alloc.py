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
