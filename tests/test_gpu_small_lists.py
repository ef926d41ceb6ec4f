"""Small rounds that list many words: the cluster's shared list of changed words (2,048 a CTA of
16) just full, overflowing, and far past it; CC from scratch on few edges over vertex ranges
either side of the 2^15 words up to which its run is one launch. Against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def star(n, leaves, rng):
    """A hub with its leaves in words of their own, chains behind some of them."""
    leaf = (1 + np.arange(leaves, dtype=np.int64)) * 32
    assert leaf[-1] < n
    leaf = (leaf + rng.integers(0, 32, leaves)) % n
    tail = leaf[rng.permutation(leaves)[: leaves // 16]]
    s = np.concatenate([np.zeros(leaves, np.int64), tail, (tail + 40) % n])
    t = np.concatenate([leaf, (tail + 40) % n, (tail + 77) % n])
    return s.astype(np.uint32), t.astype(np.uint32)


# (2^21 vertices: 58,000 changed words, some 3,600 a CTA)
@pytest.mark.parametrize("leaves", [32768, 32769, 58000])
@pytest.mark.parametrize("lg,vpt", [(21, 65536), (21, 16384), (22, 65536)])
def test_more_changed_words_than_the_list(cg, orc, lg, vpt, leaves):
    n = 1 << lg
    s, t = star(n, leaves, np.random.default_rng(leaves + lg))
    w = orc.edge_weights(s, t, 7, 1, 255)
    st = orc.Store(n, vpt, True)
    st.insert(s, t, w)
    st.compact()
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32) as eng:
        eng.insert_edges(s, t, w)
        eng.do_global_compaction()
        for make, algo in ((cg.BFS, orc.BFS), (cg.SSSP, orc.SSSP), (cg.CC, orc.CC)):
            p = make(eng, start_vertex=0, max_iterations=1000)
            got = p.execute_algorithm()
            ref, info = st.run_minprop(algo, start=0, max_iter=1000)
            assert np.array_equal(p.result(), ref), algo
            assert got["iterations"] == info["iterations"] and got["count_edges"] == info["count_edges"], algo


@pytest.mark.parametrize("lg", [20, 21, 22])
def test_cc_from_scratch_over_many_words(cg, orc, lg):
    """Up to 2^15 words the run is one launch of the cluster; with more its first round is grid-wide.
    Runs that go on from earlier values are one launch either way."""
    n, m = 1 << lg, 60000
    rng = np.random.default_rng(lg)
    s, t = rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32)
    st = orc.Store(n, 65536)
    with cg.Engine(n, 65536) as eng:
        cc = cg.CC(eng, max_iterations=1000)
        for part, (lo, hi) in enumerate(((0, 50000), (50000, m))):
            st.insert(s[lo:hi], t[lo:hi])
            st.compact()
            eng.insert_edges(s[lo:hi], t[lo:hi])
            eng.do_global_compaction()
            before = eng.launch_count()
            got = cc.execute_algorithm()
            launches = eng.launch_count() - before
            ref, info = st.run_minprop(orc.CC, start=0, max_iter=1000)
            assert np.array_equal(cc.result(), ref)
            if part == 0:
                assert got["iterations"] == info["iterations"] and got["count_edges"] == info["count_edges"]
            else:
                assert launches == 1
        cc.init_algorithm()
        before = eng.launch_count()
        cc.execute_algorithm()
        scratch = eng.launch_count() - before
        assert scratch == 2 if lg <= 20 else scratch > 5, scratch  # its initialisation and the cluster, or a loop
