"""Ingest kernels at their edges: RMAT thresholds that do not ascend or lie above every hash;
a rejected batch (the only bad endpoint first, last, on either side) leaves keys, counts and
degrees as they were; merges whose 1,024-output spans hold no, one, 64, 65 or only new edges.
Against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("abc", [(1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0), (0.5, -0.2, 0.4), (0.6, 0.3, -0.5),
                                 (2.0, -1.5, 0.1), (0.0, 0.0, 0.0)])
def test_rmat_thresholds(cg, orc, abc):
    a, b, c = abc
    with cg.Engine(1 << 12, 1024) as eng:
        gs, gt, _ = eng.generate_rmat(5, 20000, 11, seed=9, a=a, b=b, c=c)
    s, t = orc.rmat(11, 5, 20000, 9, a=a, b=b, c=c)
    assert np.array_equal(gs, s) and np.array_equal(gt, t)


@pytest.mark.parametrize("where", ["first_src", "last_src", "first_tgt", "last_tgt"])
@pytest.mark.parametrize("count", [1, 255, 5000])
def test_rejected_batch_leaves_no_trace(cg, orc, where, count):
    n, vpt = 1 << 12, 1024
    rng = np.random.default_rng(count)
    s, t = (rng.integers(0, n, 3000, dtype=np.uint32) for _ in range(2))
    bs, bt = (rng.integers(0, n, count, dtype=np.uint32) for _ in range(2))
    bad = bs if where.endswith("src") else bt
    bad[0 if where.startswith("first") else -1] = n
    st = orc.Store(n, vpt)
    st.insert(s, t)
    with cg.Engine(n, vpt) as eng:
        eng.insert_edges(s, t)
        with pytest.raises(cg.CytomError) as ei:
            eng.insert_edges(bs, bt)
        assert ei.value.code == -3
        assert eng.count_edges() == (0, 3000)
        assert all(np.array_equal(x, y) for x, y in zip(eng.degrees(), st.degrees()))
        st.insert(s[::-1].copy(), t)
        st.compact()
        eng.insert_edges(s[::-1].copy(), t)
        eng.do_global_compaction()
        got, want = eng.dump_tiles(), st.dump()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert all(np.array_equal(x, y) for x, y in zip(eng.degrees(), st.degrees()))


@pytest.mark.parametrize("old,new", [(0, 1), (0, 1024), (0, 5000), (1023, 1), (1024, 1), (1025, 2), (40000, 64),
                                     (40000, 65), (40000, 20000), (100, 40000)])
def test_merge_spans(cg, orc, old, new):
    n, vpt = 1 << 11, 512
    rng = np.random.default_rng(old + new)
    pick = rng.permutation(n * n)[: old + new].astype(np.int64)  # distinct pairs
    if (old, new) in ((40000, 64), (40000, 65)):
        pick[old:] = np.sort(pick[:old])[20000] + 1 + np.arange(new)  # the new edges next to one another
    s, t = (pick // n).astype(np.uint32), (pick % n).astype(np.uint32)
    w = orc.edge_weights(s, t, 3, 1, 1000)
    st = orc.Store(n, vpt, True)
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32) as eng:
        bfs = cg.BFS(eng, start_vertex=int(s[0]), max_iterations=1000)
        for lo, hi in ((0, old), (old, old + new)):
            if lo == hi:
                continue
            st.insert(s[lo:hi], t[lo:hi], w[lo:hi])
            st.compact()
            eng.insert_edges(s[lo:hi], t[lo:hi], w[lo:hi])
            eng.do_global_compaction()
            got, want = eng.dump_tiles(weights=True), st.dump()
            for x, y in zip(got, want):
                assert np.array_equal(x, y)
            bfs.execute_algorithm()  # the directory and chunk table written by the merge
            assert np.array_equal(bfs.result(), st.run_minprop(orc.BFS, start=int(s[0]), max_iter=1000)[0])


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("size", [1, 31, 255, 256, 257, 1500])
def test_merge_directory_of_uneven_tiles(cg, orc, size, weighted):
    """Tiles of `size` edges next to empty ones and to a full one, with source blocks close
    together and far apart: the directory that merges write and the one built at once lead
    sparse rounds to the same values."""
    n, vpt = 1 << 15, 4096
    rng = np.random.default_rng(size)
    parts = []
    for x, y in ((0, 0), (0, 7), (3, 2), (3, 3), (7, 0), (7, 7)):
        m = 20000 if (x, y) == (3, 3) else size
        src = rng.integers(0, vpt, m) if y else rng.choice(np.array([0, 31, 32, vpt - 1]), m)
        parts.append(np.stack([x * vpt + src, y * vpt + rng.integers(0, vpt, m)]))
    s, t = (a.astype(np.uint32) for a in np.concatenate(parts, 1))
    order = rng.permutation(len(s))
    s, t = s[order], t[order]
    w = orc.edge_weights(s, t, 5, 1, 1000) if weighted else None
    start = int(s[0])
    algo, cls = (orc.SSSP, cg.SSSP) if weighted else (orc.BFS, cg.BFS)
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32 if weighted else 0) as eng:
        job = cls(eng, start_vertex=start, max_iterations=1000)
        st = orc.Store(n, vpt, weighted)
        cuts = [0, len(s) // 3, len(s) - 1, len(s)]
        for lo, hi in zip(cuts, cuts[1:]):
            if lo == hi:
                continue
            part = [a[lo:hi] for a in ((s, t, w) if weighted else (s, t))]
            st.insert(*part)
            st.compact()
            eng.insert_edges(*part)
            eng.do_global_compaction()
            job.execute_algorithm()
            assert np.array_equal(job.result(), st.run_minprop(algo, start=start, max_iter=1000)[0])


@pytest.mark.parametrize("n", [1 << 10, 1 << 11, 1 << 13])
@pytest.mark.parametrize("count,bad", [((1 << 17) - 1, False), (1 << 17, False), ((1 << 17) + 1, True), (300001, False)])
def test_degrees_of_large_batches(cg, n, count, bad):
    """Degrees of batches around the size from which blocks count the first vertices by
    themselves, with fewer vertices than such counters, as many and more; a rejected batch
    takes its degrees back."""
    rng = np.random.default_rng(count + n)
    s = np.minimum(rng.geometric(0.002, count) - 1, n - 1).astype(np.uint32)
    t = rng.integers(0, n, count, dtype=np.uint32)
    with cg.Engine(n, 512) as eng:
        if bad:
            b = t.copy()
            b[count // 2] = n
            with pytest.raises(cg.CytomError):
                eng.insert_edges(s, b)
            assert not any(x.any() for x in eng.degrees())
        eng.insert_edges(s, t)
        out_deg, in_deg = eng.degrees()
        assert np.array_equal(out_deg, np.bincount(s, minlength=n)) and np.array_equal(in_deg, np.bincount(t, minlength=n))
