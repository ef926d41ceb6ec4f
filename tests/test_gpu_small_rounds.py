"""Rounds run by one thread-block cluster (graphs of few edges, small frontiers) against the
oracle's Jacobi rounds: values, round count and processed-edge count bit for bit, fresh and
incrementally. The sizes lie at the edges of the rule: vertex counts below one frontier word
and below one warp's words, tiles smaller than a word (no source directory), edge counts
either side of the dense limit, frontiers that grow past the limits and shrink again, more
changed words than the cluster's list, hubs longer than a queue chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(side):
    v = np.arange(side * side, dtype=np.uint32)
    r, d = v[v % side < side - 1], v[: side * (side - 1)]
    s = np.concatenate([r, d, r + 1, d + side])
    t = np.concatenate([r + 1, d + side, r, d])
    return s.astype(np.uint32), t.astype(np.uint32)


def star_of_paths(n):
    """A hub with many out-edges, then long paths from some of its neighbours."""
    hub = np.arange(1, 3001, dtype=np.uint32)
    path = np.arange(4000, n - 1, dtype=np.uint32)
    s = np.concatenate([np.zeros(3000, np.uint32), [2999, 17], path])
    t = np.concatenate([hub, [4000, 9000], path + 1])
    return s.astype(np.uint32), t.astype(np.uint32)


def graphs():
    rng = np.random.default_rng(3)
    rnd = lambda n, m: (rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32))  # noqa: E731
    return {
        "n16": (16, 4, *rnd(16, 40)),
        "n64": (64, 16, *rnd(64, 200)),
        "n512_tiles32": (512, 32, *rnd(512, 900)),
        "n4096_65536": (4096, 1024, *rnd(4096, 65536)),   # below the dense limit after duplicates
        "n16384_120k": (1 << 14, 4096, *rnd(1 << 14, 120000)),
        "lattice_128": (1 << 14, 2048, *lattice(128)),
        "lattice_256": (1 << 16, 65536, *lattice(256)),
        "star": (1 << 14, 4096, *star_of_paths(1 << 14)),
        "sparse_2^18": (1 << 18, 65536, *rnd(1 << 18, 400000)),  # frontiers past the limits in the middle
    }


@pytest.mark.parametrize("adaptive", [True, False])
@pytest.mark.parametrize("name", list(graphs()))
def test_small_rounds_match_oracle(cg, orc, name, adaptive):
    n, vpt, s, t = graphs()[name]
    if not adaptive and n > 1 << 14:
        pytest.skip("without adaptive scheduling only graphs below the dense limit take the cluster")
    w = orc.edge_weights(s, t, 7, 1, 255)
    st = orc.Store(n, vpt, True)
    cut = len(s) * 3 // 4
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32, adaptive_scheduling=adaptive) as eng:
        progs = {orc.BFS: cg.BFS(eng, start_vertex=0, max_iterations=100000),
                 orc.CC: cg.CC(eng, max_iterations=100000),
                 orc.SSSP: cg.SSSP(eng, start_vertex=0, max_iterations=100000)}
        for part, (lo, hi) in enumerate(((0, cut), (cut, len(s)))):
            st.insert(s[lo:hi], t[lo:hi], w[lo:hi])
            st.compact()
            eng.insert_edges(s[lo:hi], t[lo:hi], w[lo:hi])
            for algo, p in progs.items():
                got = p.execute_algorithm()
                ref, info = st.run_minprop(algo, start=0, max_iter=100000, adaptive=adaptive)
                assert np.array_equal(p.result(), ref), (algo, part)
                if part == 0:
                    assert got["iterations"] == info["iterations"], algo
                    assert got["count_edges"] == info["count_edges"], algo
        # from scratch on the whole graph, several at once, and under an iteration cap
        for p in progs.values():
            p.init_algorithm()
        for (algo, p), got in zip(progs.items(), eng.run_many(list(progs.values()))):
            ref, info = st.run_minprop(algo, start=0, max_iter=100000, adaptive=adaptive)
            assert np.array_equal(p.result(), ref), algo
            assert got["iterations"] == info["iterations"] and got["count_edges"] == info["count_edges"]
        capped = cg.SSSP(eng, start_vertex=0, max_iterations=3)
        got = capped.execute_algorithm()
        ref, info = st.run_minprop(orc.SSSP, start=0, max_iter=3, adaptive=adaptive)
        assert got["iterations"] == info["iterations"] <= 3 and np.array_equal(capped.result(), ref)
