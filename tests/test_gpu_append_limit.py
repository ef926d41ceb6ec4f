"""Appends either side of the batch size from which blocks count the first vertices' degrees in
shared memory: degrees and edges of batches with and without hubs among the low ids, and of a
rejected batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [(1 << 17) - 1, 1 << 17, (1 << 18) - 1, 1 << 18, (1 << 18) + 1])
@pytest.mark.parametrize("kind", ["hubs", "uniform"])
def test_degrees(cg, count, kind):
    n = 1 << 13
    rng = np.random.default_rng(count)
    draw = lambda: (rng.integers(0, n, count) >> (rng.integers(0, 13, count) if kind == "hubs" else 0)).astype(np.uint32)  # noqa: E731
    s, t = draw(), draw()
    with cg.Engine(n, 2048) as eng:
        eng.insert_edges(s, t)
        bad = s.copy()
        bad[count // 2] = n
        with pytest.raises(cg.CytomError) as e:
            eng.insert_edges(bad, t)
        assert e.value.code == -3
        out, inn = eng.degrees()
        assert np.array_equal(out, np.bincount(s, minlength=n)) and np.array_equal(inn, np.bincount(t, minlength=n))
        eng.do_global_compaction()
        assert eng.count_edges()[0] == len(np.unique(s.astype(np.uint64) << np.uint64(32) | t))
