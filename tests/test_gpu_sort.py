"""The store's radix sort at the sizes where its forms meet: one block (up to 8,192 keys),
small tiles (2,048 keys, up to 2^19) and large tiles (8,192 keys), each at an exact number
of tiles and one key either side, with values (weights) and without. Duplicates and
self-loops are kept in the input, so stability shows in the kept weights. Compared bit for
bit with the oracle's compaction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 2047, 2048, 2049, 8191, 8192, 8193, 10240, 10241, 1 << 19, (1 << 19) + 1, 8192 * 70 - 1,
         8192 * 70, 8192 * 70 + 1]


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("count", SIZES)
def test_sorted_store_matches_oracle(count, weighted):
    import cytom_gb300 as cg
    from oracle import oracle as orc
    n, vpt = 1 << 15, 4096  # 30-bit keys: four passes of unequal digits
    rng = np.random.default_rng(count + weighted)
    s = rng.integers(0, n, count, dtype=np.uint32)
    t = (rng.integers(0, n, count) >> rng.integers(0, 15, count)).astype(np.uint32)  # skewed towards low ids
    w = rng.integers(0, 1 << 32, count, dtype=np.uint32) if weighted else None
    st = orc.Store(n, vpt, weighted)
    st.insert(s, t, w)
    st.compact()
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32 if weighted else cg.UNWEIGHTED) as eng:
        eng.insert_edges(s, t, w)
        eng.do_global_compaction()
        got = eng.dump_tiles(weights=weighted)
    want = st.dump()
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1], want[1])
    if weighted:
        assert np.array_equal(got[2], want[2])
