"""Paths of the store's one-sweep sort that ordinary sorts do not take: a tile whose counts are not
waited for but counted again, and sorts of 2^30 keys, whose status words have 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("count", [8193, 2048 * 40 + 1, 8192 * 70 - 1, 1 << 20])
def test_counts_not_waited_for(cg, orc, count, weighted):
    n, vpt = 1 << 15, 4096
    rng = np.random.default_rng(count)
    s = rng.integers(0, n, count, dtype=np.uint32)
    t = (rng.integers(0, n, count) >> rng.integers(0, 15, count)).astype(np.uint32)
    w = rng.integers(0, 1 << 32, count, dtype=np.uint32) if weighted else None
    st = orc.Store(n, vpt, weighted)
    st.insert(s, t, w)
    st.compact()
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32 if weighted else cg.UNWEIGHTED) as eng:
        eng.set_fault_injection(idle_poll_limit=1)
        eng.insert_edges(s, t, w)
        eng.do_global_compaction()
        got = eng.dump_tiles(weights=weighted)
    want = st.dump()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    if weighted:
        assert np.array_equal(got[2], want[2])


def test_sort_of_2_30_keys(cg):
    """One tile of 65,536 vertices: the packed edges are the keys, in order and without duplicates.
    Some 130 GB of device memory."""
    import torch
    if torch.cuda.mem_get_info()[0] < 200 << 30:
        pytest.skip("needs 200 GB of free device memory")
    n, count = 1 << 16, (1 << 30) + 4097
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    s = torch.randint(0, n, (count,), device="cuda", dtype=torch.int32, generator=g)
    t = torch.randint(0, n, (count,), device="cuda", dtype=torch.int32, generator=g)
    torch.cuda.synchronize()
    with cg.Engine(n, n) as eng:
        eng.insert_edges(s, t)
        eng.do_global_compaction()
        tp, ed, _, _ = eng.dump_tiles()
    present = torch.zeros(1 << 32, device="cuda", dtype=torch.uint8)  # every possible key
    step = 1 << 28
    for k in range(0, count, step):
        present[(s[k:k + step].long() << 16) | t[k:k + step].long()] = 1
    del s, t
    distinct = int(present.sum(dtype=torch.int64))
    assert int(tp[0]) == 0 and int(tp[1]) == distinct == len(ed)
    last = -1
    for k in range(0, distinct, step):
        e = torch.from_numpy(ed[k:k + step].view(np.int32)).cuda().long() & 0xFFFFFFFF
        assert int(e[0]) > last and bool((e[1:] > e[:-1]).all()) and bool(present[e].all())
        last = int(e[-1])
