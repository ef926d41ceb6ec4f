"""The PageRank family on a graph whose in-degrees (and, for the adjoint, out-degrees) sit on
the bounds of the pull's in-degree bins, in every form: targets of no in-edge, one, four and
five (thread bin), 32 and 33 (four lanes), 256 and 257 (eight lanes), 512 and 513 (the warp
bin's bound on a store of this size), 4,096 and more (one block), and bins whose target count
leaves a warp's share of targets partly empty. FP32 values against FP64 within the family's
1e-6 relative L1 and 1e-5 relative, FP64 values within 1e-10, gradients within 1e-4 of the
largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, VPT = 1 << 13, 2048
DEGREES = [1, 4, 5, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1024, 4095, 4096, 4097, 6000]


def edges(per_degree, reverse):
    """`per_degree` targets of each in-degree; the last vertices have no out-edge."""
    rng = np.random.default_rng(per_degree)
    src, tgt, v = [], [], 0
    for d in DEGREES:
        for _ in range(per_degree if d < 300 else 1):
            src.append(rng.choice(N - 64, d, replace=False))
            tgt.append(np.full(d, v))
            v += 1
    s, t = np.concatenate(src).astype(np.uint32), np.concatenate(tgt).astype(np.uint32)
    return (t, s) if reverse else (s, t)


def close(x, ref, l1, mr):
    x = np.asarray(x, np.float64)
    e1 = np.abs(x - ref).sum() / np.abs(ref).sum()
    em = (np.abs(x - ref) / np.maximum(np.abs(ref), 1e-300)).max()
    assert e1 <= l1 and em <= mr, (e1, em)


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("per_degree", [1, 3, 37])
def test_pull_bins(cg, orc, per_degree, reverse):
    s, t = edges(per_degree, reverse)
    st = orc.Store(N, VPT)
    st.insert(s, t)
    st.compact()
    with cg.Engine(N, VPT) as eng:
        eng.insert_edges(s, t)
        ref, _ = st.pagerank_norm(tol=1e-15)
        p = cg.PageRank(eng, max_iterations=1000, tolerance=1e-14, kahan=False)
        p.execute_algorithm()
        close(p.result64(), ref, 1e-10, 1e-8)
        p = cg.PageRank(eng, max_iterations=1000, tolerance=1e-10, kahan=True)
        p.execute_algorithm()
        close(p.result(), ref, 1e-6, 1e-5)
        two = [cg.PageRank(eng, max_iterations=1000, tolerance=1e-10, kahan=True) for _ in range(2)]
        cg.run_batch(two)
        for q in two:
            close(q.result(), ref, 1e-6, 1e-5)
        ref, _ = st.pagerank_unnorm(tol=1e-14)
        p = cg.PageRankDelta(eng, delta=0.0, max_iterations=1000, tolerance=1e-9)
        p.execute_algorithm()
        close(p.result(), ref, 1e-6, 1e-5)
    w = orc.unit_weights(s, t, 5)
    c = np.random.default_rng(2).standard_normal(N)
    tele = np.random.default_rng(3).random(N) + 0.05
    tele /= tele.sum()
    with cg.Engine(N, VPT, weight_type=cg.WEIGHT_F32) as eng:
        eng.insert_edges(s, t, w.view(np.uint32))
        eng.do_global_compaction()
        wst = orc.Store(N, VPT, True)
        wst.insert(s, t, w.view(np.uint32))
        wst.compact()
        es, et, wb = orc.store_edges(wst)
        ew = wb.view(np.float32).astype(np.float64)
        for tv in (None, tele):
            ref, _ = orc.wpagerank(N, es, et, ew, t=tv, tol=1e-15)
            _, gw_ref, gt_ref, _ = orc.wpagerank_adjoint(N, es, et, ew, ref, c, t=tv, tol=1e-15)
            for kahan in (True, False):
                p = cg.WeightedPageRank(eng, max_iterations=2000, tolerance=1e-10 if kahan else 1e-14, kahan=kahan)
                p.set_teleport(tv)
                p.execute_algorithm()
                if kahan:
                    close(p.result(), ref, 1e-6, 1e-5)
                else:
                    close(p.result64(), ref, 1e-10, 1e-8)
                gw, gt, _ = p.adjoint(c)
                assert np.abs(gw - gw_ref).max() <= 1e-4 * np.abs(gw_ref).max()
                assert np.abs(gt - gt_ref).max() <= 1e-4 * np.abs(gt_ref).max()


@pytest.mark.parametrize("rounds", [1, 2, 7, 8, 9, 17])
def test_round_counts_of_captured_loop(cg, rounds):
    """Runs that end within, at and past the rounds of the captured loop's body, again on the
    same captured loop, against the loop driven by the host: the same rounds and edge counts;
    values but for the order of the dangling mass's FP64 atomics (one FP32 ulp, 1e-12)."""
    s, t = edges(3, False)
    with cg.Engine(N, VPT) as eng:
        eng.insert_edges(s, t)
        forms = [(lambda: cg.PageRank(eng, max_iterations=rounds, tolerance=0.0, kahan=True), "result", 1.2e-7),
                 (lambda: cg.PageRank(eng, max_iterations=rounds, tolerance=0.0, kahan=False), "result64", 1e-12),
                 (lambda: cg.PageRankDelta(eng, delta=0.0, max_iterations=rounds, tolerance=0.0), "result", 1.2e-7)]
        for make, result, tol in forms:
            got = []
            for host in (False, True):
                p = make()
                eng.set_profiling(host)
                for again in range(2):
                    st = p.execute_algorithm()
                    got.append((np.asarray(getattr(p, result)(), np.float64), st["iterations"], st["count_edges"]))
                eng.set_profiling(False)
            for a, b in zip(got[:2], got[2:]):
                assert a[1:] == b[1:] and a[1] <= rounds
                assert (np.abs(a[0] - b[0]) <= tol * np.abs(b[0])).all()
            assert got[0][1] == rounds
