"""Memory of the FP32 weighted PageRank: its copies of weight sums and teleport vector as float pairs
take no device memory past what building the graph's structures needed, and its gradients can do
without their per-vertex factors. Each allocation of a teleport vector, a run or an adjoint in
turn fails once: the call reports it and succeeds when repeated, or gives the same answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pairs_take_no_memory_past_the_build(cg):
    import torch
    n = 1 << 23  # 64 MiB a vector of FP64 or of pairs
    rng = np.random.default_rng(2)
    s, t = rng.integers(0, n, n, dtype=np.uint32), rng.integers(0, n, n, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, n).astype(np.float32).view(np.uint32)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    with cg.Engine(n, 65536, weight_type=cg.WEIGHT_F32) as eng:
        eng.insert_edges(s, t, w)
        eng.do_global_compaction()
        p64 = cg.WeightedPageRank(eng, max_iterations=3, tolerance=0.0, kahan=False)
        p64.execute_algorithm()  # builds the structures; the pool keeps the temporaries
        before = free()
        p = cg.WeightedPageRank(eng, max_iterations=3, tolerance=0.0, kahan=True)
        p.set_teleport(np.full(n, 1.0 / n))
        p.execute_algorithm()
        # the job's five FP32 vectors and its FP64 teleport vector
        assert before - free() <= n * (5 * 4 + 8) + (16 << 20), "a vector of pairs came on top"


def test_each_allocation_fails_once(cg, orc):
    n, vpt = 1 << 12, 1024
    rng = np.random.default_rng(2)
    s, t = rng.integers(0, n - 99, 30000, dtype=np.uint32), rng.integers(0, n, 30000, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s)).astype(np.float32)
    tele = rng.random(n) + 0.05
    tele /= tele.sum()
    c = rng.standard_normal(n)
    st = orc.Store(n, vpt, True)
    st.insert(s, t, w.view(np.uint32))
    st.compact()
    es, et, wb = orc.store_edges(st)
    ew = wb.view(np.float32).astype(np.float64)
    ref, _ = orc.wpagerank(n, es, et, ew, t=tele, tol=1e-15)
    _, gw_ref, gt_ref, _ = orc.wpagerank_adjoint(n, es, et, ew, ref, c, t=tele, tol=1e-15)
    without = {"teleport": 0, "run": 0, "adjoint": 0}
    for step in without:
        for k in range(1, 40):
            with cg.Engine(n, vpt, weight_type=cg.WEIGHT_F32) as eng:
                eng.insert_edges(s, t, w.view(np.uint32))
                eng.do_global_compaction()
                p = cg.WeightedPageRank(eng, max_iterations=2000, tolerance=1e-10, kahan=True)
                calls = {"teleport": lambda: p.set_teleport(tele), "run": p.execute_algorithm, "adjoint": lambda: p.adjoint(c)}
                fired = True
                for name, call in calls.items():
                    if name == step:
                        eng.set_fault_injection(fail_alloc_after=k)
                        try:
                            out = call()
                        except cg.CytomError as e:
                            assert e.code == -2
                            out = call()
                        else:
                            try:  # had the call k allocations at all?
                                cg.Engine(16, 16).close()
                                without[step] += 1
                            except cg.CytomError:
                                fired = False
                        eng.set_fault_injection()
                    else:
                        out = call()
                gw, gt, _ = out
                r = p.result()
                assert np.abs(r - ref).sum() <= 1e-6 * np.abs(ref).sum()
                assert np.abs(gw - gw_ref).max() <= 1e-4 * np.abs(gw_ref).max()
                assert np.abs(gt - gt_ref).max() <= 1e-4 * np.abs(gt_ref).max()
            if not fired:
                break
        assert not fired, step
    assert without["adjoint"] == 1, without
