"""FP32 forms of the weighted PageRank and its gradients where a value, a factor or a product of
the update lies outside the range in which float pairs keep their low words. Against the FP64
oracle on the same graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, VPT = 1 << 12, 1024


def solve(cg, orc, s, t, w, tele, c, n=N, vpt=VPT):
    """(ranks, dL/dw, dL/dt) of the FP32 form and of the oracle, edges in store order."""
    bits = w.astype(np.float32).view(np.uint32)
    st = orc.Store(n, vpt, True)
    st.insert(s, t, bits)
    st.compact()
    es, et, wb = orc.store_edges(st)
    ew = wb.view(np.float32).astype(np.float64)
    r, _ = orc.wpagerank(n, es, et, ew, t=tele, tol=1e-15)
    lam, gw, gt, _ = orc.wpagerank_adjoint(n, es, et, ew, r, c, t=tele, tol=1e-15)
    with cg.Engine(n, vpt, weight_type=cg.WEIGHT_F32) as eng:
        eng.insert_edges(s, t, bits)
        eng.do_global_compaction()
        p = cg.WeightedPageRank(eng, max_iterations=2000, tolerance=1e-12, kahan=True)
        p.set_teleport(tele)
        p.execute_algorithm()
        gw32, gt32, _ = p.adjoint(c)
        r32 = p.result()
    return (r32, gw32, gt32), (r, gw, gt), (es, et, ew, lam)


@pytest.mark.parametrize("scale,c_scale", [(1e33, 1e3), (1e30, 1.0), (1e-30, 1.0), (1.0, 1e-32), (1.0, 1e30)])
def test_gradients_of_extreme_weights_and_losses(cg, orc, scale, c_scale):
    """Sources of one in-edge or none whose teleport mass is small and whose out-weights are scaled:
    alpha r_u / s_u down to 1e-42, dL/dw still an FP32 normal. Every edge's gradient within 1e-5 of
    |alpha r_u / s_u| max |lambda| (lambda and P^T lambda are FP32 values converged to a few 1e-7
    of the largest), ranks within the family's bounds."""
    rng = np.random.default_rng(8)
    s, t = rng.integers(64, N, 40000, dtype=np.uint32), rng.integers(64, N, 40000, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s))
    few = np.repeat(np.arange(64, dtype=np.uint32), 3)  # sources nobody points to
    s, t = np.concatenate([s, few]), np.concatenate([t, rng.integers(64, N, len(few), dtype=np.uint32)])
    w = np.concatenate([w, rng.uniform(0.5, 1.0, len(few)) * scale])
    tele = rng.uniform(0.5, 1.5, N)
    tele[:64] *= 1e-4
    tele /= tele.sum()
    c = rng.standard_normal(N) * c_scale
    (r32, gw32, gt32), (r, gw, gt), (es, et, ew, lam) = solve(cg, orc, s, t, w, tele, c)
    assert np.abs(r32 - r).sum() <= 1e-6 * r.sum()
    out = np.bincount(es, ew, N)
    assert np.isfinite(gw32).all()
    bound = 0.85 * r[es] / out[es] * np.abs(lam).max() * 1e-5 + 1.5e-45  # and an FP32 denormal's step
    err = np.abs(gw32.astype(np.float64) - gw)
    assert (err <= bound).all(), (err / bound).max()
    assert np.abs(gt32 - gt).max() <= 1e-5 * np.abs(gt).max()


@pytest.mark.parametrize("c_scale,sparse", [(1e-37, False), (1e-33, False), (1e-33, True), (1.0, True), (1e30, False)])
def test_adjoint_of_small_losses(cg, orc, c_scale, sparse):
    """t . lambda of many small terms: 2^16 vertices, every second one dangling, loss weights equal
    (the terms' roundings then do not cancel) or on 16 vertices only. dL/dt is proportional to
    lambda: within 1e-6 of each entry (lambda is stored in FP32, 2^-24 a round, amplified by at
    most 1 / (1 - alpha) = 6.7: 4e-7) and an FP32 denormal's step."""
    n = 1 << 16
    rng = np.random.default_rng(4)
    s, t = rng.integers(0, n // 2, 1 << 18, dtype=np.uint32), rng.integers(0, n, 1 << 18, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s))
    c = np.full(n, c_scale)
    if sparse:
        c[rng.permutation(n)[16:]] = 0.0
    (r32, _, gt32), (r, _, gt), _ = solve(cg, orc, s, t, w, None, c, n=n, vpt=n)
    err = np.abs(gt32.astype(np.float64) - gt)
    bound = 1e-6 * np.abs(gt) + 1.5e-45
    assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("low,high", [(1e-36, 1e-30), (1e-42, 1.0)])
def test_ranks_of_extreme_teleports(cg, orc, low, high):
    """Teleport vectors of small size and of wide span: ranks within 1e-5 relative of the oracle where an
    FP32 normal holds them, within 1e-6 relative L1."""
    rng = np.random.default_rng(6)
    s, t = rng.integers(0, N // 2, 30000, dtype=np.uint32), rng.integers(0, N // 2, 30000, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s))
    tele = np.exp(rng.uniform(np.log(low), np.log(high), N))
    (r32, _, _), (r, _, _), _ = solve(cg, orc, s, t, w, tele, rng.standard_normal(N))
    ok = r > 1e-35  # contributions r / s and their products are FP32 too
    assert (np.abs(r32 - r)[ok] <= 1e-5 * r[ok]).all()
    assert np.abs(r32 - r).sum() <= 1e-6 * r.sum()


@pytest.mark.parametrize("what", ["loss", "teleport"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_infinities_and_nan(cg, orc, what, value):
    """One loss weight or teleport entry that is not finite: the FP32 form is finite exactly where the
    FP64 form is, in ranks and gradients, and within the family's bounds there."""
    rng = np.random.default_rng(9)
    s, t = rng.integers(0, N - 64, 3000, dtype=np.uint32), rng.integers(0, N, 3000, dtype=np.uint32)
    w = rng.uniform(0.5, 1.0, len(s)).astype(np.float32).view(np.uint32)
    c, tele = rng.standard_normal(N), rng.uniform(0.5, 1.5, N) / N
    (c if what == "loss" else tele)[700] = value
    got = []
    with cg.Engine(N, VPT, weight_type=cg.WEIGHT_F32) as eng:
        eng.insert_edges(s, t, w)
        eng.do_global_compaction()
        for kahan in (True, False):
            p = cg.WeightedPageRank(eng, max_iterations=4, tolerance=0.0, kahan=kahan)
            p.set_teleport(tele)
            p.execute_algorithm()
            gw, gt, _ = p.adjoint(c)
            got.append([np.asarray(x, np.float64) for x in (p.result(), gw, gt)])
    for a, b in zip(*got):
        ok = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), ok)
        if ok.any():
            assert np.abs(a - b)[ok].max() <= 1e-4 * np.abs(b[ok]).max()
