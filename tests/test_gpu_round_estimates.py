"""The out-edge estimate that picks the kind of a round depends on the snapshot alone: on small
graphs it holds every listed word whichever kernel lists them, and an insert beside
asynchronous runs does not change it. The edges a run scans, which follow from the kinds of its
rounds, are therefore the same in every repetition."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


def test_small_graph_scans_the_same_edges_profiled(cg):
    """2^15 pairs (v, v + 1), then 10,000 edges that lower one end of a pair each: the active
    vertices hold more than an eighth of the edges but few of them lie in any 129 words."""
    n = 1 << 16
    even = np.arange(0, n, 2, dtype=np.uint32)
    rng = np.random.default_rng(5)
    low = rng.permutation(even[100:])[:10000].astype(np.uint32)
    got = []
    for profiled in (False, True):
        with cg.Engine(n, 1024) as eng:
            eng.insert_edges(even, even + 1)
            cc = cg.CC(eng, max_iterations=1000)
            cc.execute_algorithm()
            eng.insert_edges(np.zeros(len(low), np.uint32), low)
            eng.set_profiling(profiled)
            x = cc.execute_algorithm()
            eng.set_profiling(False)
            got.append((x["iterations"], x["count_edges"], x["edges_scanned"], cc.result().tobytes()))
    assert got[0] == got[1]


CODE = """
import sys, json, numpy as np
sys.path.insert(0, {root!r})
import torch, cytom_gb300 as cg
side = 256
n = side * side
v = np.arange(n, dtype=np.uint32)
r, d = v[v % side < side - 1], v[: side * (side - 1)]
s = np.concatenate([r, d, r + 1, d + side]).astype(np.uint32)
t = np.concatenate([r + 1, d + side, r, d]).astype(np.uint32)
m = 1 << 25  # 512 out-edges a vertex: a frontier of 256 then holds more than a small round's
bs = torch.randint(0, n, (m,), device="cuda", dtype=torch.int32)
bt = torch.randint(0, n, (m,), device="cuda", dtype=torch.int32)
torch.cuda.synchronize()
want = (v // side + v % side).astype(np.uint32)
out = []
for beside in (False, True, True):
    with cg.Engine(n, n) as eng:
        eng.insert_edges(bs, bt)  # the append region has its size
        eng.clear()
        eng.insert_edges(s, t)
        eng.do_global_compaction()
        ps = [cg.BFS(eng, start_vertex=0, max_iterations=10000) for _ in range(2)]
        eng.run_many_async(ps)
        if beside:
            eng.insert_edges(bs, bt)
        x = eng.run_many_wait()
        out.append([[q["iterations"], q["count_edges"], q["edges_scanned"]] for q in x])
        if not beside:
            assert all(np.array_equal(p.result(), want) for p in ps)
print(json.dumps(out))
"""


def test_insert_beside_asynchronous_runs_changes_no_round():
    """A lattice's small frontiers, while 2^25 edges are appended: dense rounds (forced by the
    threshold) in place of small ones would scan the whole graph."""
    env = dict(os.environ, CYTOM_SPARSE_DIV="1024")
    r = subprocess.run([sys.executable, "-c", CODE.format(root=str(ROOT))], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out[0] == out[1] == out[2], out


BATCHES = """
import sys, json, numpy as np
sys.path.insert(0, {root!r})
import cytom_gb300 as cg
side = 256
n = side * side
v = np.arange(n, dtype=np.uint32)
r, d = v[v % side < side - 1], v[: side * (side - 1)]
s = np.concatenate([r, d, r + 1, d + side]).astype(np.uint32)
t = np.concatenate([r + 1, d + side, r, d]).astype(np.uint32)
out, vals = [], []
for asynchronous in (False, True):
    rng = np.random.default_rng(1)
    with cg.Engine(n, 4096, weight_type=cg.WEIGHT_U32) as eng:
        eng.insert_edges(s, t, rng.integers(1, 100, len(s), dtype=np.uint32))
        eng.do_global_compaction()
        ps = [cg.BFS(eng, start_vertex=0, max_iterations=10000), cg.SSSP(eng, start_vertex=0, max_iterations=10000)]
        rows = []
        for k in range(6):
            if asynchronous:
                eng.run_many_async(ps)
            else:
                x = eng.run_many(ps)
            m = (1 << 19) + 17 * k  # sources and targets among the last vertices, many of them repeated
            a = (n - 1 - (rng.integers(0, n, m) >> rng.integers(0, 10, m))).astype(np.uint32)
            b = (n - 1 - (rng.integers(0, n, m) >> rng.integers(0, 10, m))).astype(np.uint32)
            eng.insert_edges(a, b, rng.integers(1000, 9000, m, dtype=np.uint32))
            eng.do_global_compaction()
            if asynchronous:
                x = eng.run_many_wait()
            rows.append([[q["iterations"], q["count_edges"], q["edges_scanned"]] for q in x])
        out.append(rows)
        vals.append([p.result().tobytes() for p in ps])
assert vals[0] == vals[1]
print(json.dumps(out))
"""


def test_estimates_follow_the_batches():
    """A stream whose batches raise the degrees of the frontiers past a small round's limit, its runs
    asynchronous and not: the same rounds, so the degrees that asynchronous runs keep follow."""
    env = dict(os.environ, CYTOM_SPARSE_DIV="1024", CYTOM_AUTOTUNE="0")
    r = subprocess.run([sys.executable, "-c", BATCHES.format(root=str(ROOT))], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out[0] == out[1], out


def test_rejected_insert_beside_asynchronous_runs(cg):
    """The degrees a rejected batch raised and gave back are not seen by the runs beside it; the
    degrees themselves and later runs are those of the graph without it."""
    side = 256
    n = side * side
    v = np.arange(n, dtype=np.uint32)
    r, d = v[v % side < side - 1], v[: side * (side - 1)]
    s = np.concatenate([r, d, r + 1, d + side]).astype(np.uint32)
    t = np.concatenate([r + 1, d + side, r, d]).astype(np.uint32)
    rng = np.random.default_rng(2)
    bs, bt = rng.integers(0, n, 1 << 22, dtype=np.uint32), rng.integers(0, n, 1 << 22, dtype=np.uint32)
    bt[12345] = n
    want = (v // side + v % side).astype(np.uint32)
    got = []
    for beside in (False, True):
        with cg.Engine(n, n) as eng:
            eng.insert_edges(s, t)
            eng.do_global_compaction()
            ps = [cg.BFS(eng, start_vertex=0, max_iterations=10000) for _ in range(2)]
            eng.run_many_async(ps)
            if beside:
                with pytest.raises(cg.CytomError) as e:
                    eng.insert_edges(bs, bt)
                assert e.value.code == -3
            x = eng.run_many_wait()
            ps[0].init_algorithm()
            x.append(ps[0].execute_algorithm())
            got.append([[q["iterations"], q["count_edges"], q["edges_scanned"]] for q in x])
            assert all(np.array_equal(p.result(), want) for p in ps)
            out, inn = eng.degrees()
            assert np.array_equal(out, np.bincount(s, minlength=n)) and np.array_equal(inn, np.bincount(t, minlength=n))
    assert got[0] == got[1]


def test_without_memory_for_the_degrees(cg, orc):
    """The first asynchronous launch cannot have its copy of the degrees: the runs give the same
    values, later ones too."""
    s, t = orc.rmat(12, 0, 1 << 16, 3)
    n = 1 << 12
    st = orc.Store(n, 1024)
    st.insert(s, t)
    st.compact()
    with cg.Engine(n, 1024) as eng:
        eng.insert_edges(s, t)
        progs = [(cg.BFS(eng, start_vertex=0, max_iterations=1000), orc.BFS), (cg.CC(eng, max_iterations=1000), orc.CC)]
        eng.run_many([p for p, _ in progs])
        for fail in (1, 0):
            for p, _ in progs:
                p.init_algorithm()
            eng.set_fault_injection(fail_alloc_after=fail)
            eng.run_many_async([p for p, _ in progs])
            stats = eng.run_many_wait()
            eng.set_fault_injection()
            for (p, a), x in zip(progs, stats):
                ref, info = st.run_minprop(a, start=0, max_iter=1000)
                assert np.array_equal(p.result(), ref) and x["iterations"] == info["iterations"]
