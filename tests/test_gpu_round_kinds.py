"""The kinds of a round against one another: small rounds in a cluster of 16 CTAs, of 8, and none
(CYTOM_SMALL_ROUNDS), so that the grid-wide sparse and dense rounds also run on the graphs and
frontiers that the cluster takes otherwise: one tile, a few, a mask bit per column and per four
columns. Values against the oracle; round count, active vertices and processed-edge count of
fresh runs against the oracle and of incremental runs between the kinds."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

CODE = """
import sys, json, numpy as np
sys.path.insert(0, {root!r})
import cytom_gb300 as cg
from oracle import oracle as orc
n, vpt = {n}, {vpt}
rng = np.random.default_rng(n + vpt)
hubs = np.array([0, 1, n // 2, n - 1])
path = np.arange(0, n - 33, 3)
s = np.concatenate([np.repeat(hubs, 9000), rng.integers(0, n, 60000), path])
t = np.concatenate([rng.integers(0, n, 36000), rng.integers(0, n, 60000), path + 33])
s, t = s.astype(np.uint32), t.astype(np.uint32)
w = orc.edge_weights(s, t, 3, 1, 1000)
order = rng.permutation(len(s))
cuts = [0, len(s) * 6 // 10, len(s) * 9 // 10, len(s) - 40, len(s)]
out = []
with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32) as eng:
    progs = [(cg.BFS(eng, start_vertex=0, max_iterations=1000), orc.BFS), (cg.CC(eng, max_iterations=1000), orc.CC),
             (cg.SSSP(eng, start_vertex=0, max_iterations=1000), orc.SSSP)]
    st = orc.Store(n, vpt, True)
    for k in range(4):
        part = order[cuts[k]:cuts[k + 1]]
        eng.insert_edges(s[part], t[part], w[part])
        st.insert(s[part], t[part], w[part])
        st.compact()
        refs = [st.run_minprop(a, start=0, max_iter=1000) for _, a in progs]
        def go(p):  # a run, with the launches of its sparse rounds and applies when it is profiled
            eng.reset_kernel_stats()
            x = p.execute_algorithm()
            ks = eng.kernel_stats()
            return x, [ks[c]["launches"] if c in ks else 0 for c in ("gather", "gather_sparse", "apply")]
        for (p, a), (ref, info) in zip(progs, refs):
            x, _ = go(p)
            out.append([bool(np.array_equal(p.result(), ref)), x["iterations"], x["count_edges"], x["active_vertices"]])
        for (p, a), (ref, info) in zip(progs, refs):
            q = type(p)(eng, start_vertex=0, max_iterations=1000)
            for profiled in (False, True):
                q.init_algorithm()
                eng.set_profiling(profiled)
                x, kinds = go(q)
                eng.set_profiling(False)
                ok = np.array_equal(q.result(), ref) and x["iterations"] == info["iterations"] and x["count_edges"] == info["count_edges"]
                out.append([bool(ok), x["iterations"], x["count_edges"], x["active_vertices"]] + (kinds if profiled else []))
print(json.dumps(out))
"""

GEOMETRIES = [(1 << 16, 1 << 16), (1 << 15, 1 << 12), (1 << 16, 1 << 10), (1 << 18, 1 << 10), (1 << 14, 128)]


@pytest.mark.parametrize("n,vpt", GEOMETRIES)
def test_kinds_of_rounds_agree(n, vpt):
    got = {}
    for small in ("0", "8", "16"):
        env = dict(os.environ, CYTOM_SMALL_ROUNDS=small, CYTOM_SPARSE="1", CYTOM_SPARSE_DIV="2")
        r = subprocess.run([sys.executable, "-c", CODE.format(root=str(ROOT), n=n, vpt=vpt)], capture_output=True,
                           text=True, env=env, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        got[small] = json.loads(r.stdout.strip().splitlines()[-1])
    for small, rows in got.items():
        assert all(x[0] for x in rows), (small, rows)
        assert [x[:4] for x in rows] == [x[:4] for x in got["0"]], small
        for x in (y for y in rows if len(y) == 7):
            _, rounds, _, _, dense, other, applies = x
            if small == "0":  # every round is a gather and an apply of its own
                assert applies == rounds and dense + other == rounds, x
            else:  # a small round has no apply launch
                assert applies < rounds, x
    assert sum(x[5] for x in got["0"] if len(x) == 7) > 0  # sparse rounds ran
    assert sum(x[4] for x in got["0"] if len(x) == 7) > 0  # and dense ones
