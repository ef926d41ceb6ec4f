"""Sparse rounds over frontier lists of every shape: one tile, a few, 64 (a mask bit per column),
256 (a bit per four columns); hubs whose word reaches every column next to words that reach
one; items of no, some and thousands of edges; fewer list entries than blocks, and more than
the blocks hold at once. Sparse rounds are forced up to half of the words; bit for bit against
the oracle."""
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
n, vpt, kind = {n}, {vpt}, {kind!r}
rng = np.random.default_rng(n + vpt)
if kind == "hubs":
    hubs = np.array([0, 1, n // 2, n - 1])
    s = np.concatenate([np.repeat(hubs, 9000), rng.integers(0, n, 60000), np.arange(0, n - 33, 3)])
    t = np.concatenate([rng.integers(0, n, 36000), rng.integers(0, n, 60000), np.arange(33, n, 3)[: len(range(0, n - 33, 3))]])
else:  # every word of the list non-zero at once
    far = np.arange(32, n, 64)
    s = np.concatenate([np.zeros(len(far), int), far])
    t = np.concatenate([far, far[rng.permutation(len(far))] + 1])
s, t = s.astype(np.uint32), t.astype(np.uint32)
w = orc.edge_weights(s, t, 3, 1, 1000)
cut = len(s) * 9 // 10
order = rng.permutation(len(s))
ok = []
with cg.Engine(n, vpt, weight_type=cg.WEIGHT_U32) as eng:
    progs = [(cg.BFS(eng, start_vertex=0, max_iterations=1000), 0), (cg.SSSP(eng, start_vertex=0, max_iterations=1000), 2)]
    st = orc.Store(n, vpt, True)
    for part in (order[:cut], order[cut:]):
        for x in (eng, st):
            (x.insert_edges if x is eng else x.insert)(s[part], t[part], w[part])
        eng.do_global_compaction()
        st.compact()
        for p, algo in progs:
            p.execute_algorithm()
            ok.append(bool(np.array_equal(p.result(), st.run_minprop(algo, start=0, max_iter=1000)[0])))
print(json.dumps(ok))
"""


@pytest.mark.parametrize("n,vpt,kind", [(1 << 16, 1 << 16, "hubs"), (1 << 15, 1 << 12, "hubs"), (1 << 16, 1 << 10, "hubs"),
                                        (1 << 18, 1 << 10, "hubs"),
                                        (1 << 24, 1 << 16, "wide")])
def test_sparse_lists(n, vpt, kind):
    env = dict(os.environ, CYTOM_SPARSE="1", CYTOM_SPARSE_DIV="2")
    r = subprocess.run([sys.executable, "-c", CODE.format(root=str(ROOT), n=n, vpt=vpt, kind=kind)],
                       capture_output=True, text=True, env=env, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    ok = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(ok) == 4 and all(ok), ok
