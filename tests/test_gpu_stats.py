"""The candidate counters (recorded when RTDL_B200_STATS is set as the library
loads, hence the child process) of fixed-radius and KNN queries, on the packet
and the single-query paths."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import json
import numpy as np
import rtdl_b200 as rt
from rtdl_b200 import _native
from oracle import oracle as O

def cols(p):
    return {"id": np.arange(len(p), dtype=np.uint32), "x": p[:, 0], "y": p[:, 1], "z": p[:, 2]}

def pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c["z"])

rng = np.random.default_rng(1)
p = rng.random((8000, 3)).astype(np.float32).astype(np.float64)
p[:400] = p[0]  # more points at one place than a list holds
s = cols(p)
out = []
with rt.B200Scene(pack(s)) as scene:
    for nq in (500, 20000):
        q = cols(rng.random((nq, 3)).astype(np.float32).astype(np.float64))
        scene.query(pack(q), predicate="fixed_radius_neighbors", radius=0.08, limit=64).close()
        got = _native.last_query_stats()
        _, counts = O.fixed_radius_neighbors(q, s, radius=0.08, k_max=64, threads=8, with_counts=True)
        out.append(["frn", nq, got["in_radius"], got["max_count"], int(counts.sum()), int(counts.max())])
        for k in (1, 12):
            scene.query(pack(q), predicate="knn_rows", limit=k).close()
            got = _native.last_query_stats()
            out.append(["knn", nq, got["in_radius"], got["max_count"], nq * k, k])
print("STATS " + json.dumps(out))
"""


def test_candidates_are_counted(gpu):
    root = Path(__file__).resolve().parents[1]
    done = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, RTDL_B200_STATS="1", PYTHONPATH=str(root)))
    assert done.returncode == 0, done.stderr[-2000:]
    line = [x for x in done.stdout.splitlines() if x.startswith("STATS ")][0]
    for kind, nq, total, most, least_total, least in json.loads(line[6:]):
        if kind == "frn":
            assert (total, most) == (least_total, least), nq
        else:  # what a radius that holds the k nearest holds
            assert total >= least_total and most >= least, nq
