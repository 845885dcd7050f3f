"""KNN where far more points than k tie at the k-th distance: repeated points
whose ids come in every order along the curve (ascending, descending, shuffled,
all equal), so a list entry is displaced early, late or never.  Rows must be
the oracle's bit for bit.  Inexact sets have coordinates that FP32 cannot hold.
"""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cols(p, ids):
    d = {"id": ids.astype(np.uint32), "x": p[:, 0], "y": p[:, 1]}
    if p.shape[1] == 3:
        d["z"] = p[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("order", ["ascending", "descending", "shuffled", "equal"])
def test_repeated_points(gpu, order, dim, exact):
    rng = np.random.default_rng(11)
    sites = rng.random((6, dim))
    p = np.concatenate([np.repeat(sites, [1, 300, 257, 700, 40, 1000], axis=0), rng.random((500, dim))])
    q = np.concatenate([sites[rng.integers(0, 6, 60)], sites[rng.integers(0, 6, 60)] + rng.normal(0, 1e-3, (60, dim)),
                        rng.random((40, dim)), 20 * rng.random((8, dim))])
    if exact:
        p, q = (a.astype(np.float32).astype(np.float64) for a in (p, q))
    n = len(p)
    ids = {"ascending": np.arange(n), "descending": np.arange(n)[::-1], "shuffled": rng.permutation(n),
           "equal": np.full(n, 7)}[order]
    s = _cols(p, ids)
    with rt.B200Scene(_pack(s)) as scene:
        for nq in (len(q), 5000):  # a warp per query; packets, whose crowded queries go to a warp each
            qq = _cols(np.resize(q, (nq, dim)), np.arange(nq))
            for k in (1, 31, 32, 33, 64):
                view = scene.query(_pack(qq), predicate="knn_rows", limit=k)
                got = view.to_numpy()
                exp = O.knn_rows(qq, s, k=k, threads=8)
                assert len(got) == len(exp)
                for f in ("query_id", "neighbor_id", "neighbor_rank"):
                    assert np.array_equal(got[f], exp[f]), (f, k)
                assert np.array_equal(got["distance"].view(np.uint64), exp["distance"].view(np.uint64)), k
                view.close()
