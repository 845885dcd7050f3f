"""The number of queries up to which a call's queries walk alone depends on the
scene's points and dimension: on both sides of each line every call gives the
same rows, and those of the oracle for a sample.
"""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cols(p):
    d = {"id": np.arange(len(p), dtype=np.uint32), "x": p[:, 0], "y": p[:, 1]}
    if p.shape[1] == 3:
        d["z"] = p[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


def _first(c, n):
    return {k: v[:n] for k, v in c.items()}


# 3D: 14,208 queries, or one per 10 points; 2D: 4,736, or one per 50 points
@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("dim,ns,line", [(3, 3000, 14208), (3, 240_000, 24_000), (2, 3000, 4736), (2, 300_000, 6000)])
def test_rows_on_both_sides_of_the_line(gpu, dim, ns, line, exact):
    rng = np.random.default_rng(ns + dim)
    p = np.concatenate([rng.random((ns - 600, dim)), 0.5 + 0.001 * rng.random((600, dim))])  # a spot crowded with 600
    q = np.concatenate([rng.random((line - 40, dim)), 0.5 + 0.001 * rng.random((32, dim)), 3.0 * rng.random((9, dim))])
    if exact:
        p, q = (a.astype(np.float32).astype(np.float64) for a in (p, q))
    s, q = _cols(p), _cols(rng.permutation(q))
    sample = _first(q, 150)
    radius = (20 / (ns * 4.19)) ** (1 / 3) if dim == 3 else (20 / (ns * 3.14)) ** 0.5
    calls = [("fixed_radius_neighbors", radius, 64), ("fixed_radius_neighbors", radius, 1), ("bounded_knn_rows", radius, 8),
             ("knn_rows", 0.0, 1), ("knn_rows", 0.0, 33)]
    with rt.B200Scene(_pack(s)) as scene:
        for predicate, r, limit in calls:
            rows = []
            for n in (line, line + 1):
                v = scene.query(_pack(_first(q, n)), predicate=predicate, radius=r, limit=limit)
                rows.append(v.to_numpy().copy())
                v.close()
            few, more = rows
            for f in few.dtype.names:  # (field by field: records have padding)
                assert more[f][: len(few)].tobytes() == few[f].tobytes(), f
            if predicate == "knn_rows":
                exp = O.knn_rows(sample, s, k=limit, threads=8)
            else:
                exp = O.fixed_radius_neighbors(sample, s, radius=r, k_max=limit, threads=8)
            for f in ("query_id", "neighbor_id"):
                assert np.array_equal(few[f][: len(exp)], exp[f])
            assert np.array_equal(few["distance"][: len(exp)].view(np.uint64), exp["distance"].view(np.uint64))
        nearest = [scene.directed_hausdorff(_pack(_first(q, n)), with_nearest=True) for n in (line, line + 1)]
    (_, d0, i0), (_, d1, i1) = nearest
    assert np.array_equal(d1[:line].view(np.uint64), d0.view(np.uint64)) and np.array_equal(i1[:line], i0)
    dist, nid = O.nearest(sample, s, threads=8)
    assert np.array_equal(d0[:150].view(np.uint64), dist.view(np.uint64)) and np.array_equal(i0[:150], nid)
    assert nearest[0][0]["distance"] == d0.max()
