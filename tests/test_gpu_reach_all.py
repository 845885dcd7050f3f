"""Radii that reach every point, among them those whose square overflows FP64:
the rows, counts and overflow flags are those of all the search points and of
nothing else, whatever the last bucket of the scene is filled up with, on the
single-query and on the packet paths.

Coordinates lie in the unit box, so a radius of 4 holds every point too and
gives the expected rows.
"""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O
from rtdl_b200.batch import B200ProblemBatch
from rtdl_b200.runtime import pack_point_groups

pytestmark = pytest.mark.gpu

RADII = [float("inf"), 1e200, 1e30, 2e19]  # r^2 beyond FP64, beyond FP64, beyond FP32, beyond FP32
SIZES = [1, 5, 7, 8, 9, 1001]  # whole buckets, partly filled ones, more than a query's list holds
LIMITS = [4, 64, 100]


def _cols(n, dim, seed, exact=True):
    p = np.random.default_rng(seed).random((n, dim))
    if exact:
        p = p.astype(np.float32).astype(np.float64)
    d = {"id": np.arange(n, dtype=np.uint32), "x": p[:, 0], "y": p[:, 1]}
    if dim == 3:
        d["z"] = p[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


def _equal(got, exp):
    assert len(got) == len(exp)
    for f in ("query_id", "neighbor_id"):
        assert np.array_equal(got[f], exp[f]), f
    assert np.array_equal(got["distance"].view(np.uint64), exp["distance"].view(np.uint64))


def _rows(view):
    rows = view.to_numpy().copy()
    view.close()
    return rows


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("ns", SIZES)
@pytest.mark.parametrize("dim", [2, 3])
def test_rows_and_overflow(gpu, dim, ns, exact):
    s = _cols(ns, dim, ns, exact)
    for nq in (3, 4737):  # a warp per query; packets
        q = _cols(nq, dim, 7 * nq, exact)
        with rt.B200Scene(_pack(s)) as scene:
            for limit in LIMITS:
                exp, counts = O.fixed_radius_neighbors(q, s, radius=4.0, k_max=limit, threads=8, with_counts=True)
                for radius in RADII if nq == 3 else RADII[:1]:
                    v, overflow = scene.query(_pack(q), predicate="fixed_radius_neighbors", radius=radius,
                                              limit=limit, with_overflow=True)
                    _equal(_rows(v), exp)
                    assert np.array_equal(overflow.astype(bool), counts > limit)
                    _equal(_rows(scene.query(_pack(q), predicate="bounded_knn_rows", radius=radius, limit=limit)), exp)


@pytest.mark.parametrize("ns", SIZES)
def test_plain_call(gpu, ns):
    s, q = _cols(ns, 3, ns), _cols(40, 3, 1)
    for radius in RADII:
        got = _rows(rt.runtime.fixed_radius_neighbors(_pack(q), _pack(s), radius=radius, k_max=64))
        _equal(got, O.fixed_radius_neighbors(q, s, radius=4.0, k_max=64, threads=8))


@pytest.mark.parametrize("nq", [1, 1700])  # five requests: a warp per query; packets
@pytest.mark.parametrize("ns", SIZES)
def test_requests_on_one_scene(gpu, ns, nq):
    import torch

    s, q = _cols(ns, 3, ns), _cols(5 * nq, 3, 4)
    rec = _pack(q).records
    d_q = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    rows = torch.zeros(5 * nq * 64 * 16, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with rt.B200Scene(_pack(s)) as scene:
        off = scene.fixed_radius_neighbors_multi_device(
            d_q.data_ptr(), np.arange(6, dtype=np.uint64) * nq, radius=RADII + [4.0], k_max=64,
            rows_address=rows.data_ptr(), rows_capacity=5 * nq * 64)
    exp = O.fixed_radius_neighbors(q, s, radius=4.0, k_max=64, threads=8)
    assert off.tolist() == [p * nq * min(ns, 64) for p in range(6)]
    _equal(rows[: int(off[-1]) * 16].cpu().numpy().view(exp.dtype), exp)


@pytest.mark.parametrize("nq", [3, 700])
def test_problems_of_a_batch(gpu, nq):
    sizes = SIZES + [1]
    searches = [_cols(n, 3, n) for n in sizes]
    queries = [_cols(nq, 3, 50 + i) for i in range(len(sizes))]
    for radius in RADII:
        with B200ProblemBatch([_pack(s) for s in searches]) as batch:
            out = batch.fixed_radius_neighbors([_pack(q) for q in queries], radius=radius, k_max=64,
                                               with_overflow=True)
        flags = out.overflow.reshape(len(sizes), nq).astype(bool)
        for p, (q, s) in enumerate(zip(queries, searches)):
            exp, counts = O.fixed_radius_neighbors(q, s, radius=4.0, k_max=64, threads=8, with_counts=True)
            _equal(out.problem(p), exp)
            assert np.array_equal(flags[p], counts > 64)


@pytest.mark.parametrize("ns", SIZES)
def test_counts(gpu, ns):
    import torch

    for nq in (3, 4737):
        q2, s2, q3, s3 = _cols(nq, 2, 2), _cols(ns, 2, ns), _cols(nq, 3, 3), _cols(ns, 3, ns)
        out = [torch.zeros(nq, dtype=torch.int32, device="cuda") for _ in range(3)]
        for radius in RADII:
            for threshold in (0, 3, ns, ns + 1):
                counted = min(ns, threshold) if threshold else ns
                rows = rt.fixed_radius_count_threshold_2d(_pack(q2), _pack(s2), radius=radius, threshold=threshold)
                assert {r["neighbor_count"] for r in rows} == {counted}
                assert {r["threshold_reached"] for r in rows} == {int(0 < threshold <= ns)}
                if threshold == 0:
                    continue
                with rt.prepare_b200_fixed_radius_count_threshold_3d(_pack(s3), max_radius=radius) as prep:
                    prep.write_device_count_threshold_columns(
                        _pack(q3), radius=radius, threshold=threshold, query_ids_out=out[0],
                        neighbor_counts_out=out[1], threshold_flags_out=out[2])
                assert (out[1].cpu().numpy() == counted).all()
                assert (out[2].cpu().numpy() == int(threshold <= ns)).all()


@pytest.mark.parametrize("ns", SIZES)
def test_witnesses(gpu, ns):
    s = _cols(ns, 2, ns)
    groups = pack_point_groups([{"id": 0, "point_offset": 0, "point_count": ns, "min_x": 0.0, "min_y": 0.0,
                                 "max_x": 1.0, "max_y": 1.0}])
    for nq in (3, 200):
        q = _cols(nq, 2, 9)
        dist, nid = O.nearest(q, s, threads=8)
        for radius in RADII:
            with rt.prepare_b200_fixed_radius_count_threshold_2d(_pack(s), max_radius=radius) as prep:
                near = prep.nearest_witness_rows(_pack(q), radius=radius)
            with rt.prepare_b200_point_group_nearest_witness_2d(_pack(s), groups, max_radius=radius) as prep:
                grouped = prep.nearest_witness_rows(_pack(q), radius=radius)
                assert prep.count_threshold_reached(_pack(q), radius=radius, threshold=ns) == nq
                assert prep.count_threshold_reached(_pack(q), radius=radius, threshold=ns + 1) == 0
            for rows in (near, grouped):
                assert np.array_equal(np.array([r["neighbor_id"] for r in rows], dtype=np.uint32), nid)
                assert np.array_equal(np.array([r["distance"] for r in rows]).view(np.uint64), dist.view(np.uint64))
