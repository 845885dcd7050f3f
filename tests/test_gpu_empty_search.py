"""Calls whose search set holds no point at all: every query answers with a
count of 0, no witness and no rows, through each entry point that walks the
scene instead of returning before it.
"""
import ctypes

import numpy as np
import pytest

import rtdl_b200 as rt
from rtdl_b200 import _native
from rtdl_b200.batch import B200ProblemBatch, B200ProblemBatchGraph, concat_records
from rtdl_b200.runtime import pack_point_groups

pytestmark = pytest.mark.gpu

NQ = [1, 33, 5000]  # a lone query, a packet and a ragged one, more packets than one block's


def _points(n, dim, seed=0):
    p = np.random.default_rng(seed).random((n, dim)).astype(np.float32).astype(np.float64)
    return rt.pack_points(ids=np.arange(n, dtype=np.uint32), x=p[:, 0], y=p[:, 1], z=p[:, 2] if dim == 3 else None)


def _columns(n):
    import torch

    return [torch.full((n,), 77, dtype=torch.int32, device="cuda") for _ in range(3)]


@pytest.mark.parametrize("nq", NQ)
@pytest.mark.parametrize("threshold", [0, 1, 5])
def test_count_3d_device_outputs(gpu, nq, threshold):
    ids, counts, flags = _columns(nq)
    with rt.prepare_b200_fixed_radius_count_threshold_3d(_points(0, 3), max_radius=1.0) as prep:
        prep.write_device_count_threshold_columns(_points(nq, 3), radius=0.5, threshold=threshold, query_ids_out=ids,
                                                  neighbor_counts_out=counts, threshold_flags_out=flags)
    assert np.array_equal(ids.cpu().numpy(), np.arange(nq))
    assert not counts.cpu().numpy().any()
    assert (flags.cpu().numpy() == (threshold == 0)).all()  # the 3-D device contract: threshold 0 is reached


@pytest.mark.parametrize("nq", NQ)
@pytest.mark.parametrize("threshold", [0, 1])
def test_count_2d_device_columns(gpu, nq, threshold):
    import torch

    none = {"ids": torch.zeros(0, dtype=torch.int32, device="cuda"),
            "x": torch.zeros(0, dtype=torch.float64, device="cuda"),
            "y": torch.zeros(0, dtype=torch.float64, device="cuda"), "count": 0}
    qid = torch.arange(nq, dtype=torch.int32, device="cuda")
    qx = torch.rand(nq, dtype=torch.float64, device="cuda")
    ids, counts, flags = _columns(nq)
    torch.cuda.synchronize()
    lib, err = _native.load_library(), _native.error_buffer()
    handle = ctypes.c_void_p()
    _native.check_status(lib.rtdl_b200_prepare_fixed_radius_count_threshold_2d_device_search_columns(
        none["ids"].data_ptr() or None, none["x"].data_ptr() or None, none["y"].data_ptr() or None, 0,
        ctypes.c_double(1.0), ctypes.byref(handle), err, len(err)), err)
    try:
        _native.check_status(lib.rtdl_b200_write_prepared_fixed_radius_count_threshold_2d_device_query_columns(
            handle, qid.data_ptr(), qx.data_ptr(), qx.data_ptr(), nq, 0.5, threshold, ids.data_ptr(),
            counts.data_ptr(), flags.data_ptr(), err, len(err)), err)
    finally:
        lib.rtdl_b200_destroy_prepared_fixed_radius_count_threshold_2d(handle)
    assert np.array_equal(ids.cpu().numpy(), np.arange(nq))
    assert not counts.cpu().numpy().any() and not flags.cpu().numpy().any()


@pytest.mark.parametrize("nq", NQ)
def test_point_groups_of_empty_spans(gpu, nq):
    groups = pack_point_groups([{"id": i, "point_offset": i, "point_count": 0, "min_x": 0.0, "min_y": 0.0,
                                 "max_x": 1.0, "max_y": 1.0} for i in range(3)])
    q = _points(nq, 2)
    with rt.prepare_b200_point_group_nearest_witness_2d(_points(4, 2), groups, max_radius=1.0) as prep:
        for threshold in (0, 2):
            assert not prep.threshold_flags(q, radius=0.5, threshold=threshold).any()
            assert prep.count_threshold_reached(q, radius=0.5, threshold=threshold) == 0
        rows = prep.nearest_witness_rows(q, radius=0.5)
        assert [r["query_id"] for r in rows] == list(range(nq))
        assert all(r["neighbor_id"] == 0xFFFFFFFF and r["distance"] == 3.4028234663852886e38 for r in rows)
        assert prep.nearest_max_distance_row(q, radius=0.5) == {"query_id": 0, "neighbor_id": 0xFFFFFFFF,
                                                                "distance": float("inf")}


@pytest.mark.parametrize("nq", NQ)
def test_batch_graph_with_a_batch_of_empty_problems(gpu, nq):
    import torch

    full = [_points(300, 3, 1), _points(0, 3), _points(9, 3, 2)]
    queries = [_points(nq, 3, 3 + p) for p in range(5)]
    rec = concat_records([q.records for q in queries])
    d_q = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    off = np.arange(6, dtype=np.uint64) * nq
    rows = torch.zeros(5 * nq * 8 * 16, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with B200ProblemBatch([_points(0, 3), _points(0, 3)], dimension=3) as empty, \
            B200ProblemBatch(full, dimension=3) as batch:
        graph = B200ProblemBatchGraph([empty, batch], d_q.data_ptr(), off, radius=0.4, k_max=8,
                                      rows_address=rows.data_ptr(), rows_capacity=5 * nq * 8)
        got, status = graph.replay()
        graph.close()
        exp = batch.fixed_radius_neighbors([q for q in queries[2:]], radius=0.4, k_max=8)
        assert len(empty.fixed_radius_neighbors(queries[:2], radius=0.4, k_max=8)) == 0
    assert status == 0
    assert got[:3].tolist() == [0, 0, 0] and np.array_equal(got[2:], exp.row_offsets)
    n = int(got[-1])
    assert n > 0 and rows[: n * 16].cpu().numpy().tobytes() == exp.rows.tobytes()
