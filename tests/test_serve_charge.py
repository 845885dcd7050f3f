"""What a served request is charged at admission covers what its call allocates
on the device, and not much more.
"""
import re
from pathlib import Path

import numpy as np
import pytest

from rtdl_b200.serve import FRN, KNN, request_bytes

QUERY_CU = Path(__file__).resolve().parents[1] / "rtdl_b200" / "csrc" / "query.cu"


def test_charge_holds_the_slab_of_the_call():
    text = QUERY_CU.read_text()
    slab = int(re.search(r"constexpr int kSlab = (\d+);", text).group(1)) * 4  # u32 point indices
    ranks = 1 << int(re.search(r"constexpr uint32_t kKnnRanks = 1u << (\d+);", text).group(1))
    for dim, rec in ((2, 24), (3, 32)):
        for n in (1, 31, 32, 33, 100_000, ranks, 3 * ranks):
            for k in (1, 16, 64):
                padded = (n + 31) // 32 * 32
                for op, row, held in ((FRN, 16, padded), (KNN, 24, min(n, ranks))):
                    rest = request_bytes(op, n, k, dim) - n * (rec + row * k) - held * slab
                    # records, lists and orders of a probe: 138 bytes with the emit's lists, 109 for KNN
                    assert 138 * n <= rest <= 200 * (padded if op == FRN else n)


def _peak(fn):
    """The most device memory fn() held at once in the stream-ordered pool, beyond what was in use before."""
    from cuda.bindings import driver as cd
    from cuda.bindings import runtime as cr
    import torch

    def attr(pool, name):
        err, value = cr.cudaMemPoolGetAttribute(pool, name)
        assert err == cr.cudaError_t.cudaSuccess
        return int(value)

    err, pool = cr.cudaDeviceGetDefaultMemPool(0)
    assert err == cr.cudaError_t.cudaSuccess
    torch.cuda.synchronize()
    before = attr(pool, cr.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    (err,) = cr.cudaMemPoolSetAttribute(pool, cr.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh, cd.cuuint64_t(0))
    assert err == cr.cudaError_t.cudaSuccess
    fn()
    torch.cuda.synchronize()
    return attr(pool, cr.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh) - before


@pytest.mark.gpu
@pytest.mark.parametrize("op,limit", [(KNN, 1), (KNN, 8), (KNN, 32), (KNN, 64), (FRN, 1), (FRN, 64)])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("probes", [20_000, 300_001])
def test_charge_covers_the_call(gpu, op, limit, dim, probes):
    import torch

    import rtdl_b200 as rt

    def pack(n, seed):
        p = np.random.default_rng(seed).random((n, dim))
        return rt.pack_points(ids=np.arange(n, dtype=np.uint32), x=p[:, 0], y=p[:, 1], z=p[:, 2] if dim == 3 else None)

    rec, row = (32 if dim == 3 else 24), (16 if op == FRN else 24)
    q = torch.from_numpy(pack(probes, 1).records.view(np.uint8).copy()).cuda()
    rows = torch.empty(probes * limit * row, dtype=torch.uint8, device="cuda")
    with rt.B200Scene(pack(100_000, 2)) as scene:
        if op == FRN:
            off = np.array([0, probes // 3, probes], dtype=np.uint64)

            def call():
                scene.fixed_radius_neighbors_multi_device(q.data_ptr(), off, radius=0.005, k_max=limit,
                                                          rows_address=rows.data_ptr(), rows_capacity=probes * limit)
        else:
            def call():
                scene.query_device(q.data_ptr(), probes, predicate=KNN, limit=limit, rows_address=rows.data_ptr(),
                                   rows_capacity=probes * limit)
        held = _peak(call) + probes * (rec + row * limit)
    assert held <= request_bytes(op, probes, limit, dim) <= 1.3 * held
