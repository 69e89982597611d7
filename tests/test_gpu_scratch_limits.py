"""Calls whose preferred form needs more scratch than there is take the form that
needs less, with the same distances (whole numbers: the tolerance is zero)."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from pool_limit import pool_limit
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu


def test_ordered_batch_without_lists():
    # 64 sources: lists and masks 105 MB and the block 26; by rows 30 in all
    import torch
    g = gen.knn(100000, 6, seed=1, weights=True)
    srcs = gen.sources(g, 64, seed=2)
    want = O.msssp(g, srcs)
    out = torch.empty((64, g.n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with abi.Graph(g, weights="i32") as dg:
        with pool_limit(64 << 20):
            for k in (64, 3, 64):  # three sources fit in order
                out.fill_(0)
                torch.cuda.synchronize()
                dg.sssp_device(srcs[:k], out.data_ptr())
                assert np.array_equal(to_ref(out[:k].cpu().numpy()), want[:k]), k
            dg.close()


def test_bfs_without_records():
    # records of 1.5 M grid vertices 48 MB, the queues and bitmaps 13 and the segments
    import torch
    g = gen.grid(1250, 1200, seed=3)
    srcs = np.array([0, g.n // 2], np.int32)
    want = O.hops_ref_to_api(O.mssp(g, srcs)[0], srcs)
    out = torch.empty((2, g.n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with abi.Graph(g) as dg:
        with pool_limit(32 << 20):
            for _ in range(2):
                out.fill_(0)
                torch.cuda.synchronize()
                dg.bfs_device(srcs, out.data_ptr(), variant=abi.VARIANT_DO)
                assert np.array_equal(out.cpu().numpy(), want)
        dg.bfs_device(srcs, out.data_ptr(), variant=abi.VARIANT_DO)  # with them
        assert np.array_equal(out.cpu().numpy(), want)
