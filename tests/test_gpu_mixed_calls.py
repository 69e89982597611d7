"""One handle, calls of different forms and lengths in turn: the captured graphs
of the level kernels hold the address of the control block, and a long source
list in between must not move it.  Distances are whole numbers, so the tolerance
is zero; a guard row around each result shows writes beside it."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu

GUARD = -77


def device_rows(call, k, n):
    """call(pointer) into k rows with a row of guard words before and behind."""
    import torch
    buf = torch.full((k + 2, n), GUARD, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    call(buf[1].data_ptr())
    rows = buf.cpu().numpy()
    assert (rows[0] == GUARD).all() and (rows[-1] == GUARD).all()
    return rows[1:-1]


def test_level_kernel_bfs_between_long_weighted_lists():
    # rows of 9 to 32 entries, 40,000 vertices: single-source BFS by level kernels
    g = gen.knn(40000, 8, seed=11, weights=True)
    srcs = gen.sources(g, 6, seed=12)
    hops = O.hops_ref_to_api(O.mssp(g, srcs)[0], srcs)
    far = O.msssp(g, srcs)
    with abi.Graph(g, weights="i32") as dg:
        for i, s in enumerate(srcs):
            d = device_rows(lambda p: dg.bfs_device([s], p), 1, g.n)
            assert np.array_equal(d, hops[i:i + 1]), i
            many = np.resize(srcs, 40 << i)  # a longer list each time
            d = device_rows(lambda p: dg.sssp_device(many, p, variant=abi.VARIANT_DO), len(many), g.n)
            assert np.array_equal(to_ref(d), far[np.arange(len(many)) % len(srcs)]), i


def test_forced_weighted_levels_between_long_lists():
    g = gen.rmat(11, 8, seed=13, weights=True)
    srcs = gen.sources(g, 4, seed=14)
    want = O.msssp(g, srcs)
    with abi.Graph(g, weights="i32") as dg:
        for i, s in enumerate(srcs):
            for force in (1, 2):
                dg.set_option(abi.OPT_FORCE_VARIANT, force)
                d = device_rows(lambda p: dg.sssp_device([s], p, variant=abi.VARIANT_DO), 1, g.n)
                assert np.array_equal(to_ref(d), want[i:i + 1]), (i, force)
                dg.set_option(abi.OPT_FORCE_VARIANT, 0)
                many = np.resize(srcs, 100 << (2 * i + force))
                d, st = dg.sssp(many, variant=abi.VARIANT_DO)
                assert np.array_equal(to_ref(d), want[np.arange(len(many)) % len(srcs)]), (i, force)
                assert st.batches == len(many) and st.edges_traversed > 0
