"""Weighted batches on either side of the line between the ordered pairs and the
64-source rows: hubs with spread and with equal lengths, random graphs of low degree
and meshes, sources on both sides, against single-source calls (and the oracle for
two of them).  Lengths are whole numbers: the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu


def equal(g):
    return gen.CsrGraph(g.n, g.row_ptr, g.col, np.full(g.m, 7, np.int32), np.full(g.m, 7, np.float32), symmetric=g.symmetric)


GRAPHS = {
    "hub": (lambda: gen.rmat(16, 8, seed=1, weights=True), (16, 17, 40)),
    "hub_equal": (lambda: equal(gen.rmat(17, 16, seed=2)), (20, 40, 64)),
    "random": (lambda: gen.erdos_renyi(300000, 2400000, seed=3, weights=True), (45, 47, 64)),
    "random_dense": (lambda: gen.erdos_renyi(100000, 4000000, seed=4, weights=True), (33, 36, 64)),
    "mesh": (lambda: gen.knn(150000, 8, seed=5, weights=True), (60, 64, 70)),
}


@pytest.mark.parametrize("weights", ["i32", "f32"])
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_both_sides(graph, weights):
    import torch
    make, widths = GRAPHS[graph]
    g = make()
    srcs = gen.sources(g, max(widths), seed=6, from_lcc=False)
    kind = torch.int32 if weights == "i32" else torch.float32
    with abi.Graph(g, weights=weights) as dg:
        one = torch.empty((len(srcs), g.n), dtype=kind, device="cuda")
        many = torch.empty((len(srcs), g.n), dtype=kind, device="cuda")
        torch.cuda.synchronize()
        dg.sssp_device(srcs, one.data_ptr(), variant=abi.VARIANT_DO)
        assert np.array_equal(to_ref(one[:2].cpu().numpy()), O.msssp(g, srcs[:2]))
        for k in widths:
            many.fill_(-1)
            torch.cuda.synchronize()
            dg.sssp_device(srcs[:k], many.data_ptr())
            assert torch.equal(many[:k], one[:k]), k
