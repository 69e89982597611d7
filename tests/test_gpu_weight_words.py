"""Weights whose words need care.  Float weights of -0.0 (what -log(1.0f) gives) count as 0.0 in every weighted
form: on a bridge, in a cycle, on a leaf, and where a longer path is found
first.  Compared with the oracle on the same graph with 0.0 in their place;
distances are sums of whole numbers below 2^24, so the tolerance is zero.  A
weight in the source's row that equals the encoding of "unreached" reaches
nothing."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_nearfar import weighted

pytestmark = pytest.mark.gpu


def small():
    """Vertex 0's row and the paths behind it, as in test_weight_words."""
    src, dst = [0, 1, 2, 3, 0, 0, 1, 5], [1, 2, 3, 2, 4, 5, 5, 6]
    return weighted(7, src, dst, [0, 3, 0, 0, 0, 9, 0, 2])


def zeros(g, share, seed):
    """g with a share of its weights zero."""
    w = np.where(np.random.default_rng(seed).random(g.m) < share, 0, g.w_i32).astype(np.int32)
    return gen.CsrGraph(g.n, g.row_ptr, g.col, w, w.astype(np.float32), symmetric=g.symmetric)


GRAPHS = {"small": small, "grid": lambda: zeros(gen.grid(40, 50, seed=1, weights=True), 0.3, 2),
          "hubs": lambda: zeros(gen.rmat(11, 16, a=0.65, b=0.15, c=0.15, seed=3, weights=True), 0.2, 4),
          "all": lambda: zeros(gen.rmat(10, 8, seed=5, weights=True), 1.1, 6)}


@pytest.mark.parametrize("validate", [True, False])
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_negative_zero(graph, validate):
    g = GRAPHS[graph]()
    srcs = np.concatenate([[0], np.random.default_rng(7).integers(0, g.n, 66)]).astype(np.int32)
    want = O.msssp(g, srcs)
    g.w_f32 = np.where(g.w_f32 == 0, np.float32(-0.0), g.w_f32)
    assert np.signbit(g.w_f32).any()
    with abi.Graph(g, weights="f32", validate=validate) as dg:
        # one source and a batch in order; by rows with a light stage (traced), by pushes, by pulls
        for nsrc, variant, force, trace in ((1, abi.VARIANT_DO, 0, 0), (67, abi.VARIANT_AUTO, 0, 0), (5, abi.VARIANT_AUTO, 0, 0),
                                            (67, abi.VARIANT_AUTO, 0, 1), (67, abi.VARIANT_AUTO, 1, 0),
                                            (67, abi.VARIANT_AUTO, 2, 0), (3, abi.VARIANT_DO, 2, 0)):
            dg.set_option(abi.OPT_FORCE_VARIANT, force)
            dg.trace(trace)
            d, _ = dg.sssp(srcs[:nsrc], variant=variant)
            assert np.array_equal(d, want[:nsrc]), (nsrc, variant, force, trace)


def test_negative_weights_of_an_unvalidated_handle_end():
    # not part of the contract, but the levels' limit of n holds for them
    g = weighted(4, [0, 1, 2, 1], [1, 2, 1, 3], [5, 3, -4, 1])
    with abi.Graph(g, weights="i32", validate=False) as dg:
        for srcs, variant in (([0], abi.VARIANT_DO), ([0, 1], abi.VARIANT_AUTO)):
            d, st = dg.sssp(srcs, variant=variant)
            assert d.shape == (len(srcs), 4) and st.levels <= 2 * g.n


@pytest.mark.parametrize("weights", ["i32", "f32"])
def test_source_row_weight_of_unreached(weights):
    top = abi.INT32_MAX if weights == "i32" else abi.FLT_MAX
    g = weighted(5, [0, 1, 0, 3], [1, 2, 3, 4], [1, 1, 5, 2])
    g.w_i32[0], g.w_f32[0] = abi.INT32_MAX, abi.FLT_MAX
    with abi.Graph(g, weights=weights) as dg:
        for srcs, variant in (([0], abi.VARIANT_DO), ([0, 0, 0], abi.VARIANT_AUTO)):
            d, _ = dg.sssp(srcs, variant=variant)
            assert (d == np.array([0, top, top, 5, 7], d.dtype)).all(), (variant, d)
