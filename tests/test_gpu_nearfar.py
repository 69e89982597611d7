"""The ordered weighted traversal (csrc/nearfar.cu) against the oracle, at the
sizes where its lists, row forms and batch strides change.  Distances are
sums of whole numbers below 2^24, so the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu


def weighted(n, src, dst, w):
    """Directed CSR of an edge list, rows in list order."""
    src = np.asarray(src, np.int64)
    order = np.argsort(src, kind="stable")
    rp = np.zeros(n + 1, np.int32)
    np.add.at(rp, src + 1, 1)
    w = np.asarray(w, np.int32)[order]
    return gen.CsrGraph(n, np.cumsum(rp).astype(np.int32), np.asarray(dst, np.int32)[order], w, w.astype(np.float32))


def path(n, w):
    k = np.arange(n - 1)
    return weighted(n, k, k + 1, np.resize(w, n - 1))


def fan(leaves):
    """0 -> every leaf (weights 1, 2, ..) -> a chain back to one sink, heavy
    edges first: leaves wait in the far list and come back one bucket at a
    time; rows of 127, 128 and 129 entries straddle the segment form."""
    k = np.arange(1, leaves + 1)
    n = leaves + 2
    return weighted(n, np.concatenate([0 * k, k]),
                    np.concatenate([k, np.full(leaves, n - 1)]), np.concatenate([k, 2 * leaves - k]))


GRAPHS = {
    "one_vertex": lambda: weighted(1, [0], [0], [5]),
    "no_edges": lambda: weighted(3, [], [], []),
    "path_one_cta": lambda: path(700, [3, 1, 50]),
    "path_zero_weights": lambda: path(300, [0]),
    "path_gaps": lambda: path(90, [1, 1, 90000]),
    "fan127": lambda: fan(127),
    "fan128": lambda: fan(128),
    "fan1025": lambda: fan(1025),  # more than a single-CTA list holds
    "grid": lambda: gen.grid(37, 53, seed=5, weights=True),
    "rmat_hubs": lambda: gen.rmat(11, 16, a=0.65, b=0.15, c=0.15, seed=6, weights=True),
}


@pytest.mark.parametrize("weights", ["i32", "f32"])
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_single_source(graph, weights):
    g = GRAPHS[graph]()
    srcs = np.unique(np.array([0, g.n // 2, g.n - 1], np.int32))
    with abi.Graph(g, weights=weights) as dg:
        for _ in range(2):  # a second call starts from the first one's lists
            d, st = dg.sssp(srcs, variant=abi.VARIANT_DO)
            assert np.array_equal(to_ref(d), O.msssp(g, srcs))


@pytest.mark.parametrize("nsrc", [2, 4, 5, 8, 9, 17, 33, 64, 65, 130])
@pytest.mark.parametrize("graph", ["grid", "fan128", "rmat_hubs"])
def test_batch_strides(graph, nsrc):
    # batches are 4, 8, 16, 32 or 64 distances wide, the last one ragged
    g = GRAPHS[graph]()
    srcs = np.random.default_rng(nsrc).integers(0, g.n, nsrc).astype(np.int32)
    with abi.Graph(g, weights="f32" if nsrc % 2 else "i32") as dg:
        d, st = dg.sssp(srcs)
        assert np.array_equal(to_ref(d), O.msssp(g, srcs))
        assert st.batches == (nsrc + 63) // 64


def test_calls_of_other_widths_in_between():
    # one handle, wide and narrow batches, single sources and forced levels
    # in turn: every call finds the lists and masks another form left behind
    g = gen.knn(3000, 6, seed=9, weights=True)
    srcs = gen.sources(g, 70, seed=10)
    want = O.msssp(g, srcs)
    with abi.Graph(g, weights="i32") as dg:
        for k, force in ((70, 0), (3, 0), (1, 0), (40, 1), (64, 0), (5, 2), (70, 0)):
            dg.set_option(abi.OPT_FORCE_VARIANT, force)
            d, _ = dg.sssp(srcs[:k])
            assert np.array_equal(to_ref(d), want[:k]), (k, force)
