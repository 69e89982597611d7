"""The batched min-plus traversal's light stage and bounds (csrc/msssp.cu)
against the oracle: weights that do and do not tell light edges apart, zero
and real-valued weights, sources that never reach the hub, graphs without a
hub, rows of every length around the segments.  A traced call takes these
kernels at any size.  Distances are compared exactly: any order of relaxations
reaches the same least sums, whole numbers below 2^24 or single-precision sums
along the path."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu


def reweighted(g, w):
    w = np.asarray(w)
    return gen.CsrGraph(g.n, g.row_ptr, g.col, w.astype(np.int32), w.astype(np.float32), symmetric=g.symmetric)


def two_parts():
    """An RMAT graph with a hub and a second component that never reaches it."""
    a, b = gen.rmat(11, 16, seed=1), gen.rmat(9, 8, seed=2)
    rp = np.concatenate([a.row_ptr, a.row_ptr[-1] + b.row_ptr[1:]]).astype(np.int32)
    return gen.CsrGraph(a.n + b.n, rp, np.concatenate([a.col, b.col + a.n]).astype(np.int32), symmetric=True)


TOPOLOGY = {"rmat": lambda: gen.rmat(12, 16, seed=3), "dense": lambda: gen.rmat(8, 64, seed=4),
            "two_parts": two_parts, "er": lambda: gen.erdos_renyi(4000, 60000, seed=5),
            "grid": lambda: gen.grid(30, 40, seed=6), "sparse": lambda: gen.rmat(12, 2, seed=7)}
WEIGHTS = {"spread": lambda r, m: r.integers(1, 64, m), "equal": lambda r, m: np.full(m, 7),
           "two": lambda r, m: np.where(r.random(m) < 0.2, 1, 1000), "zero": lambda r, m: r.integers(0, 3, m),
           "wide": lambda r, m: r.integers(1, 1 << 18, m)}


@pytest.mark.parametrize("weights", sorted(WEIGHTS))
@pytest.mark.parametrize("topology", sorted(TOPOLOGY))
def test_stages(topology, weights):
    rng = np.random.default_rng(len(topology) + 10 * len(weights))
    g = TOPOLOGY[topology]()
    g = reweighted(g, WEIGHTS[weights](rng, g.m))
    srcs = rng.integers(0, g.n, 70).astype(np.int32)
    want = O.msssp(g, srcs)
    for w in ("i32", "f32"):
        for seg in (1024, 128):
            with abi.Graph(g, weights=w) as dg:
                dg.set_option(abi.OPT_PULL_SEGMENT, seg)
                dg.trace(True)
                for nsrc in (70, 64, 2):
                    d, _ = dg.sssp(srcs[:nsrc])
                    bad = np.argwhere(to_ref(d) != want[:nsrc])
                    assert bad.size == 0, (w, seg, nsrc, bad[:5])


@pytest.mark.parametrize("real", [False, True])
def test_large_batch(real):
    g = gen.rmat(16, 16, seed=8, weights=True)
    srcs = gen.sources(g, 66, seed=9)
    if real:
        w = np.random.default_rng(10).random(g.m).astype(np.float32) * 60
        g = gen.CsrGraph(g.n, g.row_ptr, g.col, g.w_i32, w, symmetric=True)
        with abi.Graph(g, weights="f32") as dg:
            d, _ = dg.sssp(srcs)
            one, _ = dg.sssp(srcs, variant=abi.VARIANT_DO)
        assert np.array_equal(d, one)
        return
    want = O.msssp(g, srcs)
    for w in ("i32", "f32"):
        with abi.Graph(g, weights=w) as dg:
            for _ in range(2):
                d, st = dg.sssp(srcs)
                assert np.array_equal(to_ref(d), want) and st.pull_levels > 0
