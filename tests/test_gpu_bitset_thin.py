"""Batches of up to 64 sources on graphs whose rows are all short: both phases
of a push run as one there, up to and past the levels that are bit-sliced, with
equal sources, next to graphs with one longer row that keep the two phases.
Hop distances are compared exactly, closeness to 1e-6 relative."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_bfs_persistent import caterpillar

pytestmark = pytest.mark.gpu

GRAPHS = {
    "rows127": lambda: caterpillar([3, 125, 0, 125] * 12, True),   # the longest short row, 50 levels
    "rows128": lambda: caterpillar([3, 125, 0, 126] * 12, True),   # the shortest long row
    "directed": lambda: caterpillar([1, 5, 0, 120] * 20, False),
    "grid": lambda: gen.grid(13, 300, seed=1),
    "knn": lambda: gen.knn(5000, 8, seed=2),
    "er": lambda: gen.erdos_renyi(40000, 120000, seed=3),
}


@pytest.mark.parametrize("nsrc", [1, 5, 64])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_short_rows(name, nsrc):
    g = GRAPHS[name]()
    srcs = np.random.default_rng(nsrc).integers(0, g.n, nsrc).astype(np.int32)
    srcs[nsrc // 2:] = np.where(np.arange(nsrc - nsrc // 2) % 3, srcs[nsrc // 2:], srcs[0])
    ref, edges, _ = O.mssp(g, srcs)
    want = O.hops_ref_to_api(ref, srcs)
    exp = np.array([O.closeness_hops(ref[i], srcs[i]) for i in range(nsrc)])
    with abi.Graph(g) as dg:
        for ratio in (4, 1000):  # pulls as usual, and hardly any push
            dg.set_option(abi.OPT_PUSH_RATIO, ratio)
            for _ in range(2):
                out, st = dg.bfs(srcs, variant=abi.VARIANT_BITSET)
                assert np.array_equal(out, want) and st.edges_traversed == edges
            cc, _, _ = dg.closeness(srcs)
            assert np.all(np.abs(cc - exp) <= 1e-6 * np.maximum(1.0, np.abs(exp)))
