"""Single-source BFS of graphs of low degree at the sizes and growths where its form
changes (records on one SM, level kernels, the persistent launch alone), against the
oracle.  Hop distances are integers: the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_growth_rule import lattice3

pytestmark = pytest.mark.gpu

GRAPHS = {f"random_{n}_{d}": (lambda n=n, d=d: gen.erdos_renyi(n, int(n * d), seed=n))
          for n in (5999, 6000, 25999, 26000, 32769, 45000, 45001, 200000) for d in (1.2, 2.5, 4, 7, 11)}
GRAPHS.update({"knn_6000": lambda: gen.knn(6000, 8, seed=1), "knn_33000": lambda: gen.knn(33000, 8, seed=2),
               "grid": lambda: gen.grid(200, 250), "lattice": lambda: lattice3(30)})


@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_forms(graph):
    g = GRAPHS[graph]()
    srcs = np.concatenate([gen.sources(g, 2, seed=3, from_lcc=False), [0, g.n - 1]]).astype(np.int32)
    want = O.hops_ref_to_api(O.mssp(g, srcs)[0], srcs)
    with abi.Graph(g) as dg:
        for variant in (abi.VARIANT_DO, abi.VARIANT_PUSH):
            d, st = dg.bfs(srcs, variant=variant)
            assert np.array_equal(d, want), variant
        dg.set_option(abi.OPT_SMALL_LEVELS, 0)
        d, _ = dg.bfs(srcs, variant=abi.VARIANT_DO)
        assert np.array_equal(d, want)
