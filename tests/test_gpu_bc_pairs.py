"""Betweenness of deep batches: pairs by level on graphs of short rows, up to
more levels than are counted in shared memory, next to graphs with one row that
is long enough for the level rows.  Float rounding bounds the difference, 1e-4
relative, as for the other betweenness tests."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_bfs_persistent import caterpillar, csr

pytestmark = pytest.mark.gpu


def looped_path(n):
    """A path with a self loop at its middle."""
    k = np.arange(n - 1)
    return csr(n, np.concatenate([k, [n // 2]]), np.concatenate([k + 1, [n // 2]]), False)


GRAPHS = {
    "path4097": lambda: looped_path(4097),
    "path5000": lambda: looped_path(5000),
    "grid": lambda: gen.grid(20, 45, seed=1),
    "knn": lambda: gen.knn(3000, 8, seed=2),
    "rows127": lambda: caterpillar([0] * 40 + [125, 3, 60] * 4, True),
    "rows128": lambda: caterpillar([0] * 40 + [126, 3, 60] * 4, True),
    "directed": lambda: caterpillar([0] * 40 + [120, 3, 60] * 4, False),
}


@pytest.mark.parametrize("nsrc", [1, 66, 200])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_deep(name, nsrc):
    g = GRAPHS[name]()
    srcs = np.random.default_rng(nsrc).integers(0, g.n, nsrc).astype(np.int32)
    srcs[0] = 0
    want = O.bc(g, srcs)
    with abi.Graph(g) as dg:
        for _ in range(2):
            got, st = dg.betweenness(srcs)
            np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-6 * max(1.0, float(np.abs(want).max())))
    assert st.levels >= 32
