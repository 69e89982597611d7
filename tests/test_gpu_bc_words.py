"""Betweenness from level words, where its kernels change form: one to five
blocks of 64 sources, every batch width, rows around the lengths at which they
are cut into segments, and graphs around the depth from which level rows take
the words' place.  Terms are float32, added in another grouping than the
oracle's: the bar is float rounding, 1e-4 relative, as for the other
betweenness tests."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu


def csr(n, edges):
    e = np.array(sorted(edges), np.int64).reshape(-1, 2)
    rp = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int32)
    return gen.CsrGraph(n, rp, e[:, 1].astype(np.int32))


def stars(directed):
    """Hubs of 63 to 193 leaves in a cycle, leaves shared between hubs."""
    hubs, leaves = [63, 64, 65, 127, 128, 129, 191, 192, 193], 200
    n, rng, edges = len(hubs) + leaves, np.random.default_rng(3), set()
    for h, d in enumerate(hubs):
        for x in rng.permutation(leaves)[:d]:
            edges.add((h, len(hubs) + int(x)))
            if not directed or (h + x) % 3:
                edges.add((len(hubs) + int(x), h))
        edges.add((h, (h + 1) % len(hubs)))
    return csr(n, edges)


def ladder(depth):
    """Two vertices per level, joined both ways: depth levels below vertex 0."""
    edges = set()
    for l in range(depth):
        for a in (2 * l, 2 * l + 1):
            for b in (2 * l + 2, 2 * l + 3):
                edges |= {(a, b), (b, a)}
    return csr(2 * depth + 2, edges)


GRAPHS = {"stars": lambda: stars(False), "stars_directed": lambda: stars(True), "depth30": lambda: ladder(30),
          "depth31": lambda: ladder(31), "depth32": lambda: ladder(32), "depth40": lambda: ladder(40),
          "er": lambda: gen.erdos_renyi(1500, 6000, seed=8), "rmat": lambda: gen.rmat(11, 16, seed=9),
          "pair": lambda: csr(2, {(0, 1)}), "loops": lambda: csr(3, {(0, 0), (0, 1), (1, 2), (2, 2)})}


@pytest.mark.parametrize("width", [0, 1, 2, 4])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_blocks_and_rows(name, width):
    g = GRAPHS[name]()
    rng = np.random.default_rng(5)
    with abi.Graph(g) as dg:
        dg.set_option(abi.OPT_BITSET_WIDTH, width)
        for nsrc in (1, 64, 300, 65, 129):
            srcs = rng.integers(0, g.n, nsrc).astype(np.int32)
            want = O.bc(g, srcs)
            got, st = dg.betweenness(srcs)
            assert st.batches == -(-nsrc // 64)
            np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-6 * max(1.0, float(np.abs(want).max())))
