"""The batched traversal's persistent launch: word widths, ragged batches,
graphs from one vertex to one that needs every CTA, few and many levels, both
directions, one handle through all of them, next to the traced form that
launches every step by itself.  Hop distances are integers: the tolerance is
zero; closeness is summed in 64-bit integers and agrees to 1e-6 relative."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu


def path(n):
    rp = np.minimum(np.arange(n + 1), n - 1).astype(np.int32)
    return gen.CsrGraph(n, rp, np.arange(1, n, dtype=np.int32))


GRAPHS = {
    "one": lambda: gen.CsrGraph(1, np.zeros(2, np.int32), np.zeros(0, np.int32)),
    "no_edges": lambda: gen.CsrGraph(33, np.zeros(34, np.int32), np.zeros(0, np.int32)),
    "pair": lambda: path(2),
    "path": lambda: path(700),                        # past the bit-sliced levels
    "grid": lambda: gen.grid(150, 120, seed=2),
    "er": lambda: gen.erdos_renyi(3000, 20000, seed=4),
    "hubs": lambda: gen.rmat(13, 16, seed=5),         # heavy rows, several segments
    "all_ctas": lambda: gen.rmat(17, 8, seed=6),
}


@pytest.mark.parametrize("force", [0, 1, 2, 3])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_widths_and_batches(name, force):
    g = GRAPHS[name]()
    rng = np.random.default_rng(len(name))
    srcs = rng.integers(0, g.n, 300).astype(np.int32)
    ref, _, _ = O.mssp(g, srcs)
    want = O.hops_ref_to_api(ref, srcs)
    with abi.Graph(g) as dg:
        dg.set_option(abi.OPT_FORCE_VARIANT, force)
        for width, nsrc in [(4, 300), (1, 65), (2, 1), (4, 256), (1, 64), (2, 300)]:
            dg.set_option(abi.OPT_BITSET_WIDTH, width)
            out, st = dg.bfs(srcs[:nsrc], variant=abi.VARIANT_BITSET)
            assert np.array_equal(out, want[:nsrc]), (width, nsrc)
            dg.trace(True)
            out, traced = dg.bfs(srcs[:nsrc], variant=abi.VARIANT_BITSET)
            dg.trace(False)
            assert np.array_equal(out, want[:nsrc]), (width, nsrc)
            assert (st.levels, st.edges_traversed) == (traced.levels, traced.edges_traversed)
            cc, _, _ = dg.closeness(srcs[:nsrc])
            exp = np.array([O.closeness_hops(ref[i], srcs[i]) for i in range(nsrc)])
            assert np.all(np.abs(cc - exp) <= 1e-6 * np.maximum(1.0, np.abs(exp))), (width, nsrc)
