"""The persistent launch of the single-source BFS where it changes form: rows
around the lengths that have a record, are walked by a lane and are cut into
segments; levels that outgrow one CTA's lists; vertex counts around the bitmap
that fits its shared memory; both directions, next to the level kernels of the
traced form.  Hop distances are integers: the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu


def csr(n, src, dst, symmetric):
    if symmetric:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    return gen.CsrGraph(n, rp, dst[order].astype(np.int32), symmetric=symmetric)


def tree(branch, depth, symmetric=True):
    n = (branch ** (depth + 1) - 1) // (branch - 1)
    child = np.arange(1, n)
    return csr(n, (child - 1) // branch, child, symmetric)


def caterpillar(lens, symmetric):
    """A path whose vertices carry as many leaves as `lens` says, and on."""
    src, dst, n = [], [], len(lens)
    src += list(range(n - 1))
    dst += list(range(1, n))
    for i, k in enumerate(lens):
        src += [i] * k
        dst += list(range(n, n + k))
        n += k
    return csr(n, np.array(src), np.array(dst), symmetric)


ROWS = [6, 7, 8, 9, 14, 15, 16, 29, 30, 31, 32, 33]
GRAPHS = {
    "one": lambda: csr(1, np.zeros(0, np.int64), np.zeros(0, np.int64), True),
    "pair": lambda: csr(2, np.array([0]), np.array([1]), False),
    "grid": lambda: gen.grid(90, 70, seed=1),
    "path": lambda: csr(3000, np.arange(2999), np.arange(1, 3000), False),
    "records8": lambda: caterpillar([0] * 300 + [4, 5, 6] * 40, True),
    "records32": lambda: caterpillar([0] * 100 + ROWS[:11] * 10, True),
    "records_none": lambda: caterpillar([0] * 100 + ROWS * 10, True),
    "records_directed": lambda: caterpillar([0] * 100 + ROWS[:11] * 10, False),
    "segments": lambda: caterpillar([0, 1, 125, 126, 127, 128, 129, 255, 256, 257, 5000, 3, 2000] * 3, True),
    "tree7": lambda: tree(7, 5),         # a level past the lists, rows with records
    "tree7_directed": lambda: tree(7, 5, False),
    "tree40": lambda: tree(40, 3),       # 64,000 vertices at once, no records
    "knn": lambda: gen.knn(3000, 8, seed=2),
    "er": lambda: gen.erdos_renyi(20000, 100000, seed=3),
    "rmat": lambda: gen.rmat(14, 16, seed=4),
}


def check(g, srcs, dg, **kw):
    ref, edges, _ = O.mssp(g, srcs)
    want = O.hops_ref_to_api(ref, srcs)
    got, st = dg.bfs(srcs, **kw)
    assert np.array_equal(got, want), kw
    assert st.edges_traversed == edges
    return st


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_forms(name):
    g = GRAPHS[name]()
    rng = np.random.default_rng(len(name))
    srcs = np.concatenate([[0, g.n - 1], rng.integers(0, g.n, 3)]).astype(np.int32)
    with abi.Graph(g) as dg:
        for force in (0, 1, 2):
            dg.set_option(abi.OPT_FORCE_VARIANT, force)
            for small in (1, 0):
                dg.set_option(abi.OPT_SMALL_LEVELS, small)
                st = check(g, srcs, dg, variant=abi.VARIANT_DO)
                check(g, srcs[:1], dg, variant=abi.VARIANT_PUSH)
                dg.trace(True)
                traced = check(g, srcs, dg, variant=abi.VARIANT_DO)
                dg.trace(False)
                assert st.levels == traced.levels


@pytest.mark.parametrize("rows,cols", [(1264, 1265), (1265, 1265)])
def test_bitmap_limit(rows, cols):
    g = gen.grid(rows, cols, seed=5)
    with abi.Graph(g) as dg:
        check(g, np.array([rows * cols // 2 + 7], np.int32), dg, variant=abi.VARIANT_DO)
