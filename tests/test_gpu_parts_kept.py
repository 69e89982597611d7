"""What a handle's parts are after dawn_graph_set_parts refused new ones, and
where the scratch of the single-CTA tasks cannot be had.  Hop distances against a
BFS of every part alone: the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from pool_limit import pool_limit
from test_gpu_parts_small import ring_with_chords

pytestmark = pytest.mark.gpu


def check(dg, graphs, srcs):
    blocks, _ = dg.multi_bfs(srcs)
    for g, s, b in zip(graphs, srcs, blocks):
        assert np.array_equal(b, O.hops_ref_to_api(O.mssp(g, s)[0], s)), g.n


def test_refused_parts_leave_the_earlier_ones():
    rng = np.random.default_rng(1)
    graphs = [ring_with_chords(n, n) for n in (900, 3, 1200, 40)] + [ring_with_chords(3, 5)] * 60
    srcs = [rng.integers(0, g.n, 20).astype(np.int32) for g in graphs]
    u, off = gen.disjoint_union(graphs)
    with abi.Graph(u) as dg:
        dg.set_parts(off)
        check(dg, graphs, srcs)
        # larger parts, more of them, none: an edge leaves one, an end is wrong
        cut = np.linspace(0, u.n, 500).astype(np.int32)
        for bad in ([0, 450, u.n], np.unique(cut), [0, 900, u.n + 1], [0, 900, 900, u.n]):
            rc = abi.lib().dawn_graph_set_parts(dg.handle, len(bad) - 1, abi._ptr(np.ascontiguousarray(bad, np.int32)))
            assert rc == abi.ERR_INVALID_ARG
            check(dg, graphs, srcs)
        dg.set_parts([0, u.n])  # other parts after the refused ones
        check(dg, [u], [np.array([0, 1500], np.int32)])
        dg.set_parts(off)
        check(dg, graphs, srcs)


def test_without_memory_for_single_cta_tasks():
    # word arrays of a part of 40,000 vertices for every SM: 400 MB; the slots of
    # the clusters that take its place: 130
    rng = np.random.default_rng(2)
    graphs = [ring_with_chords(n, n) for n in (40000, 700)] + [ring_with_chords(300, 5)] * 300
    srcs = [rng.integers(0, g.n, 9).astype(np.int32) for g in graphs]
    u, off = gen.disjoint_union(graphs)
    with abi.Graph(u) as dg:
        with pool_limit(256 << 20):
            dg.set_parts(off)
            check(dg, graphs, srcs)
            dg.synchronize()
            dg.close()
    with abi.Graph(u) as dg:  # and with it
        dg.set_parts(off)
        check(dg, graphs, srcs)
