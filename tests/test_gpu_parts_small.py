"""Many graphs in one call, at the sizes where a part's words stop fitting a
quarter, half and all of one SM's shared memory and where its ids stop fitting
16 bits, against a BFS of every part alone.  Hop distances are integers: the
tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu

SMEM = 231424  # the device's 227 KB less 1 KB, in whole 128-byte lines


def around(nbytes):
    """Part sizes just within and just beyond `nbytes` of 32-bit words."""
    fit = (nbytes - 16) // 4 - 1
    return [fit, fit + 1]


SIZES = {
    "tiny": [1, 2, 31, 32, 33, 1000],
    "quarter": around(SMEM // 4 - 1024),
    "half": around(SMEM // 2 - 1024),
    "32_bits": around(SMEM),
    "16_bit_ids": [65535, 65536],
    "mixed": [5, 40000, 300, 120000, 64],
}


def ring_with_chords(n, seed):
    """A directed ring (so that every vertex has a row) with random chords."""
    rng = np.random.default_rng(seed)
    extra = 3 * n
    src = np.concatenate([np.arange(n), rng.integers(0, n, extra)])
    dst = np.concatenate([(np.arange(n) + 1) % n, rng.integers(0, n, extra)])
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    return gen.CsrGraph(n, rp, dst[order].astype(np.int32))


@pytest.mark.parametrize("nsrc", [1, 17, 70])
@pytest.mark.parametrize("sizes", sorted(SIZES))
def test_part_sizes(sizes, nsrc):
    rng = np.random.default_rng(nsrc)
    # many more parts of three vertices: few parts would go to the clusters
    graphs = [ring_with_chords(n, 7 + n) for n in SIZES[sizes] + [3] * 320]
    srcs = [rng.integers(0, g.n, nsrc).astype(np.int32) for g in graphs]
    u, off = gen.disjoint_union(graphs)
    with abi.Graph(u) as dg:
        dg.set_parts(off)
        for _ in range(2):  # the second call finds the first one's words
            blocks, st = dg.multi_bfs(srcs)
        assert st.batches == len(graphs) * -(-nsrc // 64)
    edges = 0
    for p, (g, s) in enumerate(zip(graphs, srcs)):
        ref, e, _ = O.mssp(g, s)
        assert np.array_equal(blocks[p], O.hops_ref_to_api(ref, s)), (p, g.n)
        edges += e
    assert st.edges_traversed == edges


@pytest.mark.parametrize("length", [31, 32, 33, 34, 70, 300])
def test_deep_levels(length):
    # levels around 32 leave the bit slices; two sources share a path, one of
    # them twice
    rows = [gen.grid(1, length), gen.grid(2, length)]
    srcs = [np.array([0, length - 1, 0], np.int32), np.array([length // 2, 2 * length - 1], np.int32)]
    u, off = gen.disjoint_union(rows)
    with abi.Graph(u, symmetric=True) as dg:
        dg.set_parts(off)
        blocks, _ = dg.multi_bfs(srcs)
    for g, s, b in zip(rows, srcs, blocks):
        assert np.array_equal(b, O.hops_ref_to_api(O.mssp(g, s)[0], s))


def test_set_parts_again():
    # other parts on the same handle, and a traced call in between
    a, b = ring_with_chords(500, 1), ring_with_chords(300, 2)
    u, off = gen.disjoint_union([a, b])
    whole = O.hops_ref_to_api(O.mssp(u, [3, 600])[0], [3, 600])
    with abi.Graph(u) as dg:
        dg.set_parts([0, u.n])
        one, _ = dg.multi_bfs([[3, 600]])
        dg.set_parts(off)
        dg.trace(True)
        traced, _ = dg.multi_bfs([[3], [100]])
        dg.trace(False)
        two, _ = dg.multi_bfs([[3], [100]])
    assert np.array_equal(one[0], whole)
    for got in (traced, two):
        assert np.array_equal(got[0][0], whole[0][:500]) and np.array_equal(got[1][0], whole[1][500:])
