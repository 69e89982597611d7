"""How neighbourhoods grow (csrc/runtime.cu, read_growth), restated on the CPU:
the mean factor per level until a vertex's neighbourhood holds 8,192 vertices or
half of the graph, within 16 levels, the largest of four samples.  Random graphs
of low degree lie at 2 and above, meshes below, whatever the degree."""

import numpy as np
import pytest

from dawn_gb300 import gen


def growth(g):
    reach = max(64, min(8192, g.n // 2))
    deg, most = np.diff(g.row_ptr), 1.0
    for b in range(4):
        v0 = g.n * (2 * b + 1) // 8
        some = np.flatnonzero(deg[v0:v0 + 1024] > 0)
        if not len(some):
            continue
        seen = np.zeros(g.n, bool)
        level = np.array([v0 + some[0]])
        seen[level] = True
        count, steps = 1, 0
        while count < reach and len(level) and steps < 16:
            nxt = np.concatenate([g.col[g.row_ptr[v]:g.row_ptr[v + 1]] for v in level])
            level = np.unique(nxt[~seen[nxt]])
            seen[level] = True
            count, steps = count + len(level), steps + 1
        if steps and count >= reach:
            most = max(most, count ** (1 / steps))
    return most


def lattice3(k):
    i = np.arange(k ** 3).reshape(k, k, k)
    u = np.concatenate([i[:-1].ravel(), i[:, :-1].ravel(), i[:, :, :-1].ravel()])
    v = np.concatenate([i[1:].ravel(), i[:, 1:].ravel(), i[:, :, 1:].ravel()])
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=k ** 3))]).astype(np.int32)
    return gen.CsrGraph(k ** 3, rp, dst[order].astype(np.int32), symmetric=True)


@pytest.mark.parametrize("degree,lo,hi", [(2.5, 2.0, 3.2), (4, 3.5, 4.8), (7, 4.8, 8.5), (10, 4.8, 12)])
@pytest.mark.parametrize("n", [6000, 20000, 100000])
def test_random_graphs_grow(n, degree, lo, hi):
    for seed in range(3):
        assert lo <= growth(gen.erdos_renyi(n, int(n * degree), seed=seed)) < hi


def test_meshes_do_not():
    for g in (gen.grid(80, 90), gen.grid(300, 300), gen.knn(6000, 8, seed=1), gen.knn(60000, 8, seed=2),
              gen.knn(30000, 3, seed=3), lattice3(19), lattice3(40)):
        assert growth(g) < 2.0, (g.n, g.m)
