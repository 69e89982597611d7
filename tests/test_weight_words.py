"""The threshold rule of the ordered weighted traversal (csrc/nearfar.cu),
restated on the CPU over weight words.  Distances wait in a far list while they
lie above a threshold T; T rises by a step when the near list is empty, and to
the least distance left plus a step when a scan moved nothing.  It ends for
every non-negative weight only if no word ever lies at or above the word of
"unreached": a float -0.0 (0x80000000) would, so handles hold 0.0 for it."""

import numpy as np
import pytest

INF = {"i32": 0x7FFFFFFF, "f32": 0x7F7FFFFF}


def word(x, kind):
    """csrc/runtime.cu, weight_word."""
    w = int(np.float32(x).view(np.uint32)) if kind == "f32" else int(np.uint32(x))
    return 0 if kind == "f32" and w == 0x80000000 else w


def add(a, b, kind):
    if kind == "i32":
        return (a + b) & 0xFFFFFFFF
    with np.errstate(over="ignore"):
        return int((np.uint32(a).view(np.float32) + np.uint32(b).view(np.float32)).view(np.uint32))


def distances(n, edges, source, kind, step, raw=False, queue_all=False, most=10000):
    """Words of the distances, None if the rule does not end.  queue_all: neighbours
    of the source are queued whatever their weight."""
    inf, w_of = INF[kind], (lambda x: int(np.float32(x).view(np.uint32))) if raw else (lambda x: word(x, kind))
    rows = [[] for _ in range(n)]
    for u, v, w in edges:
        rows[u].append((v, w_of(w)))
    D = [inf] * n
    last = {v: w for v, w in rows[source]}
    near, far = [], []
    T = min(add(0, step, kind), inf - 1)
    for v, w in last.items():
        d = 0 if v == source else w
        D[v] = d
        if d < inf or queue_all:
            (near if d <= T else far).append(v)
    D[source] = 0
    scanned = False
    for _ in range(most):
        if near:
            now, near = near, []
            for u in now:
                for v, w in rows[u]:
                    c = add(D[u], w, kind)
                    if c < D[v]:
                        D[v] = c
                        (near if c <= T else far).append(v)
            scanned = False
            continue
        if not far:
            return D
        old, T = T, min(add(min(D[v] for v in far if D[v] > T) if scanned else T, step, kind), inf - 1)
        if scanned and T <= old:
            return None
        near = [v for v in set(far) if old < D[v] <= T]
        far = [v for v in set(far) if D[v] > T]
        scanned = not near
    return None


def least(n, edges, source):
    """Bellman-Ford in float64.  The source's row gives each neighbour its last
    entry (src/algorithm/cpu/sssp.cpp:41-46) and is relaxed only through a self
    loop."""
    loop = any(u == v == source for u, v, _ in edges)
    D = np.full(n, np.inf)
    for u, v, w in edges:
        if u == source:
            D[v] = w
    D[source] = 0.0
    for _ in range(n):
        for u, v, w in edges:
            if u != source or loop:
                D[v] = min(D[v], D[u] + w)
    return D


# a zero-length bridge, leaf and cycle, and a vertex that another path reaches first
EDGES = [(0, 1, -0.0), (1, 2, 3.0), (2, 3, -0.0), (3, 2, -0.0), (0, 4, -0.0), (0, 5, 9.0), (1, 5, -0.0), (5, 6, 2.0)]


def test_zero_signs_do_not_reach_the_words():
    want = least(7, EDGES, 0)
    for step in (1e-6, 0.5, 3.0, 100.0):
        s = word(step, "f32")
        assert distances(7, EDGES, 0, "f32", s, raw=True, most=2000) != distances(7, EDGES, 0, "f32", s)
        got = np.array(distances(7, EDGES, 0, "f32", s), np.uint32).view(np.float32)
        assert np.array_equal(got, want.astype(np.float32)), step


@pytest.mark.parametrize("kind", ["i32", "f32"])
def test_rule_ends(kind):
    rng = np.random.default_rng(3)
    for trial in range(60):
        n = int(rng.integers(2, 30))
        top = int(rng.choice([1, 3, 60, 1 << 20]))
        edges = [(int(a), int(b), int(w)) for a, b, w in zip(rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n),
                                                             rng.integers(0, top, 3 * n))]
        got = distances(n, edges, 0, kind, word(int(rng.choice([1, 7, 4096])), kind))
        want = least(n, edges, 0)
        assert got is not None
        got = np.array(got, np.uint32)
        got = got.view(np.float32).astype(np.float64) if kind == "f32" else got.astype(np.float64)
        got[got >= (np.float64(np.finfo(np.float32).max) if kind == "f32" else INF["i32"])] = np.inf
        assert np.array_equal(got, want), trial


@pytest.mark.parametrize("kind", ["i32", "f32"])
def test_source_row_weight_of_unreached(kind):
    # the largest weight there is equals the encoding of "unreached"
    top = INF[kind] if kind == "i32" else float(np.finfo(np.float32).max)
    edges = [(0, 1, top), (1, 2, 1.0), (0, 3, 5.0), (3, 4, 2.0)]
    step = word(3, kind)
    assert distances(5, edges, 0, kind, step, queue_all=True) is None
    assert distances(5, edges, 0, kind, step) == [0, INF[kind], INF[kind], word(5, kind), word(7, kind)]
