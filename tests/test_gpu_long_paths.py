"""Paths longer than the levels that one CTA runs alone in one step (32,768): the
step ends, hands its list over and goes on.  Distances are known exactly."""

import numpy as np
import pytest

from dawn_gb300 import abi, gen
from test_gpu_nearfar import weighted

pytestmark = pytest.mark.gpu

N = 70001


def path(hub, weight):
    """0 - 1 - .. - N-1 both ways, with `hub` leaves at the far end."""
    k, leaf = np.arange(N - 1), N + np.arange(hub)
    src = np.concatenate([k, k + 1, np.full(hub, N - 1), leaf])
    dst = np.concatenate([k + 1, k, leaf, np.full(hub, N - 1)])
    return weighted(N + hub, src, dst, np.full(len(src), weight))


def steps(g, hub, s):
    d = np.abs(np.arange(g.n) - s)
    d[N:] = abs(N - 1 - s) + 1
    return d


@pytest.mark.parametrize("hub", [0, 200])  # with records and the bitmap in shared memory, and without
def test_hops(hub):
    g = path(hub, 1)
    with abi.Graph(g) as dg:
        for s in (0, 32768, N - 1):
            d, st = dg.bfs([s], variant=abi.VARIANT_DO)
            assert np.array_equal(d[0], steps(g, hub, s)), s
            assert st.levels == steps(g, hub, s).max() + 1
            assert st.edges_traversed == g.m


@pytest.mark.parametrize("weight", [0, 1, 3])
@pytest.mark.parametrize("weights", ["i32", "f32"])
def test_weighted(weights, weight):
    for hub in (0, 200):
        g = path(hub, weight)
        with abi.Graph(g, weights=weights) as dg:
            for srcs, variant in (([0], abi.VARIANT_DO), ([5, N - 1], abi.VARIANT_AUTO)):
                d, _ = dg.sssp(srcs, variant=variant)
                for i, s in enumerate(srcs):
                    assert np.array_equal(d[i].astype(np.int64), weight * steps(g, hub, s)), (hub, s)


@pytest.mark.parametrize("hub", [0, 200])
def test_others_wait_for_one_step_only(hub):
    # half a million levels by one CTA are a second or two; the other CTAs wait a
    # third of one at most, which one step's levels do not take (without a hub the
    # levels go by records, all in one step, on graphs of 1.6 million vertices at
    # most: a few seconds)
    n = 500001
    k, leaf = np.arange(n - 1), n + np.arange(hub)
    g = weighted(n + hub, np.concatenate([k, np.full(hub, n - 1)]), np.concatenate([k + 1, leaf]), np.full(n - 1 + hub, 0))
    want = np.concatenate([np.arange(n), np.full(hub, n)])
    with abi.Graph(g, weights="i32") as dg:
        dg.set_option(abi.OPT_WAIT_POLLS, 1 << (19 if hub else 23))
        d, _ = dg.bfs([0], variant=abi.VARIANT_DO)
        assert np.array_equal(d[0], want)
        dg.set_option(abi.OPT_WAIT_POLLS, 1 << 19)
        d, _ = dg.sssp([0], variant=abi.VARIANT_DO)
        assert not d.any()
