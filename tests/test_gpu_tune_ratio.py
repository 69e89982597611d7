"""The autotuner and the push ratio: until a ratio is set, batches of graphs of 16
entries a vertex and more push at another one than the option answers.  Tuning
with one source, where no ratio is tried, must leave that as it is, and tuning
with several must start from it.  Seen in the levels that push."""

import numpy as np
import pytest

from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu


def pushes(dg, srcs):
    d, st = dg.bfs(srcs, variant=abi.VARIANT_BITSET)
    return d, (st.push_levels, st.pull_levels)


@pytest.fixture(scope="module")
def case():
    """A dense graph on which the two ratios take different directions."""
    for seed in range(40):
        g = gen.rmat(13, 16, seed=seed)
        srcs = gen.sources(g, 3, seed=seed)
        with abi.Graph(g) as dg:
            _, unset = pushes(dg, srcs)
            dg.set_option(abi.OPT_PUSH_RATIO, 4)
            _, four = pushes(dg, srcs)
        if unset != four:
            assert g.m >= 16 * g.n
            return g, srcs, unset
    pytest.fail("no graph tells the ratios apart")


def test_one_source(case):
    g, srcs, unset = case
    with abi.Graph(g) as dg:
        for use_cache in (False, True):
            t = dg.autotune(srcs[:1], use_cache=use_cache)
            assert t["push_ratio"] == 4 == dg.get_option(abi.OPT_PUSH_RATIO)
            assert pushes(dg, srcs)[1] == unset


def test_batch_starts_from_the_default(case):
    g, srcs, unset = case
    with abi.Graph(g) as dg:
        want, _ = pushes(dg, srcs)
        t = dg.autotune(srcs)
        assert t["push_ratio"] == dg.get_option(abi.OPT_PUSH_RATIO)
        assert t["ms"] <= t["default_ms"] * 1.0001
        dg.set_option(abi.OPT_PUSH_RATIO, 2)  # the default of such a graph
        dg.set_option(abi.OPT_AUTO_LEARNED, 0)
        d, levels = pushes(dg, srcs)
        assert np.array_equal(d, want) and levels == unset
