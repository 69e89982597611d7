"""Lists of the ordered weighted traversal (csrc/nearfar.cu) that stay short for
hundreds of phases while long rows come and go, against the oracle.  Distances
are sums of whole numbers below 2^24, so the tolerance is zero."""

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi
from test_gpu_nearfar import weighted
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu


def hub_chain(hubs, leaves, spacing):
    """A path on which every spacing-th vertex has a row of `leaves` + 1 entries."""
    n = spacing * hubs
    k, h = np.arange(n - 1), np.repeat(spacing * np.arange(hubs), leaves)
    leaf = n + np.arange(leaves * hubs)
    return weighted(n + leaves * hubs, np.concatenate([k, h]), np.concatenate([k + 1, leaf]),
                    np.concatenate([1 + k % 3, 1 + leaf % 7]))


@pytest.mark.parametrize("leaves", [126, 127, 130])  # the longest row that one CTA walks alone, and longer
@pytest.mark.parametrize("spacing", [2, 5])
def test_long_rows_come_and_go(leaves, spacing):
    g = hub_chain(60, leaves, spacing)
    srcs = np.array([0, 1, 7, spacing * 30], np.int32)
    want = O.msssp(g, srcs)
    for weights in ("i32", "f32"):
        with abi.Graph(g, weights=weights) as dg:
            for _ in range(20):
                d, _ = dg.sssp(srcs[:1], variant=abi.VARIANT_DO)
                assert np.array_equal(to_ref(d), want[:1])
                d, _ = dg.sssp(srcs)
                assert np.array_equal(to_ref(d), want)


def test_threshold_below_its_own_rounding():
    # a distance of 1e11 behind an edge that the sample of the weights misses: the
    # threshold's step, some mean weights of 1, does not raise it at all, and pairs
    # beyond it are reached by the least distance that a scan leaves
    m = 200000
    w = np.ones(m, np.float32)
    free = np.setdiff1d(np.arange(m), np.arange(65536, dtype=np.int64) * m // 65536)
    w[free[0]] = 1e11
    w[free[5::700]] = 1e6
    k = np.arange(m)
    g = weighted(m + 1, k, k + 1, np.ones(m))
    g.w_f32 = w
    want = np.zeros(m + 1, np.float32)
    for i in range(m):
        want[i + 1] = want[i] + w[i]
    assert np.float32(1e11) + np.float32(512 * 16) > np.float32(1e11) == np.float32(1e11) + np.float32(512)
    with abi.Graph(g, weights="f32") as dg:
        d, _ = dg.sssp([0], variant=abi.VARIANT_DO)
        assert np.array_equal(d[0], want)
        d, _ = dg.sssp([0, 0, 0])
        assert (d == want).all()
