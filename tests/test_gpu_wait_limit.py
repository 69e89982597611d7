"""Launches whose waits run out: with one poll a wait, a CTA of a grid of dozens
gives up before the last one has arrived.  Every call that synchronises reports
it, with statistics or without; an asynchronous one through the next call or the
synchronisation; and the handle gives the oracle's results again afterwards."""

import ctypes

import numpy as np
import pytest

import oracle as O
from dawn_gb300 import abi, gen
from test_gpu_sssp import to_ref

pytestmark = pytest.mark.gpu

DEFAULT = 1 << 27


def calls(dg, g, srcs):
    """Host-synchronising calls without statistics: name -> status."""
    L, n, k = abi.lib(), g.n, len(srcs)
    s, h = np.ascontiguousarray(srcs, np.int32), dg.handle
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    d, cc = np.empty((k, n), np.int32), np.empty(k)
    bc = np.empty(n)
    return {
        "bfs_one": lambda: L.dawn_bfs(h, p(s), 1, p(d), abi.VARIANT_DO, None),
        "bfs_list": lambda: L.dawn_bfs(h, p(s), 5, p(d), abi.VARIANT_DO, None),
        "bfs_batch": lambda: L.dawn_bfs(h, p(s), k, p(d), abi.VARIANT_AUTO, None),
        "sssp_one": lambda: L.dawn_sssp(h, p(s), 1, p(d), abi.VARIANT_DO, None),
        "sssp_batch": lambda: L.dawn_sssp(h, p(s), 9, p(d), abi.VARIANT_AUTO, None),
        "closeness": lambda: L.dawn_closeness(h, p(s), k, 0, p(cc), None, None, None),
        "closeness_weighted": lambda: L.dawn_closeness(h, p(s), 9, 1, p(cc), None, None, None),
        "betweenness": lambda: L.dawn_betweenness(h, p(s), k, p(bc), None),
    }


@pytest.mark.parametrize("graph", ["rmat", "grid"])
def test_reported_and_recovered(graph):
    g = gen.rmat(14, 8, seed=1, weights=True) if graph == "rmat" else gen.grid(90, 140, seed=1, weights=True)
    srcs = gen.sources(g, 300, seed=2)
    hops = O.hops_ref_to_api(O.mssp(g, srcs)[0], srcs)
    far = O.msssp(g, srcs[:9])
    with abi.Graph(g, weights="i32") as dg:
        # (float32 terms overflow on the grid's hundreds of levels, the oracle's do not)
        bc, _ = dg.betweenness(srcs)
        if graph == "rmat":
            want = O.bc(g, srcs)
            assert np.allclose(bc, want, rtol=1e-4, atol=1e-6 * np.abs(want).max())
        for name, call in calls(dg, g, srcs).items():
            dg.set_option(abi.OPT_WAIT_POLLS, 1)
            assert call() == abi.ERR_TIMEOUT, name
            assert "wait ran out" in abi.lib().dawn_last_error().decode()
            dg.set_option(abi.OPT_WAIT_POLLS, DEFAULT)
            assert call() == abi.OK, name
            dg.synchronize()
            d, _ = dg.bfs(srcs[:5], variant=abi.VARIANT_DO)
            assert np.array_equal(d, hops[:5]), name
            d, _ = dg.bfs(srcs)
            assert np.array_equal(d, hops), name
            d, _ = dg.sssp(srcs[:9])
            assert np.array_equal(to_ref(d), far), name
            got, _ = dg.betweenness(srcs)
            assert np.allclose(got, bc, rtol=1e-6, atol=0, equal_nan=True), name


@pytest.mark.parametrize("by", ["synchronize", "next_call"])
@pytest.mark.parametrize("nsrc", [1, 300])
def test_asynchronous_calls(nsrc, by):
    import torch
    g = gen.rmat(14, 8, seed=1)
    srcs = gen.sources(g, nsrc, seed=2)
    hops = O.hops_ref_to_api(O.mssp(g, srcs)[0], srcs)
    out = torch.empty((nsrc, g.n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with abi.Graph(g) as dg:
        dg.set_option(abi.OPT_WAIT_POLLS, 1)
        dg.bfs_device(srcs, out.data_ptr(), stats=False)
        if by == "next_call":
            torch.cuda.synchronize()
        dg.set_option(abi.OPT_WAIT_POLLS, DEFAULT)
        with pytest.raises(abi.DawnError) as e:
            dg.synchronize() if by == "synchronize" else dg.bfs_device(srcs, out.data_ptr(), stats=False)
        assert e.value.status == abi.ERR_TIMEOUT
        dg.bfs_device(srcs, out.data_ptr(), stats=False)
        dg.synchronize()
        assert np.array_equal(out.cpu().numpy(), hops)


def test_option_range():
    g = gen.rmat(8, 4, seed=3)
    with abi.Graph(g) as dg:
        assert dg.get_option(abi.OPT_WAIT_POLLS) == DEFAULT
        for bad in (0, -1, 1 << 31):
            with pytest.raises(abi.DawnError):
                dg.set_option(abi.OPT_WAIT_POLLS, bad)
