"""Betweenness of an empty source list is zero everywhere, whatever an earlier
call left in the buffers."""

import numpy as np
import pytest

from dawn_gb300 import abi, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc", [3, 200])
def test_no_sources(nsrc):
    import torch
    g = gen.rmat(9, 8, seed=1)
    with abi.Graph(g) as dg:
        before, _ = dg.betweenness(gen.sources(g, nsrc, seed=2))
        assert before.any()
        bc, st = dg.betweenness([])
        assert not bc.any() and st.levels == 0 and st.batches == 0
        out = torch.full((g.n,), 5.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        rc = abi.lib().dawn_betweenness_device(dg.handle, None, 0, out.data_ptr(), None)
        dg.synchronize()
        assert rc == abi.OK and not out.any()
