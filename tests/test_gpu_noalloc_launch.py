"""swap_update_up_noalloc with more ions than one launch takes: an error (the
deposit does not run), not moments of nothing; the next call is not affected."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_hybrid
from swap_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2**38, 2**62])  # 2^31 blocks, the first count that no launch takes, and more
def test_a_deposit_that_cannot_be_launched_is_reported(n):
    import torch

    h = make_hybrid(cells=(8, 6, 5), ppc=3)
    N = int(h.ni_tot[0])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda()  # noqa: E731
    xp, vp, bp, dens = dev(h.xp), dev(h.vp), dev(h.beta_p), torch.ones(h.np.size, dtype=torch.float64, device="cuda")
    up = torch.full((h.up.size,), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def call(dims, n):
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        return h.lib.swap_update_up_noalloc(C.byref(dims), C.byref(h.params), C.byref(h._coords_c), p(xp), p(vp),
                                            p(bp), n, p(dens), p(up), None)

    nodes = h.cfg.nodes
    assert call(abi.Dims(*nodes, 8, n), n) == 2  # SWAP_ECUDA
    assert call(abi.Dims(*nodes, 8, h.ni_max), N) == 0
    assert torch.isfinite(up).all() and not (up == 7.0).any()
    h.close()
