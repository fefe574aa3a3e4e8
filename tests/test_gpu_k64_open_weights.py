"""The cells and weights that an FP64 step leaves behind on an open x axis, for
the entries that read them next (update_np and the like): after the first half
of the step those of every ion that stayed; after a whole step those too, as
long as no ion left in its second half move (they are stale then)."""
import numpy as np
import pytest

from conftest import relerr
from swap_gb300 import abi
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu


def _still_box(leaver):
    """A plasma at rest in an open box without inflow, one ion `leaver` before the far face at v = 1."""
    cfg = config(0, cells=(12, 4, 4), ppc=12, seed=6, dt=0.05, ntsub=4, u=(0.0, 0.0, 0.0), vth=1e-6)
    h = Hybrid(cfg)
    h.load_maxwellian()
    n = int(h.ni_tot[0])
    x1, xn = h.coords.qx[0], h.coords.qx[-2]
    h.xp[:n, 0] = np.clip(h.xp[:n, 0], x1 + 0.01, xn - 0.2)
    for l in (5, 700, 1501) if leaver is not None else ():
        h.xp[l, 0] = xn - leaver
        h.vp[l] = h.vp1[l] = (1.0, 0.0, 0.0)
    h.set_sources(abi.make_sources(seed=3, x_open=1, inflow_ppc=0))
    h.mark_host_dirty()
    return h, n


def _update_np_again(h):
    h.sync_to_host()
    want = h.np.copy()
    h.update_np(h.np)
    h.sync_to_host(h.np)
    return relerr(h.np, want)


# the bar: a node's density is a sum of some hundred terms, each rounded to 1.1e-16 of it at most, in another order
@pytest.mark.parametrize("leaver,left", [(0.01, 3), (0.04, 0), (None, 0)])
def test_first_half_keeps_the_weights(leaver, left):
    h, n = _still_box(leaver)
    h._check(h.lib.swap_ion_step_pre(h.ctx))
    assert int(h.ni_tot[0]) == n - left
    assert _update_np_again(h) < 1e-13
    h.update_up(h.vp, h.np, h.up)
    h.close()


@pytest.mark.parametrize("leaver,left", [(0.01, 3), (0.1, 0), (None, 0)])
def test_whole_step_keeps_the_weights_unless_an_ion_left_late(leaver, left):
    h, n = _still_box(leaver)
    h.ion_step()
    assert int(h.ni_tot[0]) == n - left
    assert _update_np_again(h) < 1e-13
    h.close()


def test_an_ion_that_left_late_makes_them_stale():
    h, n = _still_box(0.04)
    h.ion_step()
    assert int(h.ni_tot[0]) == n - 3
    with pytest.raises(abi.SwapError, match="get_interp_weights"):
        h.update_np(h.np)
    h.get_interp_weights(h.xp)
    h.update_np(h.np)
    h.close()
