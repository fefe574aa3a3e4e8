"""The FP64 cell search (get_interp_weights, gutsp.f:1396-1404) at positions
where its index arithmetic can go wrong, against numpy's comparisons."""
import numpy as np
import pytest

from swap_gb300 import abi
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu

FAR = (np.inf, -np.inf, 1e300, -1e300, 3.5e38, 1e12, 4294967301.0, 2147483649.0, 2147483647.5, -2147483649.5, np.nan)


def _make(cells=(7, 5, 6), ppc=4, coords=None):
    cfg = config(0, cells=cells, ppc=ppc, seed=2)
    h = Hybrid(cfg, coords=coords)
    h.load_maxwellian()
    h.mark_host_dirty()
    return h


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_positions_far_outside_are_reported(axis):
    h = _make()
    keep = h.xp.copy(order="F")
    for bad in FAR:
        h.xp[11, axis] = bad
        h.mark_host_dirty(h.xp)
        with pytest.raises(abi.SwapError, match="EDOMAIN"):
            h.get_interp_weights(h.xp)
        h.xp[...] = keep
        h.mark_host_dirty(h.xp)
        h.get_interp_weights(h.xp)
    h.close()
