"""The FP32 form's conversion refuses an ion outside the box whatever the
spacing: also one whose distance in cells does not fit 32 bits, and whose low
word would name a cell inside."""
import numpy as np
import pytest

from swap_gb300 import abi
from swap_gb300.grid import grd7
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1e-6, 2.0**-20, 1.0])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_an_ion_far_outside_is_refused(d, axis):
    cfg = config(0, cells=(8, 8, 8), ppc=2, seed=4)
    h = Hybrid(cfg, coords=grd7(*cfg.nodes, d, d, d))
    h.load_maxwellian()
    keep = h.xp.copy(order="F")
    h.mark_host_dirty()
    h.f32_begin()  # as loaded it is inside
    q1 = (h.coords.qx, h.coords.qy, h.coords.qz)[axis][0]
    for cells in (8.5, 40000.5, 2.0**31 + 3.5, 2.0**32 + 5.5, 2.0**33 + 0.5, -0.5, 5.5 - 2.0**32):
        h.xp[3, axis] = q1 + cells * np.float64(np.float32(d))
        h.mark_host_dirty()
        with pytest.raises(abi.SwapError, match="EDOMAIN"):
            h.f32_begin()
        h.xp[...] = keep
        h.mark_host_dirty()
        h.f32_begin()
    h.close()
