"""The oracle's grid (initial.f:147-301) against the package's for every axis
length around its stretch loops' bounds: the same bits, no NaN."""
import numpy as np
import pytest

import pyoracle
from swap_gb300.grid import Coords, grd7


@pytest.mark.parametrize("n", [3, 4, 20, 21, 22, 40, 41, 42, 43, 44, 66])
def test_the_oracles_grid_is_the_packages(n):
    o = pyoracle.Oracle(n, 5, n + 1, 4, 0.05, 4, 1.0, 1.0, dx=0.7, dy=1.3, delz=0.9)
    got, want = o.coords(), grd7(n, 5, n + 1, 0.7, 1.3, 0.9)
    for name in Coords.ARRAYS:
        assert np.array_equal(got[name], getattr(want, name)), name
    o.close()
