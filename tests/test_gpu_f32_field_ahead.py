"""The FP32 field kernels of grids beyond L2 (at least B_AHEAD_NODES nodes),
which ask for the rows of later planes ahead of use: one step against the FP64
form's, on grids whose rows and planes end inside a block and whose planes are
larger than what is asked for.  One ion at each cell's centre and a wave in B
keep both forms far from cells without ions.  Bars: FP32 stencils on values
rounded to FP32 (2^-24), differences over one cell of a wave over 32 cells and
more (a factor of about 10 in aj and E), ten subcycles."""
import numpy as np
import pytest

from conftest import rel_l2
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu


def _make(cells):
    cfg = config(0, cells=cells, ppc=1, seed=2)
    h = Hybrid(cfg)
    h.load_maxwellian()
    N = int(h.ni_tot[0])
    h.xp[:N] = np.floor(h.xp[:N] - 1.0) + 1.5  # q(1) = 1, unit cells
    nx, ny, nz = h.b1.shape[:3]
    x, y, z = np.meshgrid(*(2 * np.pi * (np.arange(n) - 1.0) / (n - 2) for n in (nx, ny, nz)), indexing="ij")
    for n in ("b1", "b12", "b1p2", "bt"):
        b = getattr(h, n)
        b[..., 0] += 0.05 * np.sin(y + z)
        b[..., 1] += 0.05 * np.sin(z + x)
        b[..., 2] += 0.05 * np.sin(x + y)
    h.mark_host_dirty()
    return h


@pytest.mark.parametrize("cells", [(132, 124, 132), (612, 332, 12)])
def test_step_beyond_l2(cells):
    a, b = _make(cells), _make(cells)
    a.f32_begin()
    a.f32_run(1)
    a.f32_end()
    b.ion_step()
    a.sync_to_host()
    b.sync_to_host()
    for name, tol in (("b1", 1e-6), ("np", 1e-5), ("up", 1e-5), ("aj", 1e-4), ("E", 1e-4)):
        # (interior: the FP64 form leaves the ghosts of the corrector's aj as they were)
        x, y = (getattr(h, name)[1:-1, 1:-1, 1:-1] for h in (a, b))
        assert rel_l2(x, y) < tol, (name, rel_l2(x, y))
    a.close()
    b.close()
