"""The FP32 form's field step in one launch (small grids: a cluster of blocks,
then a cooperative grid) at the sizes where its forms change: the smallest
box, the last one of the cluster form and the first of the grid form, the last
of the grid form and the first that takes one launch per half kernel.

Each is held to the FP64 oracle by the bars of test_gpu_f32.py (B within 1e-5,
the moments within 1e-4), and two runs agree bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2
from helpers import make_hybrid, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(8, 8, 8), (16, 16, 16), (20, 16, 16), (76, 32, 32), (80, 32, 32)])
def test_step_against_the_oracle_and_itself(cells):
    h = make_hybrid(cells=cells, ppc=6, seed=9, db=0.03)
    o = oracle_for(h, nthreads=8)
    r = make_hybrid(cells=cells, ppc=6, seed=9, db=0.03)
    for x in (h, r):
        x.f32_begin()
        x.f32_run(2)
        x.f32_end()
        x.sync_to_host()
    for _ in range(2):
        o.ion_step()
    assert rel_l2(h.b1, o.b1) < 1e-5 and rel_l2(h.b12, o.b12) < 1e-5
    for n in ("np", "up", "E"):
        assert rel_l2(getattr(h, n), getattr(o, n)) < 1e-4, n
    for n in ("b1", "b12", "np", "up", "aj", "E", "xp", "vp"):
        assert np.array_equal(getattr(h, n), getattr(r, n)), n
    h.close()
    r.close()


def test_courant_violation_takes_the_replayed_count():
    """A thin node halves dtsub on the host (gutsf.f:1776-1822); the loop
    launched ahead of that look leaves the state alone."""
    h = make_hybrid(cells=(8, 8, 8), ppc=6, seed=2, db=0.0, dt=2.0, ntsub=4)
    o = oracle_for(h)
    h.f32_begin()
    h.f32_run(1)
    h.f32_end()
    h.sync_to_host()
    o.ion_step()
    assert rel_l2(h.b1, o.b1) < 1e-5
    assert rel_l2(h.np, o.np) < 1e-4
    h.close()
