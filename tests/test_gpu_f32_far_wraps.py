"""Ions of the FP32 form that travel about once around a short axis in a step:
those that end next to their own cell and deposit within their brick's window
are no far movers (swap_f32_far_movers; at most 65536 of those fit a step), the
others are, as counted with numpy; the density is the oracle's either way."""
import numpy as np
import pytest

from conftest import rel_l2
from helpers import oracle_for
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu

HALF = np.array([0.0, 0.25, 0.75, 1.0, 2.25, 3.0, 3.25, 3.5, 3.75, 4.0, 4.25, 4.5, 5.75])  # cells in half a step


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_the_count_and_the_density(axis):
    cells = (8, 8, 8)
    cfg = config(0, cells=cells, ppc=2, seed=3, dt=0.5, ntsub=4, u=(0.0, 0.0, 0.0), vth=1e-6)
    h = Hybrid(cfg)
    h.load_maxwellian()
    n = int(h.ni_tot[0])
    rng = np.random.default_rng(axis)
    c0 = np.stack([rng.integers(0, 8, n) for _ in range(3)], 1)
    half = rng.choice(HALF, n) * rng.choice([-1.0, 1.0], n)
    h.xp[:n] = 1.0 + c0 + 0.5
    h.vp[:n] = 0.0
    h.vp[:n, axis] = half / 0.25
    h.vp1[...] = h.vp
    for b in (h.b0, h.b1, h.b12, h.b1p2, h.bt):  # no field: every ion goes straight
        b[...] = 0.0
    h.mark_host_dirty()
    o = oracle_for(h)
    x = c0[:, axis] + 0.5
    cell = (lambda v: np.floor(v)) if axis == 1 else (lambda v: np.ceil(v) - 1)
    mid, end = cell(x + half) % 8, cell(x + 2 * half) % 8
    step = (end - c0[:, axis] + 1) % 8 - 1  # nearest image, -1 .. 6
    window = (mid - c0[:, axis] // 4 * 4 + 1) % 8 - 1  # within the brick's window: -1 .. 4
    far = (step > 1) | (window > 4)
    h.f32_begin()
    h.f32_run(1)
    assert h.f32_far_movers() == far.sum()
    h.f32_end()
    h.sync_to_host()
    o.ion_step()
    assert int(h.ni_tot[0]) == n
    assert rel_l2(h.np, o.np) < 1e-6  # FP32 sums of a few tens of terms
    assert np.allclose(np.sort((h.xp[:n, axis] - 1.0) % 8), np.sort((x + 2 * half) % 8), atol=1e-6)
    h.close()
