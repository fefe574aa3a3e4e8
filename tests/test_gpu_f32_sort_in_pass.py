"""The FP32 form's sorted moves made by the next step's pass 1 (grids above the
one-launch field step, inside a run of several steps): a run of n steps equals
n runs of one step, which move the ions at their end, bit for bit -- without
sources, with inflow, outflow and cloud ions staged into the order, and with
ions that travel several cells a step."""
import numpy as np
import pytest

from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu
CELLS = (64, 60, 40)  # 153600 cells, above FIELD_LOOP_NODES


def _make(kind):
    n = {"plain": 0, "sources": 2, "far": 0}[kind]
    cfg = config(n, cells=CELLS, ppc=4, seed=12)
    if kind == "sources":
        cfg.sources.update(cx_a=0.0, nu_ion=0.02)  # no charge exchange; several cloud ions a step
    h = Hybrid(cfg, ni_max=cfg.ni_max_hint(8) + 50000)
    h.load_maxwellian()
    N = int(h.ni_tot[0])
    if kind == "far":  # one ion in 401 moves 2.6 cells a step
        h.vp[5:N:401, 0] = 52.0
        h.vp1[5:N:401, 0] = 52.0
    if cfg.sources:
        h.set_sources(cfg.make_sources())
    h.mark_host_dirty()
    h.f32_begin()
    return h


@pytest.mark.parametrize("kind", ["plain", "sources", "far"])
def test_run_of_steps_equals_single_steps(kind):
    a, b = _make(kind), _make(kind)
    a.f32_run(4)
    for _ in range(4):
        b.f32_run(1)
    assert a.f32_count() == b.f32_count()
    if kind == "far":
        assert a.f32_far_movers() == b.f32_far_movers() > 0
    assert np.array_equal(a.f32_key_starts(), b.f32_key_starts())
    for h in (a, b):
        h.f32_end()
        h.sync_to_host()
    N = int(a.ni_tot[0])
    assert N == int(b.ni_tot[0])
    if kind == "sources":
        assert N != a.cfg.n_particles
    for n in ("xp", "vp", "vp1", "mrat", "beta_p"):
        assert np.array_equal(getattr(a, n)[:N], getattr(b, n)[:N]), n
    for n in ("b1", "b12", "np", "up", "E", "aj"):
        assert np.array_equal(getattr(a, n), getattr(b, n)), n
    a.close()
    b.close()
