"""The places that the sort of a run of several steps leaves to the next pass 1
(4 bytes an ion): reserved by the first such run, not by swap_f32_begin, so a
caller that takes single steps needs no more memory than their moves do."""
import numpy as np
import pytest

from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu


def test_single_steps_need_no_places():
    import torch

    room = 1 << 26  # 256 MB of places, far above what an allocation is rounded to
    cfg = config(0, cells=(64, 60, 40), ppc=1, seed=3)  # 153600 cells, above FIELD_LOOP_NODES
    h = Hybrid(cfg, ni_max=room, work_arrays=False)
    h.load_maxwellian()
    h.mark_host_dirty()
    h.f32_begin()
    h.f32_run(1)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    before = free()
    h.f32_run(1)
    assert free() == before
    h.f32_run(2)
    assert before - free() >= 4 * room
    # the blocks are taken over by the next state, whichever runs come first
    h.f32_end()
    after = free()
    h.f32_begin()
    h.f32_run(1)
    h.f32_run(3)
    assert abs(free() - after) < 4 * room // 8
    h.f32_end()
    h.sync_to_host()
    assert np.isfinite(h.b1).all() and int(h.ni_tot[0]) == cfg.n_particles
    h.close()
