"""pdf_set_sweep_schedule on a small scene: the inverse's memory is given back, the
sweeps solve; a schedule that is refused leaves the inverse in use."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def cloth(n):
    return scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, sphere_center=(0, 0, -0.5), sphere_radius=0.25,
                                  pins=True)


def check(g, s, p):
    o = Oracle(s, p)
    for _ in range(2):
        assert g.step(1).n_contacts == o.step(1).n_contacts > 0
    for a, b in zip(g.state(), o.state()):  # the FP64 step's parity bound
        assert np.abs(a - b).max() < 1e-6 * np.abs(b).max()


def test_pinned_schedule_gives_the_inverse_back():
    import torch
    s, p = cloth(53), abi.params(time_step=5e-3, iterations=6)
    g = native.Simulation(s, p)
    before = torch.cuda.mem_get_info()[0]
    g.set_sweep_schedule(32, 1, 1, 1)
    assert torch.cuda.mem_get_info()[0] - before > 0.9 * 8 * 53 ** 4
    g.set_sweep_schedule(64, 2, 1, 1)  # and again, without one
    check(g, s, p)


def test_refused_schedule_keeps_the_inverse():
    s, p = cloth(38), abi.params(time_step=5e-3, iterations=6)
    g = native.Simulation(s, p)
    solve_bytes = g.time_phase(0, 1)[1]
    # the whole cloth as one block, four of its CTAs on an SM
    assert native.lib().pdf_set_sweep_schedule(g.h, 32, 7, 1, 3) == abi.PDF_INVALID_ARG
    assert g.time_phase(0, 1)[1] == solve_bytes
    check(native.Simulation(s, p), s, p)
    g.set_state(s.pos, np.zeros_like(s.pos) if s.vel is None else s.vel)
    check(g, s, p)
