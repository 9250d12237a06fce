"""Small FP64 scenes without memory for the inverse, or for any part of its
construction, are created all the same and solve by the sweeps."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# the inverse, its rows, then four buffers for each of four branches; 18: all there
@pytest.mark.parametrize("room", [0, 1, 2, 3, 6, 17, 18])
def test_memory_that_ends(room, monkeypatch):
    s = scenes.cloth_on_sphere(n=20, side=1.0, z=-0.2455, mu=0.3, layers=2, spacing=0.02, sphere_center=(0, 0, -0.5),
                               sphere_radius=0.25, pins=True)
    p = abi.params(time_step=5e-3, iterations=10)
    monkeypatch.setenv("PDF_DENSE_ROOM", str(room))
    g = native.Simulation(s, p)
    # the autotuner has timed the sweeps exactly where they are what solves
    assert (max(g.stats().sweep_cut_level_ms) > 0) == (room < 18)
    o = Oracle(s, p)
    for _ in range(2):
        assert g.step(1).n_contacts == o.step(1).n_contacts > 0
    for a, b in zip(g.state(), o.state()):  # the FP64 step's parity bound
        assert np.abs(a - b).max() < 1e-6 * np.abs(b).max()
