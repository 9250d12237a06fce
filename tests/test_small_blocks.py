"""A cloth small enough to be one subtree block: its root supernode (180-odd
columns) is wider than a span of the block's forward sweep, so the spans of a
tile add into y, which must not hold the solve before."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("precision", [abi.PDF_FP64, abi.PDF_FP32_REFINE])
def test_whole_cloth_in_one_block(precision, mode):
    s = scenes.cloth_on_sphere(n=24, side=1.0, z=-0.2455, mu=0.3, sphere_center=(0, 0, -0.5), sphere_radius=0.25,
                               pins=True)
    kw = dict(time_step=5e-3, iterations=20)
    g = native.Simulation(s, abi.params(precision=precision, **kw))
    g.set_sweep_schedule(64, 7, mode, 1)
    assert g.stats().sweep_blocks == 1
    o = Oracle(s, abi.params(**kw))
    for _ in range(2):
        rg, ro = g.step(1), o.step(1)
        assert rg.n_contacts == ro.n_contacts > 0
    for a, b in zip(g.state(), o.state()):  # the schedules' bound
        assert np.abs(a - b).max() < 1e-6 * np.abs(b).max()
