"""FP32 sweeps keep layers that overlap in one dissection; layers that lie apart,
and every FP64 scene, are dissected component by component.  Two 62 x 62 layers:
too large for the explicit inverse."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing,together", [(0.02, True), (0.2, False)])
def test_layers_of_fp32_scenes(spacing, together):
    s = scenes.cloth_on_sphere(n=62, side=1.0, z=-0.2455, mu=0.3, layers=2, spacing=spacing,
                               sphere_center=(0, 0, -0.5), sphere_radius=0.25, pins=True)
    kw = dict(time_step=5e-3, iterations=10)
    g = native.Simulation(s, abi.params(precision=abi.PDF_FP32_REFINE, **kw))
    d = native.Simulation(s, abi.params(precision=abi.PDF_FP64, **kw))
    assert (g.stats().factor_nnz > d.stats().factor_nnz) == together
    o = Oracle(s, abi.params(**kw))
    for _ in range(2):
        assert g.step(1).n_contacts == o.step(1).n_contacts > 0
    for a, b in zip(g.state(), o.state()):  # the FP32 solves' bound
        assert np.abs(a - b).max() < 1e-5 * np.abs(b).max()
