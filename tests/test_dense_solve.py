"""Small scenes solve by one product with the explicit inverse: sizes around a
warp's 32 columns and its unrolled loop (256), several components, pins, and both
sides of the 64 MiB limit (FP64: 2896 columns, FP32: 4096), against the oracle;
and the sweeps, pinned on the same handle, give the same trajectory."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

# relative bounds of the step's parity tests: FP64, and FP32 with refinement
REL = {abi.PDF_FP64: 1e-6, abi.PDF_FP32_REFINE: 1e-5}


def scene(n, layers):
    return scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, layers=layers, spacing=0.02,
                                  sphere_center=(0, 0, -0.5), sphere_radius=0.25, pins=n > 4)


@pytest.mark.parametrize("precision,n,layers", [
    (abi.PDF_FP64, 3, 1), (abi.PDF_FP64, 6, 1), (abi.PDF_FP64, 16, 1), (abi.PDF_FP64, 17, 3),
    (abi.PDF_FP32_REFINE, 4, 2), (abi.PDF_FP32_REFINE, 23, 1), (abi.PDF_FP32_REFINE, 30, 3),
    (abi.PDF_FP64, 53, 1), (abi.PDF_FP64, 54, 1), (abi.PDF_FP32_REFINE, 64, 1), (abi.PDF_FP32_REFINE, 65, 1)])
def test_step_matches_oracle(precision, n, layers):
    s = scene(n, layers)
    g = native.Simulation(s, abi.params(time_step=5e-3, iterations=10, precision=precision))
    o = Oracle(s, abi.params(time_step=5e-3, iterations=10))
    for _ in range(3):
        rg, ro = g.step(1), o.step(1)
        assert rg.n_contacts == ro.n_contacts
    for a, b in zip(g.state(), o.state()):
        assert np.abs(a - b).max() < REL[precision] * np.abs(b).max()
    g.set_sweep_schedule(32, 1, 1, 1)
    g.step(1)
    o.step(1)
    for a, b in zip(g.state(), o.state()):
        assert np.abs(a - b).max() < REL[precision] * np.abs(b).max()
