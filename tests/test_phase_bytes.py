"""The algorithmic bytes that pdf_time_phase reports are those of the kernels that
run: the inverse of small scenes, or the sweeps; detection without triangle boxes."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers", [(12, 1), (30, 1), (20, 3)])
def test_solve_bytes_of_small_scenes(n, layers):
    s = scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, layers=layers, spacing=0.02,
                               sphere_center=(0, 0, -0.5), sphere_radius=0.25)
    g = native.Simulation(s, abi.params(time_step=5e-3, iterations=4))
    g.step(1)
    v = n * n
    assert g.time_phase(0, 1)[1] == layers * (8 * v * v + 100 * v)
    g.set_sweep_schedule(32, 1, 1, 1)
    sweeps = g.time_phase(0, 1)[1]
    assert sweeps != layers * (8 * v * v + 100 * v) and sweeps > 16 * g.stats().factor_nnz_true


def test_detection_bytes():
    n = 40
    s = scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, sphere_center=(0, 0, -0.5), sphere_radius=0.25)
    g = native.Simulation(s, abi.params(time_step=5e-3, iterations=4, self_collision=True, self_tol=1e-3))
    g.step(1)
    v, t, obstacles = n * n, 2 * (n - 1) ** 2, 1
    assert g.time_phase(3, 1)[1] == obstacles * 25 * v + 24 * v + 12 * t + 2 * 112 * (t - 1)
