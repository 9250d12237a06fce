"""Small scenes in FP32 are as exact as with the FP32 sweeps.

Scenes small enough for the explicit inverse (FP64 solves) keep the sweeps in
FP32: rounding the inverse's entries to FP32 puts v of such cloths two to four
times as far from the FP64 solve's.  The distance to an FP64 run of the scene is
compared with that of a handle on which the sweeps are pinned, over six bumpy
cloths; the two are equal but for the order of additions, for which the bound
leaves a factor of 1.5 in the geometric mean (single cloths scatter by as much).
"""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes

pytestmark = pytest.mark.gpu


def bumpy(n, layers, seed):
    s = scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, layers=layers, spacing=0.0015,
                               sphere_center=(0, 0, -0.5), sphere_radius=0.25)
    rng = np.random.default_rng(seed)
    s.pos = s.pos.copy()
    for _ in range(12):
        k = 2 * np.pi / rng.uniform(0.15, 0.75)
        a, ph = rng.uniform(0, 2 * np.pi, 2)
        s.pos[:, 2] += 1e-4 * np.sin(k * (s.pos[:, 0] * np.cos(a) + s.pos[:, 1] * np.sin(a)) + ph)
    return s


def distance(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,layers", [(25, 1), (43, 1), (33, 2)])
def test_as_exact_as_the_sweeps(n, layers):
    ratios = []
    for seed in range(6):
        kw = dict(time_step=2.5e-3, iterations=20)
        v = []
        for precision, pin in ((abi.PDF_FP64, False), (abi.PDF_FP32_REFINE, False), (abi.PDF_FP32_REFINE, True)):
            g = native.Simulation(bumpy(n, layers, seed), abi.params(precision=precision, **kw))
            if pin:
                g.set_sweep_schedule(32, 1, 1, 1)
            assert g.step(2).n_contacts > 0
            v.append(g.state()[1])
            g.close()
        ratios.append(distance(v[1], v[0]) / distance(v[2], v[0]))
    assert np.exp(np.mean(np.log(ratios))) < 1.5
