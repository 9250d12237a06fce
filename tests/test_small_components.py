"""Scenes of very many small components: those of up to a leaf's 40 vertices share
a leaf, since a block of the sweeps costs the same whatever it holds.  Sizes around
the leaf, mixed with larger cloths, against the oracle."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def patches(sizes):
    s = scenes.Scene(friction=((0.3, 0.3), (0.3, 0.3)))
    m = int(np.ceil(np.sqrt(len(sizes))))
    P, T, at = [], [], 0
    for k, n in enumerate(sizes):
        p, t = scenes.grid_mesh(n, 0.02 * n, z=0.002, center=(0.2 * (k % m), 0.2 * (k // m)))
        P.append(p)
        T.append(t + at)
        at += n * n
    s.add_mesh(np.concatenate(P), np.concatenate(T).astype(np.int32), area_density=0.1, bending=1e-2, stretching=1e2,
               material=0)
    s.add_plane((0, 0, 0), (0, 0, 1), material=1)
    return s


# 4 vertices each; around the leaf (36 and 49); tiny ones between larger cloths
@pytest.mark.parametrize("sizes,blocks", [([2] * 3000, 300), ([6, 7] * 200, 400),
                                          (([2] * 30 + [20] + [3] * 20) * 12, 12 * 30)])
@pytest.mark.parametrize("precision", [abi.PDF_FP64, abi.PDF_FP32_REFINE])
def test_small_components(sizes, blocks, precision):
    s = patches(sizes)
    s.vel = np.zeros_like(s.pos)
    s.vel[:, 2] = -0.5
    kw = dict(time_step=5e-3, iterations=8)
    g, o = native.Simulation(s, abi.params(precision=precision, **kw)), Oracle(s, abi.params(**kw))
    # FP32 halves sets that overlap down to 40 vertices: leaves of more than 20
    assert g.stats().sweep_blocks <= (blocks if precision == abi.PDF_FP64 else 2 * blocks)
    for _ in range(2):
        assert g.step(1).n_contacts == o.step(1).n_contacts
    # the step's parity bounds: FP64, and FP32 with refinement; v against the speed of
    # the impact (patches on the floor come to rest: the oracle's v is 1e-18)
    rel = 1e-6 if precision == abi.PDF_FP64 else 1e-5
    for a, b, scale in zip(g.state(), o.state(), (np.abs(s.pos).max(), 0.5)):
        assert np.abs(a - b).max() < rel * scale
