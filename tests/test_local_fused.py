"""The one-launch local step of small scenes (8 lanes a vertex): vertices with
more neighbours than lanes, borders, several meshes, pins, contacts, damping, and
vertex counts around the 16 of a CTA, against the oracle; and a scene above the
kernel's limit, which keeps the two launches."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

# the bounds of the step's parity tests: FP64, and FP32 with refinement
REL = {abi.PDF_FP64: 1e-6, abi.PDF_FP32_REFINE: 1e-5}


def wheel(spokes, rings, seed):
    """A disc: the centre has `spokes` neighbours; slightly bumpy, so that its
    bending rows have non-zero rest curvature."""
    rng = np.random.default_rng(seed)
    a = 2 * np.pi * np.arange(spokes) / spokes
    p = [[0.0, 0.0, 0.0]]
    for r in range(1, rings + 1):
        p += [[0.1 * r * np.cos(x), 0.1 * r * np.sin(x), 0.0] for x in a]
    at = lambda r, s: 1 + (r - 1) * spokes + s % spokes  # noqa: E731
    t = [[0, at(1, s), at(1, s + 1)] for s in range(spokes)]
    for r in range(1, rings):
        for s in range(spokes):
            t += [[at(r, s), at(r + 1, s), at(r + 1, s + 1)], [at(r, s), at(r + 1, s + 1), at(r, s + 1)]]
    p = np.array(p)
    p[:, 2] += 0.004 * rng.standard_normal(len(p))
    return p, np.array(t, dtype=np.int32)


def compare(s, precision, steps=2, **kw):
    g = native.Simulation(s, abi.params(precision=precision, **kw))
    o = Oracle(s, abi.params(**kw))
    for _ in range(steps):
        rg, ro = g.step(1), o.step(1)
        assert rg.n_contacts == ro.n_contacts
    for a, b in zip(g.state(), o.state()):
        assert np.abs(a - b).max() < REL[precision] * np.abs(b).max()
    return rg


# (no FP32 case of the widest wheel: its motion amplifies FP32 rounding to the bound)
@pytest.mark.parametrize("spokes,rings,precision", [
    (s, r, p) for s, r in [(3, 5), (7, 2), (8, 2), (9, 3), (40, 3)] for p in REL
    if s < 40 or p == abi.PDF_FP64])
def test_valences_around_the_lanes(spokes, rings, precision):
    s = scenes.Scene(friction=((0.3, 0.4), (0.4, 0.3)))
    for k in range(2):
        p, t = wheel(spokes, rings, k)
        p[:, 0] += 2.0 * k
        s.add_mesh(p, t, area_density=0.1, bending=1e-2, stretching=1e2, material=k)
    s.add_pin(1, 1e3)
    s.add_plane((0, 0, -0.02), (0, 0, 1))
    rep = compare(s, precision, time_step=4e-3, iterations=8, air_damping=0.3)
    assert rep.n_contacts > 0


@pytest.mark.parametrize("precision", [abi.PDF_FP64, abi.PDF_FP32_REFINE])
@pytest.mark.parametrize("n", [2, 4, 5, 110, 128, 129])
def test_sizes_up_to_and_above_the_limit(n, precision):
    s = scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.3, sphere_center=(0, 0, -0.5), sphere_radius=0.25,
                               pins=n > 4)
    compare(s, precision, time_step=5e-3, iterations=4)
