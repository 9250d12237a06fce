"""The 8-lane hierarchy walks against the oracle: vertex counts around the 16 a
CTA holds, one-triangle meshes, vertices with more candidates than the walk's
buffer (their pairs are then sorted by triangle too) and more overlapping nodes
than it takes side by side, and a step above the one-lane limit."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle import oracle as orc
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def heap(layers, n, side, gap, seed=0):
    rng = np.random.default_rng(seed)
    P, T = [], []
    for k in range(layers):
        p, t = scenes.grid_mesh(n, side, z=k * gap)
        p[:, :2] += 0.1 * side / (n - 1) * rng.standard_normal((len(p), 2))
        p[:, 2] += 0.2 * gap * rng.standard_normal(len(p))
        P.append(p)
        T.append(t + k * n * n)
    return np.concatenate(P), np.concatenate(T).astype(np.int32)


# layers, n, side, gap, tolerance: from one cell to over 100 candidates a vertex
CASES = [(1, 2, 0.1, 1e-3, 2e-3), (2, 2, 0.1, 1e-3, 2e-3), (1, 4, 0.1, 1e-3, 2e-3), (3, 7, 0.1, 8e-4, 1e-3),
         (12, 10, 0.1, 2e-4, 1e-3), (20, 9, 0.02, 1e-4, 2e-3), (2, 60, 1.0, 1.2e-3, 1.5e-3)]


@pytest.mark.parametrize("layers,n,side,gap,tol", CASES)
def test_candidates(layers, n, side, gap, tol):
    pos, tris = heap(layers, n, side, gap)
    exp = orc.self_candidates(pos, tris, tol)
    got = native.detect_candidates(pos, tris, tol, cap=len(exp) + 16)
    assert np.array_equal(got, exp)


def test_one_triangle():
    pos = np.array([[0.0, 0, 0], [0.1, 0, 0], [0, 0.1, 0], [0.02, 0.02, 1e-3], [1.0, 1.0, 1.0]])
    tris = np.array([[0, 1, 2]], dtype=np.int32)
    exp = orc.self_candidates(pos, tris, 2e-3)
    assert len(exp) == 4
    assert np.array_equal(native.detect_candidates(pos, tris, 2e-3), exp)


def test_step_above_the_one_lane_limit():
    pos, tris = heap(2, 190, 1.0, 8e-4, seed=1)  # 72,200 vertices
    s = scenes.Scene(friction=((0.4,),))
    s.add_mesh(pos, tris, area_density=0.1, bending=1e-2, stretching=1e3)
    p = abi.params(time_step=1e-3, iterations=1, self_collision=True, self_tol=1e-3)
    g, o = native.Simulation(s, p), Oracle(s, p)
    rg, ro = g.step(1), o.step(1)
    assert rg.n_self_contacts == ro.n_self_contacts > 0
    sg, so = g.self_contacts(), o.self_contacts()
    for k in ("vertex", "partner", "face"):
        assert np.array_equal(sg[k], so[k]), k
