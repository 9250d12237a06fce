"""The parallel pairing of self contacts against the serial oracle, where its
waits can go wrong: long chains of dependent vertices, vertices numbered at
random (a wait may point anywhere), several hits and more neighbours than a
thread lists at a time, and vertex counts around the 32 a warp claims."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle import oracle as orc
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def shuffled(pos, tris, seed):
    order = np.random.default_rng(seed).permutation(len(pos))
    place = np.argsort(order)
    return pos[order], place[tris].astype(np.int32)


def layers(n, count, gap, seed, shuffle, noise=0.15):
    rough = 0.2 if count <= 128 else 0.02  # a tall stack stays in contact throughout
    rng = np.random.default_rng(seed)
    h = 1.0 / (n - 1)
    P, T = [], []
    for k in range(count):
        p, t = scenes.grid_mesh(n, 1.0, z=k * gap)
        p[:, :2] += noise * h * rng.standard_normal((len(p), 2))
        p[:, 2] += rough * gap * rng.standard_normal(len(p))
        P.append(p)
        T.append(t + k * n * n)
    pos, tris = np.concatenate(P), np.concatenate(T).astype(np.int32)
    return shuffled(pos, tris, seed) if shuffle else (pos, tris)


def fan(spokes, rings, gap, shuffle):
    """Two facing discs whose centre vertex has `spokes` neighbours (more than
    48: the list of vertices to wait for is filled several times)."""
    P, T = [], []
    for k in range(2):
        a = 2 * np.pi * (np.arange(spokes) + 0.3 * k) / spokes
        p = [[0.01 * k, 0.004 * k, k * gap]]
        for r in range(1, rings + 1):
            p += [[0.1 * r * np.cos(x), 0.1 * r * np.sin(x), k * gap] for x in a]
        at = lambda r, s: 1 + (r - 1) * spokes + s % spokes  # noqa: E731
        t = [[0, at(1, s), at(1, s + 1)] for s in range(spokes)]
        for r in range(1, rings):
            for s in range(spokes):
                t += [[at(r, s), at(r + 1, s), at(r + 1, s + 1)], [at(r, s), at(r + 1, s + 1), at(r, s + 1)]]
        T.append(np.array(t) + k * len(p))
        P.append(np.array(p))
    pos, tris = np.concatenate(P), np.concatenate(T).astype(np.int32)
    return shuffled(pos, tris, 3) if shuffle else (pos, tris)


CASES = [("layers", 4, 2, 8e-4, False), ("layers", 5, 2, 8e-4, True), ("layers", 33, 2, 8e-4, False),
         ("layers", 33, 3, 6e-4, True), ("layers", 90, 2, 7e-4, False), ("layers", 64, 3, 5e-4, True),
         ("fan", 70, 2, 8e-4, False), ("fan", 120, 3, 8e-4, True)]


@pytest.mark.parametrize("kind,n,count,gap,shuffle", CASES)
def test_pairing_is_the_serial_one(kind, n, count, gap, shuffle):
    pos, tris = layers(n, count, gap, 7, shuffle) if kind == "layers" else fan(n, count, gap, shuffle)
    tol = 1e-3
    o = orc.self_collisions(pos, tris, tol)
    assert len(o["vertex"]) > 0
    g = native.detect_self_collisions(pos, tris, tol)
    for k in ("vertex", "partner", "face", "normal"):
        assert np.array_equal(g[k], o[k]), k


# the last two: more self contacts than the self-friction kernel has threads,
# and more levels (one a layer) than the level kernel's table holds
@pytest.mark.parametrize("kind,n,count,gap,shuffle", [CASES[1], CASES[3], CASES[4], CASES[5], ("layers", 4, 160, 8e-4, False)])
def test_step_pairs_as_the_oracle(kind, n, count, gap, shuffle):
    """The step's path: hits in slots, two meshes sharing the scratch, registers
    emptied between steps."""
    s = scenes.Scene(friction=((0.4,),))
    for k in range(2):
        pos, tris = layers(n, count, gap, 7 + k, shuffle)
        s.add_mesh(pos + [3.0 * k, 0.0, 0.0], tris, area_density=0.1, bending=1e-2, stretching=1e3)
    s.add_plane((0, 0, -0.0145), (0, 0, 1))
    p = abi.params(time_step=1e-3, iterations=3, self_collision=True, self_tol=1e-3)
    g, o = native.Simulation(s, p), Oracle(s, p)
    for _ in range(2):
        q, v = o.state()
        g.set_state(q, v)
        rg, ro = g.step(1), o.step(1)
        assert rg.n_self_contacts == ro.n_self_contacts > 0
        sg, so = g.self_contacts(), o.self_contacts()
        for k in ("vertex", "partner", "face", "normal"):
            assert np.array_equal(sg[k], so[k]), k
        lg, og = g.self_levels()
        lo, oo = o.self_levels()
        assert np.array_equal(lg, lo)
        for a, b in zip(lg[:-1], lg[1:]):  # the order inside a level is free
            assert set(og[a:b]) == set(oo[a:b])
        # the bound of the step's parity tests
        qg, qo = g.state()[0], o.state()[0]
        assert np.abs(qg - qo).max() < 1e-6 * np.abs(qo).max()
    if count > 128:
        assert rg.n_levels > 128
