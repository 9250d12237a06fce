"""What FP32 results depend on besides the scene: the factor's dissection and the
grouping of the sums.  Neither may follow a rule made for speed, or a timing, so
that a scene's results stay those of the schedules that were there before.

The last test is the accuracy itself, with self contacts: the distance of v to an
FP64 run, against that of a handle on which a schedule is pinned.  The two differ
by the order of additions alone; single scenes scatter by as much as half, so the
geometric mean over six of them is held to 1.5.
"""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes

pytestmark = pytest.mark.gpu


def bumpy(n, layers, seed, spacing=0.0015):
    s = scenes.cloth_on_sphere(n=n, side=1.0, z=-0.2455, mu=0.4, layers=layers, spacing=spacing,
                               sphere_center=(0, 0, -0.5), sphere_radius=0.25)
    rng = np.random.default_rng(seed)
    s.pos = s.pos.copy()
    for i in range(layers):
        p = s.pos[i * n * n:(i + 1) * n * n]
        for _ in range(12):
            k = 2 * np.pi / rng.uniform(0.1, 0.5)
            a, ph = rng.uniform(0, 2 * np.pi, 2)
            p[:, 2] += 1.5e-4 * np.sin(k * (p[:, 0] * np.cos(a) + p[:, 1] * np.sin(a)) + ph)
    return s


def fp32(s, **kw):
    return native.Simulation(s, abi.params(precision=abi.PDF_FP32_REFINE, **kw))


# below, between and above the sizes at which FP64 scenes merge 4, 3 and 2 levels
@pytest.mark.parametrize("n", [24, 62, 141, 142, 448])
def test_three_merged_levels_at_every_size(n, monkeypatch):
    g = fp32(bumpy(n, 1, 0), time_step=2.5e-3)
    monkeypatch.setenv("PDF_ND_MERGE", "3")
    h = fp32(bumpy(n, 1, 0), time_step=2.5e-3)
    assert g.stats().factor_nnz == h.stats().factor_nnz
    assert g.stats().n_supernodes == h.stats().n_supernodes


@pytest.mark.parametrize("n,layers", [(24, 1), (90, 2), (256, 2), (500, 1)])
def test_items_of_32_columns(n, layers):
    g = fp32(bumpy(n, layers, 0), time_step=2.5e-3)
    st = g.stats()
    assert st.sweep_chunk == 32 and list(st.sweep_chunk_ms)[1:] == [0.0, 0.0]
    g.set_sweep_schedule(64, 1, 1, 1)  # a caller may still ask for others
    assert g.stats().sweep_chunk == 64


@pytest.mark.parametrize("n,layers", [(40, 3), (64, 2)])
def test_self_contacts_as_exact_as_pinned(n, layers):
    kw = dict(time_step=2.5e-3, iterations=20, self_collision=True, self_tol=1e-3)
    ratios = []
    for seed in range(6):
        s = bumpy(n, layers, seed)
        v = []
        for sim, pin in ((native.Simulation(s, abi.params(**kw)), False), (fp32(s, **kw), False), (fp32(s, **kw), True)):
            if pin:
                sim.set_sweep_schedule(32, 1, 1, 1)
            rep = sim.step(1)
            assert rep.n_self_contacts > 100
            v.append((rep.n_contacts, rep.n_self_contacts, sim.state()[1]))
            sim.close()
        assert v[0][:2] == v[1][:2] == v[2][:2]
        d = [np.linalg.norm(x[2] - v[0][2]) for x in v[1:]]
        ratios.append(d[0] / d[1])
    assert np.exp(np.mean(np.log(ratios))) < 1.5
