"""The self-friction kernel's cluster (csrc/step_kernels.cu): as many CTAs as the
device can host together, down to one, which always runs; its launch is checked.
Every size gives the oracle's step, with more contacts than a small cluster has
threads."""
import os
import re

import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_cluster_launch_goes_unchecked():
    src = open(os.path.join(ROOT, "climatenet_b200", "csrc", "step_kernels.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    calls = re.findall(r"([^;{}]*)cudaLaunchKernelEx\(", src)
    assert calls and all(re.search(r"(return|=|CK\()\s*$", c) for c in calls)
    assert "cudaOccupancyMaxActiveClusters" in src


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PDF_FP64, abi.PDF_FP32_REFINE])
@pytest.mark.parametrize("ctas", [1, 2, 4, 8, 16])
def test_every_cluster_size(ctas, precision, monkeypatch):
    monkeypatch.setenv("PDF_SELF_CTAS", str(ctas))
    n, h = 33, 1.0 / 32
    rng = np.random.default_rng(5)
    s = scenes.Scene(friction=((0.4,),))
    P, T = [], []
    for k in range(3):
        p, t = scenes.grid_mesh(n, 1.0, z=6e-4 * k)
        p[:, :2] += 0.15 * h * rng.standard_normal((len(p), 2))
        p[:, 2] += 1.2e-4 * rng.standard_normal(len(p))
        P.append(p)
        T.append(t + k * n * n)
    s.add_mesh(np.concatenate(P), np.concatenate(T).astype(np.int32), area_density=0.1, bending=1e-2, stretching=1e3)
    s.add_plane((0, 0, -1e-3), (0, 0, 1))
    kw = dict(time_step=1e-3, iterations=5, self_collision=True, self_tol=1e-3)
    g, o = native.Simulation(s, abi.params(precision=precision, **kw)), Oracle(s, abi.params(**kw))
    for _ in range(2):
        rg, ro = g.step(1), o.step(1)
        assert rg.n_self_contacts == ro.n_self_contacts > 512
    # the bounds of the step's parity tests: FP64, and FP32 with refinement
    rel = 1e-6 if precision == abi.PDF_FP64 else 1e-5
    qg, qo = g.state()[0], o.state()[0]
    assert np.abs(qg - qo).max() < rel * np.abs(qo).max()
