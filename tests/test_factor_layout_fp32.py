"""pdf_factor_check checks the factor that the handle of these parameters would
have: FP32 scenes are dissected by rules of their own (layers that overlap together,
three merged levels at every size).  The emulation itself is in 64 bits."""
import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle


# layers that overlap, layers apart, tiny ones gathered, and a single cloth
@pytest.mark.parametrize("n,layers,spacing", [(62, 2, 0.02), (62, 2, 0.2), (4, 40, 0.02), (90, 1, 0.02)])
def test_fp32_factor_solves_the_system(n, layers, spacing):
    s = scenes.cloth_on_sphere(n=n, layers=layers, spacing=spacing, side=1.0, pins=layers == 1)
    kw = dict(time_step=2e-3, iterations=5)
    b = np.random.default_rng(n).standard_normal((s.n_vertices, 3))
    x = native.factor_check(s, abi.params(precision=abi.PDF_FP32_REFINE, **kw), b)
    o = Oracle(s, abi.params(**kw))
    xo = o.solve(b)
    assert np.abs(x - xo).max() <= 1e-9 * np.abs(xo).max()
    assert np.abs(o.lhs() @ x - b).max() <= 1e-9 * np.abs(b).max()
    # another dissection rounds otherwise (FP64: apart, four merged levels)
    assert not np.array_equal(x, native.factor_check(s, abi.params(**kw), b))
