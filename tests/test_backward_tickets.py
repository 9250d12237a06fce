"""The backward block sweep's tickets (csrc/sweep_kernels.cu).

The launches of one solve after the first are programmatic dependents: every
kernel of the chain lets the next one start at once, so before its
griddepcontrol.wait a kernel may run beside any earlier one of its chain, and
reads only what none of them writes.  The forward block sweep rewinds the
backward sweep's ticket queue, so the backward sweep must not touch the queue
before its wait.

The first test reads that off the kernel source; the second restates the chain
as a state machine, with the first ticket drawn before the wait and taken from
the CTA's index, under random interleavings; the third (GPU) runs many solves
back to back on a schedule without upper levels, where the backward sweep is
the forward sweep's direct dependent.
"""
import os
import random
import re

import numpy as np
import pytest

from climatenet_b200 import abi, native, scenes
from oracle.oracle import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def kernels():
    """name -> body of every kernel of the sweeps."""
    src = open(os.path.join(ROOT, "climatenet_b200", "csrc", "sweep_kernels.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(k_\w+)\s*\(", src):
        start = src.index("{", m.end())
        depth, end = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
            if depth == 0:
                break
        out[m.group(1)] = src[start:end]
    return out


def test_dependents_touch_no_queue_before_their_wait():
    bodies = kernels()
    dependents = [n for n in bodies if "griddep_wait()" in bodies[n]]
    assert {"k_block_backward", "k_upper_level"} <= set(dependents)
    for n in dependents:
        before = bodies[n][:bodies[n].index("griddep_wait()")]
        assert "sy.queue" not in before and "sy.epoch" not in before and "sy.fdone" not in before, n


def solves(n_solves, n_blocks, n_ctas, early, seed):
    """Blocks taken by the backward sweep of each solve: its CTAs may start while
    the forward launch has not yet rewound the queue.  early: the first ticket is
    drawn from the queue before the wait; else it is the CTA's index."""
    rng = random.Random(seed)
    queue, taken = 0, []
    for _ in range(n_solves):
        blocks = []
        ctas = [None] * n_ctas  # a CTA's current ticket; None: not started
        rewound, waited = False, [False] * n_ctas
        done = [False] * n_ctas
        while not all(done):
            acts = [] if rewound else ["rewind"]
            for c in range(n_ctas):
                if done[c]:
                    continue
                if ctas[c] is None or rewound:  # the wait ends after the forward launch
                    acts.append(c)
            a = rng.choice(acts)
            if a == "rewind":
                queue, rewound = 0, True
            elif ctas[a] is None:
                if early:
                    ctas[a], queue = queue, queue + 1
                else:
                    ctas[a] = a
            elif not waited[a]:
                waited[a] = True
            elif ctas[a] >= n_blocks:
                done[a] = True
            else:
                blocks.append(ctas[a])
                ctas[a], queue = queue + (0 if early else n_ctas), queue + 1
        taken.append(sorted(blocks))
    return taken


@pytest.mark.parametrize("n_blocks,n_ctas", [(1, 1), (1, 4), (5, 2), (7, 7), (40, 8)])
def test_every_block_is_taken_once(n_blocks, n_ctas):
    for seed in range(200):
        assert solves(4, n_blocks, n_ctas, False, seed) == [list(range(n_blocks))] * 4


def test_tickets_drawn_before_the_wait_lose_and_repeat_blocks():
    lost = repeated = False
    for seed in range(200):
        for t in solves(4, 5, 2, True, seed):
            lost |= len(set(t)) < 5
            repeated |= len(set(t)) < len(t)
    assert lost and repeated


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PDF_FP64, abi.PDF_FP32_REFINE])
def test_solves_back_to_back_without_upper_levels(precision):
    s = scenes.cloth_on_sphere(n=24, side=1.0, z=-0.2455, mu=0.3, layers=12, spacing=0.02, sphere_center=(0, 0, -0.5),
                               sphere_radius=0.25, pins=True)
    kw = dict(time_step=5e-3, iterations=40)
    g = native.Simulation(s, abi.params(precision=precision, **kw))
    g.set_sweep_schedule(64, 7, 1, 1)
    st = g.stats()
    assert st.sweep_blocks > 0
    if precision == abi.PDF_FP64:  # a cloth is one block
        assert st.sweep_blocks == 12 and st.sweep_upper_levels == 0
    o = Oracle(s, abi.params(**kw))
    for _ in range(4):
        assert g.step(1).n_contacts == o.step(1).n_contacts
    # the step's parity bounds: FP64, and FP32 with refinement
    rel = 1e-6 if precision == abi.PDF_FP64 else 1e-5
    for a, b in zip(g.state(), o.state()):
        assert np.abs(a - b).max() < rel * np.abs(b).max()
