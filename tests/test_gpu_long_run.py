"""Dynamics past the point where a run changes to a graph of several steps: the same steps as launched one by one.

The kernels and their order are the same, and the sums do not depend on the order of the additions, so the states are
equal to the last bit.
"""
import numpy as np
import pytest

from interaxplugin import Context
from interaxplugin import workloads as W

pytestmark = pytest.mark.gpu


def _run(rigid, graphs, parts):
    system, pos, box = W.water_box(216, W.box_length_for(216), 0.9, seed=4, three_body_cutoff=0.6, rigid=rigid)
    ctx = Context(system)
    ctx._check(ctx._lib.ix_set_graphs(ctx._ctx, int(graphs)))
    ctx.setPositions(pos)
    x, v = pos, np.zeros_like(pos)
    for steps in parts:
        ctx.setPositions(x)
        x, v, energy = ctx.runVelocityVerlet(steps, 0.0002, v)
    return x, v, energy


@pytest.mark.parametrize("rigid", [True, False])
def test_a_long_run_is_its_steps_one_by_one(rigid):
    parts = [300, 270]                   # the change after 512 steps, in the second part, and two steps left over
    for a, b in zip(_run(rigid, True, parts), _run(rigid, False, parts)):
        assert np.array_equal(a, b)
