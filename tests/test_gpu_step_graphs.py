"""When dynamics change to a graph of several steps: after a long run with one step size, not in short runs that take
turns with two; and what a pair list that overflows inside such a graph gives: the steps of a list that never did."""
import ctypes

import numpy as np
import pytest

from interaxplugin import Context, InteraxDispersionForce, System
from interaxplugin import workloads as W

pytestmark = pytest.mark.gpu


def _counts(ctx):
    captures, several = ctypes.c_longlong(), ctypes.c_longlong()
    ctx._check(ctx._lib.ix_get_graph_counts(ctx._ctx, ctypes.byref(captures), ctypes.byref(several)))
    return captures.value, several.value


def test_a_long_run_takes_several_steps_at_once():
    system, pos, _ = W.water_box(64, W.box_length_for(64), 0.6, seed=4, three_body_cutoff=0.5, rigid=True)
    ctx = Context(system)
    ctx.setPositions(pos)
    ctx.runVelocityVerlet(512, 0.0002, np.zeros_like(pos))
    assert _counts(ctx)[1] == 0
    ctx.runVelocityVerlet(44, 0.0002, np.zeros_like(pos))
    assert _counts(ctx)[1] == 5                       # and four steps by themselves


def test_turns_of_two_step_sizes():
    system, pos, _ = W.water_box(64, W.box_length_for(64), 0.6, seed=4, three_body_cutoff=0.5, rigid=True)
    ctx = Context(system)
    ctx.setPositions(pos)
    ctx.runVelocityVerlet(520, 0.0002, np.zeros_like(pos))
    captures, several = _counts(ctx)
    for turn in range(8):
        ctx.runVelocityVerlet(8, (0.0001, 0.0002)[turn % 2], np.zeros_like(pos))
    # each turn captures its step, and none of them eight
    assert _counts(ctx) == (captures + 8, several)


def _meeting(capacity, graphs):
    """Two droplets without mutual neighbors that fly into one another after more than 512 steps."""
    grid = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)[:96] * 0.4
    rng = np.random.default_rng(3)
    half = grid + rng.uniform(-0.02, 0.02, size=grid.shape)
    x = np.concatenate([half, half + [0.2, 0.2, 5.0]])
    v = np.zeros_like(x)
    v[:96, 2], v[96:, 2] = 3.0, -3.0                 # 6 nm/ps: from 3.4 nm apart to the list cutoff in 600 steps of 0.7 fs
    system = System()
    force = InteraxDispersionForce()
    for i in range(len(x)):
        system.addParticle(40.0)
        force.addParticle(2.0, 0.05, 0.002, 1.2e-3, 0.025)
    force.setNonbondedMethod(InteraxDispersionForce.CutoffNonPeriodic)
    force.setCutoffDistance(0.8)
    force.setUseLongRangeCorrection(False)
    system.addForce(force)
    ctx = Context(system)
    ctx._check(ctx._lib.ix_set_graphs(ctx._ctx, int(graphs)))
    if capacity:
        ctx.setListCapacity(capacity, 0)
    ctx.setPositions(x)
    return ctx, v


def test_overflow_inside_several_steps():
    dt, steps = 0.0007, 760
    for capacity in range(1, 64):                     # the smallest list that holds the droplets apart
        ctx, v = _meeting(capacity, True)
        ctx.getState()
        if ctx.getListStats()[0] == capacity:
            break
    early, v = _meeting(capacity, True)
    early.runVelocityVerlet(512, dt, v)
    assert early.getListStats() == (capacity, 0, 0)   # no overflow before the change
    ctx, v = _meeting(capacity, True)
    x, w, energy = ctx.runVelocityVerlet(steps, dt, v)
    tiles, _, reruns = ctx.getListStats()
    assert tiles > capacity and reruns > 0 and _counts(ctx)[1] > 0
    plain, v = _meeting(0, False)
    x0, w0, energy0 = plain.runVelocityVerlet(steps, dt, v)
    assert plain.getListStats()[2] == 0 and _counts(plain) == (0, 0)
    assert np.array_equal(x, x0) and np.array_equal(w, w0) and energy == energy0
