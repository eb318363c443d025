"""The pair list at the sizes where its parts change: one particle to a few blocks of 32 (an odd and an even number of
blocks pair differently), every kind of boundary, moving particles across rebuilds, and a box so uneven that a block's
candidates exceed what the list keeps per block; against brute force and the FP64 oracle."""
import numpy as np
import pytest

import pyoracle
from interaxplugin import Context, InteraxDispersionForce, System
from parity import ENERGY_TOL, FORCE_RMS_TOL, errors

pytestmark = pytest.mark.gpu


def _system(n, method, cutoff, box, active=None, exclude=True):
    system = System()
    if box is not None:
        system.setDefaultPeriodicBoxVectors(*box)
    force = InteraxDispersionForce()
    for i in range(n):
        system.addParticle(12.0)
        on = active is None or active[i]
        force.addParticle(2.0 + 0.1 * (i % 3), 0.05, 0.002, 1.2e-3 if on else 0.0, 0.025)
    if exclude:
        for i in range(0, n - 1, 3):
            force.addExclusion(i, i + 1)
    force.setNonbondedMethod(method)
    force.setCutoffDistance(cutoff)
    force.setUseLongRangeCorrection(False)
    system.addForce(force)
    return system


def _points(rng, n, box):
    """Points in the box at least 0.14 nm apart, nearest images included."""
    m = np.array(box)
    out = np.empty((0, 3))
    while len(out) < n:
        p = rng.uniform(0, 1, 3) @ m
        d = out - p
        for k in (2, 1, 0):
            d = d - np.round(d[:, k] / m[k, k])[:, None] * m[k]
        if not len(out) or (d ** 2).sum(1).min() > 0.14 ** 2:
            out = np.vstack([out, p])
    return out


def _pairs(x, box, cutoff, active):
    d = x[None] - x[:, None]
    if box is not None:
        m = np.array(box)
        for k in (2, 1, 0):
            d = d - np.floor(d[..., k] / m[k, k] + 0.5)[..., None] * m[k]
    near = (d ** 2).sum(-1) < cutoff ** 2
    near &= active[None] & active[:, None]
    for i in range(0, len(x) - 1, 3):
        near[i, i + 1] = near[i + 1, i] = False
    return int(np.triu(near, 1).sum())


CUBE = ((2.3, 0, 0), (0, 2.3, 0), (0, 0, 2.3))
SKEW = ((2.4, 0, 0), (0.6, 2.3, 0), (-0.5, 0.4, 2.2))


@pytest.mark.parametrize("kind", ["none", "nonperiodic", "cube", "skew"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 127, 129, 320, 353])
def test_sizes_and_boundaries(n, kind):
    rng = np.random.default_rng(n)
    method = {"none": InteraxDispersionForce.NoCutoff, "nonperiodic": InteraxDispersionForce.CutoffNonPeriodic}.get(
        kind, InteraxDispersionForce.CutoffPeriodic)
    box = dict(cube=CUBE, skew=SKEW).get(kind)
    cutoff = 1.0 if kind != "none" else 50.0
    x = _points(rng, n, box or CUBE)
    if box:
        x = x + rng.integers(-2, 3, size=(n, 3)) @ np.array(box)     # images
    active = np.arange(n) % 5 != 4
    system = _system(n, method, cutoff, box, active)
    ctx = Context(system)
    for step in range(3):                                             # the second within the skin, the third beyond it
        ctx.setPositions(x)
        state = ctx.getState()
        assert ctx.getCounts()[0] == _pairs(x, box, cutoff, active)
        e, f = pyoracle.evaluate(system, x, None if box is None else np.array(box))
        if ctx.getCounts()[0]:
            e_err, f_err = errors(state.getPotentialEnergy(), state.getForces(), e, f)
            assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (step, e_err, f_err)
        else:
            assert state.getPotentialEnergy() == 0.0 and not state.getForces().any()
        x = x + rng.uniform(-1, 1, size=(n, 3)) * (0.004 if step == 0 else 0.02) + (0.0 if step == 0 else 0.1)


@pytest.mark.parametrize("n", [2305, 8193])
def test_larger_lists_and_their_growth(n):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    box = np.eye(3) * side * 0.28
    x = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 0.28
    x = x + rng.uniform(-0.07, 0.07, size=x.shape)
    system = _system(n, InteraxDispersionForce.CutoffPeriodic, 0.9, box)
    ctx = Context(system)
    ctx.setPositions(x)
    state = ctx.getState()
    e, f = pyoracle.evaluate(system, x, box)
    e_err, f_err = errors(state.getPotentialEnergy(), state.getForces(), e, f)
    assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (e_err, f_err)
    small = Context(system)
    small.setListCapacity(16, 0)                                      # grown after an overflow: the same sums
    small.setPositions(x)
    again = small.getState()
    assert np.array_equal(again.getForces(), state.getForces())
    assert np.array_equal(again.getTermEnergies(), state.getTermEnergies())


def test_dense_droplet_beyond_the_kept_entries():
    # 30,000 particles within 2 nm of a 20 nm box, most of them without parameters: every block is a candidate of every
    # other, more than the list keeps per block, and the tiles exceed the estimate from the mean density
    rng = np.random.default_rng(7)
    n, cutoff = 30000, 0.9
    box = ((20.0, 0, 0), (0, 20.0, 0), (0, 0, 20.0))
    x = 9.0 + rng.uniform(0, 2.0, size=(n, 3))
    active = np.zeros(n, bool)
    active[rng.choice(n, 500, replace=False)] = True
    # the interacting ones on a lattice, so that none are in contact
    grid = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)[:500] * 0.25
    x[active] = 9.0 + grid + rng.uniform(-0.03, 0.03, size=grid.shape)
    system = _system(n, InteraxDispersionForce.CutoffPeriodic, cutoff, box, active, exclude=False)
    ctx = Context(system)
    ctx.setPositions(x)
    state = ctx.getState()
    some = np.flatnonzero(active)
    small = _system(len(some), InteraxDispersionForce.CutoffPeriodic, cutoff, box, exclude=False)
    for k, i in enumerate(some):                                      # the same parameters
        small.getForce(0).setParticleParameters(k, 2.0 + 0.1 * (i % 3), 0.05, 0.002, 1.2e-3, 0.025, False)
    e, f = pyoracle.evaluate(small, x[some], np.array(box))
    e_err, f_err = errors(state.getPotentialEnergy(), state.getForces()[some], e, f)
    assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (e_err, f_err)
    assert not state.getForces()[~active].any()
