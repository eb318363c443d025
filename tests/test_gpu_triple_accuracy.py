"""The error of the three-body forces against FP64, over clusters whose sites all see one another (the wide triple kernel,
sums of hundreds of terms) and periodic boxes (the fast one, with and without damping).

The bounds are 1.1 times the mean errors of kernels that kept every force of a triple and added them in short runs
(measured on the same inputs); sums in rows as long as the list, with approximate quotients, exceed the first by a third.
"""
import numpy as np
import pytest

import pyoracle
from interaxplugin import Context, InteraxThreeBodyForce, System

pytestmark = pytest.mark.gpu


def _system(n, cutoff, box, damped, rng):
    system = System()
    if box:
        system.setDefaultPeriodicBoxVectors((box, 0, 0), (0, box, 0), (0, 0, box))
    force = InteraxThreeBodyForce()
    for i in range(n):
        system.addParticle(1.0)
        force.addSite([i], rng.uniform(0.001, 0.002), rng.uniform(700.0, 1300.0), rng.uniform(0.02, 0.05), i, False)
    force.setCutoffDistance(cutoff)
    force.setUsesPeriodicBoundaryConditions(box is not None)
    if damped:
        force.setDampingMethod(force.TangToennies)
    system.addForce(force)
    return system


def _positions(n, box, rng):
    """Sites of a jittered lattice of spacing 0.31 nm: the n nearest the origin, or n of a whole box."""
    side = int(np.ceil(n ** (1 / 3) - 1e-9)) if box else int(np.ceil(n ** (1 / 3))) + 3
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.31
    if not box:
        grid = grid - grid.mean(0) + rng.uniform(-0.15, 0.15, 3)
        grid = grid[np.argsort((grid ** 2).sum(1))][:n]
    return grid + rng.uniform(-0.06, 0.06, size=grid.shape)


@pytest.mark.parametrize("n,cutoff,box,damped,bound", [(258, 100.0, None, False, 3.0e-7),
                                                       (290, 100.0, None, True, 3.15e-7),
                                                       (3375, 0.75, 15 * 0.31, False, 3.27e-7)])
def test_force_error(n, cutoff, box, damped, bound):
    error = []
    for seed in range(6):
        rng = np.random.default_rng([n, seed])
        system = _system(n, cutoff, box, damped, rng)
        x = _positions(n, box, rng)
        ctx = Context(system)
        ctx.setPositions(x)
        f = ctx.getState().getForces()
        _, want = pyoracle.evaluate(system, x, None if box is None else np.eye(3) * box)
        error.append(np.sqrt(((f - want) ** 2).sum() / (want ** 2).sum()))
    print(f"mean relative RMS error {np.mean(error):.3e}")
    assert np.mean(error) <= bound
