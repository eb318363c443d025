"""Which triples the three-body kernels see, and from which sites: the order of the cell grid's lists (ties of the
ordering coordinate, boxes of three cells, dense lists of the fast kernel, lists that overflowed) and the lists of the
two triple kernels around the length where one hands over to the other, against the FP64 oracle."""
import numpy as np
import pytest

import pyoracle
from interaxplugin import Context, InteraxThreeBodyForce, System
from parity import ENERGY_TOL, FORCE_RMS_TOL, errors

pytestmark = pytest.mark.gpu


def _system(positions, cutoff, box=None, damped=False, per_molecule=1, alchemical=(), seed=0):
    rng = np.random.default_rng(seed)
    system = System()
    if box is not None:
        system.setDefaultPeriodicBoxVectors((box, 0, 0), (0, box, 0), (0, 0, box))
    force = InteraxThreeBodyForce()
    for i in range(len(positions)):
        system.addParticle(1.0)
        force.addSite([i], rng.uniform(0.001, 0.002), rng.uniform(700.0, 1300.0), rng.uniform(0.02, 0.05),
                      i // per_molecule, i in alchemical)
    force.setCutoffDistance(cutoff)
    force.setUsesPeriodicBoundaryConditions(box is not None)
    if damped:
        force.setDampingMethod(force.TangToennies)
        force.setCentroidDampingRadius(0.15)
    system.addForce(force)
    return system


def _check(system, positions, box=None, capacity=0, parameters=None):
    ctx = Context(system)
    if capacity:
        ctx.setListCapacity(0, capacity)
    for name, value in (parameters or {}).items():
        ctx.setParameter(name, value)
    ctx.setPositions(positions)
    reference = pyoracle.evaluate(system, positions, None if box is None else np.eye(3) * box, parameters=parameters)
    first = ctx.getState()
    count = ctx.getCounts()[1]
    for state in (first, ctx.getState()):       # the second with the lists grown, after an overflow
        e_err, f_err = errors(state.getPotentialEnergy(), state.getForces(), *reference)
        assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (e_err, f_err)
        assert ctx.getCounts()[1] == count
    return count


def _triples(positions, cutoff, box, per_molecule=1):
    """Triples of three molecules with every distance (nearest images) within the cutoff."""
    d = positions[None] - positions[:, None]
    d -= box * np.round(d / box)
    near = (d ** 2).sum(-1) < cutoff ** 2
    mol = np.arange(len(positions)) // per_molecule
    near &= mol[None] != mol[:, None]
    n = near.astype(np.int64)
    return int((n @ n * n).sum()) // 6


def _spaced(rng, n, edge, gap):
    out = np.empty((0, 3))
    while len(out) < n:
        p = rng.uniform(0, edge, 3)
        d = out - p
        d -= edge * np.round(d / edge)
        if not len(out) or (d ** 2).sum(1).min() > gap * gap:
            out = np.vstack([out, p])
    return out


@pytest.mark.parametrize("damped", [False, True])
@pytest.mark.parametrize("cells,cutoff,n,capacity", [(3.0, 0.45, 190, 0), (3.0, 0.45, 190, 3), (4.3, 0.5, 700, 0),
                                                     (3.0, 0.3, 2, 0), (3.0, 0.3, 3, 0)])
def test_cell_grid_lists(cells, cutoff, n, capacity, damped):
    rng = np.random.default_rng(n + capacity)
    box = cells * (cutoff + 0.1 + 1e-3) + 1e-9
    x = _spaced(rng, n, box, 0.12)
    x += box * rng.integers(-2, 3, size=x.shape)                # images: the order must not depend on them
    system = _system(x, cutoff, box, damped, per_molecule=2 if n > 3 else 1, alchemical=(1, 5), seed=n)
    count = _check(system, x, box, capacity, {"lambda_sterics": 0.7})
    assert count == _triples(x, cutoff, box, 2 if n > 3 else 1)


def test_ties_of_the_ordering_coordinate():
    # a lattice in planes of equal x, on the boundary among them: whole rows of sites are ordered by their index
    side, box = 7, 2.1
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * (box / side)
    grid[:, 1:] += np.random.default_rng(3).uniform(-0.02, 0.02, size=(len(grid), 2))
    count = _check(_system(grid, 0.55, box), grid, box)
    assert count == _triples(grid, 0.55, box)


@pytest.mark.parametrize("cutoff,spacing", [(0.6, 0.21), (0.6, 0.19), (0.6, 0.165)])
def test_dense_cell_grid_lists(cutoff, spacing):
    # half lists of about 57, 76 and 115 sites: past the length at which an index-ordered list changes kernels, and
    # (the last) past what the fast kernel holds
    side = int(np.ceil(3 * (cutoff + 0.101) / spacing)) + 1
    box = side * spacing
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * spacing
    grid = grid + np.random.default_rng(5).uniform(-0.02, 0.02, size=grid.shape)
    count = _check(_system(grid, cutoff, box), grid, box)
    assert count == _triples(grid, cutoff, box)


@pytest.mark.parametrize("damped", [False, True])
@pytest.mark.parametrize("n", [4, 9, 33, 64, 65, 66, 129, 258, 290])
def test_cluster_lists_around_the_kernels_limits(n, damped):
    rng = np.random.default_rng(n)
    edge = 0.31 * n ** (1.0 / 3.0)
    x = _spaced(rng, n, edge + 0.3, 0.15)
    count = _check(_system(x, 100.0, None, damped, seed=n), x)
    assert count == n * (n - 1) * (n - 2) // 6


def test_small_periodic_box_needs_images_between_neighbors():
    # the cutoff beyond a third of the box: two neighbors of a site can be nearest through another image
    rng = np.random.default_rng(11)
    box, cutoff = 1.2, 0.55
    x = _spaced(rng, 60, box, 0.16)
    count = _check(_system(x, cutoff, box), x, box)
    assert count == _triples(x, cutoff, box)
