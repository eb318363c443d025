"""Evaluations and alchemical windows whose status comes back without a page-locked slot, as on a host that has none left
(ix_set_pinned_status): the same results, with lists that overflow in the first evaluation among them.  The lists grow
only after every kernel that reads them: a site list that has grown holds nothing before its next build."""
import numpy as np
import pytest

from interaxplugin import Context
from interaxplugin import workloads as W

pytestmark = pytest.mark.gpu

VALUES = np.array([0.0, 0.45, 1.0])


def _context(softcore, pinned, capacity):
    system, pos, _ = W.water_box(216, W.box_length_for(216), 0.9, seed=4, three_body_cutoff=0.6,
                                 alchemical_waters=range(8), softcore_radius=softcore)
    ctx = Context(system)
    ctx._check(ctx._lib.ix_set_pinned_status(ctx._ctx, int(pinned)))
    ctx.setListCapacity(*capacity)
    ctx.setPositions(pos)
    return ctx


@pytest.mark.parametrize("capacity", [(0, 0), (0, 3), (8, 3)])
@pytest.mark.parametrize("softcore", [0.0, 0.15])
def test_windows_without_a_slot(softcore, capacity):
    want_e, want_f = _context(softcore, True, (0, 0)).computeWindows("lambda_sterics", VALUES)
    ctx = _context(softcore, False, capacity)
    counts = []
    for _ in range(2):                      # the lists overflow in the first call and have grown in the second
        energies, forces = ctx.computeWindows("lambda_sterics", VALUES)
        # the lists' capacity decides which triple kernel takes a site, so the sums differ in their last bits
        assert np.allclose(energies, want_e, rtol=1e-6, atol=1e-6 * np.abs(want_e).sum(1).max())
        assert np.abs(forces - want_f).max() <= 1e-5 * np.abs(want_f).max()
        counts.append(ctx.getCounts())
    assert counts[0] == counts[1]
    assert ctx.getListStats()[1] > 3


@pytest.mark.parametrize("capacity", [(0, 0), (8, 3)])
def test_states_without_a_slot(capacity):
    states = [_context(0.0, pinned, capacity).getState() for pinned in (True, False)]
    assert np.array_equal(states[0].getForces(), states[1].getForces())
    assert np.array_equal(states[0].getTermEnergies(), states[1].getTermEnergies())
