"""Pair lists of i-blocks with more candidate blocks than the list search keeps for each: every block of a triclinic box
above 12,288 particles, where none is pruned, and most of a box a few cutoffs wide.  The results are the FP64 oracle's,
and a rebuild costs no more than its tiles: the candidates of a tile are found without a search from the i-block on,
which is cubic in the number of blocks (a rebuild then took 8 evaluations of 24,000 particles in a triclinic box and 2
with the long cutoff; it takes about 1 and 0.3)."""
import ctypes

import numpy as np
import pytest
import torch

import pyoracle
from interaxplugin import Context
from interaxplugin import workloads as W
from parity import ENERGY_TOL, FORCE_RMS_TOL, errors

pytestmark = pytest.mark.gpu


def _box(waters, cutoff, skew):
    edge = W.box_length_for(waters)
    system, pos, _ = W.water_box(waters, edge, cutoff, seed=waters, three_body=False)
    box = np.diag([edge] * 3)
    if skew:
        box[1, 0], box[2, 0], box[2, 1] = 0.1 * edge, 0.05 * edge, -0.1 * edge
    return system, np.asarray(pos), box


@pytest.mark.parametrize("waters,cutoff,skew", [(4100, 0.9, True), (4100, 2.3, False), (5003, 2.4, False)])
def test_against_the_oracle(waters, cutoff, skew):
    system, pos, box = _box(waters, cutoff, skew)
    ctx = Context(system)
    ctx.setPeriodicBoxVectors(*box)
    ctx.setPositions(pos)
    state = ctx.getState()
    scale = []
    e, f = pyoracle.evaluate(system, pos, box, abs_energy=scale)
    e_err, f_err = errors(state.getPotentialEnergy(), state.getForces(), e, f, max(scale[0], abs(e)))
    assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (e_err, f_err)
    # the same list by another order of the particles' cells: moved as a whole, in rectangular and triclinic frames
    ctx.setPositions(pos + 0.37)
    moved = ctx.getState()
    assert np.abs(moved.getForces() - state.getForces()).max() <= 1e-5 * np.abs(f).max()


@pytest.mark.parametrize("cutoff,skew,limit", [(1.0, True, 3.0), (2.6, False, 1.0)])
def test_time_of_a_rebuild(cutoff, skew, limit):
    system, pos, box = _box(8000, cutoff, skew)
    ctx = Context(system)
    ctx.setPeriodicBoxVectors(*box)
    ctx.setPositions(pos)
    ctx.getState()
    lib, stream = ctx._lib, torch.cuda.ExternalStream(ctx._lib.ix_get_stream(ctx._ctx))
    frames = [torch.as_tensor(pos + shift, device="cuda") for shift in (0.0, 0.2)]
    out = torch.zeros(len(pos), 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def time(used):
        best = np.inf
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record(stream)
            for k in range(8):
                ctx._check(lib.ix_compute_device_f64(ctx._ctx, 7, ctypes.c_void_p(frames[k % used].data_ptr()), None,
                                                     ctypes.c_void_p(out.data_ptr()), None))
            end.record(stream)
            end.synchronize()
            best = min(best, start.elapsed_time(end) / 8)
        return best

    alone, rebuilt = time(1), time(2)
    assert rebuilt - alone <= limit * alone, (alone, rebuilt)
