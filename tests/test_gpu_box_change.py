"""A box that changes while the particles stay where they are, or move less than the lists allow (a barostat's trial, a
strained cell): the lists hold images and neighbors of the box they were built with, so they are built anew."""
import ctypes

import numpy as np
import pytest
import torch

import pyoracle
from interaxplugin import Context
from interaxplugin import workloads as W
from parity import ENERGY_TOL, FORCE_RMS_TOL, errors

pytestmark = pytest.mark.gpu


def _boxes(edge):
    yield np.diag([edge * 1.01] * 3)
    yield np.diag([edge * 0.995, edge * 1.01, edge])
    yield np.array([[edge, 0, 0], [0.02 * edge, edge, 0], [0, -0.01 * edge, edge]])
    yield np.diag([edge] * 3)


@pytest.mark.parametrize("waters", [216, 2500])
def test_the_lists_follow_the_box(waters):
    edge = W.box_length_for(waters)
    system, pos, box = W.water_box(waters, edge, 0.85, seed=3, three_body_cutoff=0.5)
    rng = np.random.default_rng(waters)
    pos = np.asarray(pos) + np.repeat(rng.integers(-2, 3, size=(waters, 3)), 3, axis=0) * edge      # images
    ctx = Context(system)
    ctx.setPositions(pos)
    ctx.getState()
    x = torch.as_tensor(pos, device="cuda")
    f = torch.zeros(len(pos), 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for new in _boxes(edge):
        ctx.setPeriodicBoxVectors(*new)
        state = ctx.getState()
        scale = []
        e_ref, f_ref = pyoracle.evaluate(system, pos, new, abs_energy=scale)
        e_err, f_err = errors(state.getPotentialEnergy(), state.getForces(), e_ref, f_ref, max(scale[0], abs(e_ref)))
        assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (new, e_err, f_err)
    # the same through the device entry point, which takes the box with the positions
    for new in _boxes(edge):
        box9 = np.ascontiguousarray(new, dtype=np.float64).reshape(9)
        ctx._check(ctx._lib.ix_compute_device_f64(ctx._ctx, 15, ctypes.c_void_p(x.data_ptr()),
                                                  box9.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(f.data_ptr()),
                                                  None))
        ctx._check(ctx._lib.ix_synchronize(ctx._ctx))
        _, f_ref = pyoracle.evaluate(system, pos, new)
        err = np.sqrt(((f.cpu().numpy() - f_ref) ** 2).sum() / (f_ref ** 2).sum())
        assert err <= FORCE_RMS_TOL, (new, err)
