"""Alchemical windows by the terms' alchemical part: each window against the context evaluated at that value.

The windows take the alchemical pairs and triples alone beside one evaluation at 0 when the pair terms on the parameter
share their alchemical particles and all or none have a soft core, and whole evaluations otherwise; the cases here are
the forms that the choice tells apart (which terms depend, linear or soft core, exact or order-2 overlap, periodic or
not, short and long three-body lists, more windows than are evaluated together).  The alchemical factor scales pairs
with exactly one alchemical particle and triples with an alchemical site (kernels/interaxPairForce.cu,
kernels/interaxThreeBodyForce.cu).
"""
import numpy as np
import pytest

from interaxplugin import Context
from interaxplugin import workloads as W
from interaxplugin.forces import (InteraxDispersionForce, InteraxExchangeForce, InteraxShortRangeForce,
                                  InteraxThreeBodyForce)
from parity import ENERGY_TOL, FORCE_RMS_TOL, errors

pytestmark = pytest.mark.gpu

PAIRS = (InteraxDispersionForce, InteraxExchangeForce, InteraxShortRangeForce)


def _flag(system, kinds, waters):
    """The alchemical flags of the given forces set to exactly these waters."""
    for f in system._forces:
        if not isinstance(f, kinds):
            continue
        if isinstance(f, InteraxThreeBodyForce):
            for s in range(f.getNumSites()):
                f.setSiteParameters(s, *f.getSiteParameters(s)[:-1], s in waters)
        else:
            for k in range(f.getNumParticles()):
                f.setParticleParameters(k, *f.getParticleParameters(k)[:-1], k // 3 in waters)


def _box(**kw):
    return W.water_box(216, W.box_length_for(216), 0.9, seed=4, three_body_cutoff=0.6, alchemical_waters=range(8), **kw)


def _cluster(softcore):
    system, pos, box = W.water_cluster(60, seed=9)
    _flag(system, PAIRS + (InteraxThreeBodyForce,), set(range(0, 60, 2)))
    for f in system._forces:
        if isinstance(f, PAIRS):
            f.setSoftcoreRadius(softcore)
    return system, pos, box


def _case(name):
    if name == "many soft-core windows":
        return _box(softcore_radius=0.15), np.linspace(0.0, 1.0, 70)
    if name == "order-2 overlap":
        return _box(overlap_method=InteraxExchangeForce.InteraxOrder2), np.array([0.0, 0.3, 1.0])
    if name == "half of a cluster":
        return _cluster(0.0), np.array([0.0, 0.6, 1.0])
    if name == "half of a cluster, soft core":
        return _cluster(0.1), np.array([0.0, 0.6, 1.0])
    built = _box(softcore_radius=0.15 if name == "other soft cores" else 0.0)
    system = built[0]
    if name == "dispersion alone":
        _flag(system, PAIRS[1:] + (InteraxThreeBodyForce,), set())
    elif name == "triples alone":
        _flag(system, PAIRS, set())
    elif name == "other particles":
        _flag(system, PAIRS[1], set(range(4, 12)))
    elif name == "other soft cores":
        system._forces[1].setSoftcoreRadius(0.0)
    elif name == "another parameter":
        system._forces[1].setAlchemicalParameterName("lambda_exchange")
    return built, np.array([0.0, 0.45, 1.0])


@pytest.mark.parametrize("name", ["many soft-core windows", "order-2 overlap", "half of a cluster",
                                  "half of a cluster, soft core", "dispersion alone", "triples alone", "other particles",
                                  "other soft cores", "another parameter"])
def test_each_window_is_the_evaluation_at_its_value(name):
    (system, pos, box), values = _case(name)
    ctx = Context(system)
    if box is not None:
        ctx.setPeriodicBoxVectors(*np.asarray(box))
    ctx.setPositions(pos)
    if name == "another parameter":
        ctx.setParameter("lambda_exchange", 0.7)
    for _ in range(2):               # the second pass replays the graph
        energies, forces = ctx.computeWindows("lambda_sterics", values)
    alone = ctx.computeWindows("lambda_sterics", values, getForces=False)
    assert np.array_equal(alone, energies)
    for w, lam in enumerate(values):
        ctx.setParameter("lambda_sterics", lam)
        st = ctx.getState()
        terms = st.getTermEnergies()
        e_err, f_err = errors(energies[w].sum(), forces[w], terms.sum(), st.getForces(),
                              abs_energy=np.abs(terms).sum())
        assert e_err <= ENERGY_TOL and f_err <= FORCE_RMS_TOL, (lam, e_err, f_err)
        assert np.allclose(energies[w], terms, rtol=1e-6, atol=1e-6 * np.abs(terms).sum())
