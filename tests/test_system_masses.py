"""The masses a System hands to a Context, however the System came about: kept by an earlier build of this package (whose
Systems kept no array of them), copied, or added to through a copy that shares its lists."""
import copy
import pickle

from interaxplugin import System


def _system():
    system = System()
    for mass in (1.5, 2.0):
        system.addParticle(mass)
    return system


def test_a_system_kept_by_an_earlier_build():
    state = _system().__dict__.copy()
    state.pop("_mass_array", None)
    system = System.__new__(System)
    system.__dict__.update(state)
    assert system._masses_array().tolist() == [1.5, 2.0]
    system.addParticle(3.0)
    assert system._masses_array().tolist() == [1.5, 2.0, 3.0]


def test_copies():
    system = _system()
    assert system._masses_array().tolist() == [1.5, 2.0]
    for other in (copy.deepcopy(system), pickle.loads(pickle.dumps(system))):
        other.addParticle(4.0)
        assert other._masses_array().tolist() == [1.5, 2.0, 4.0]
        assert system._masses_array().tolist() == [1.5, 2.0]
    shared = copy.copy(system)                    # the same list of masses
    shared.addParticle(5.0)
    assert system.getNumParticles() == 3
    assert system._masses_array().tolist() == shared._masses_array().tolist() == [1.5, 2.0, 5.0]
