"""Which form of the NEP kernel a call takes (host rule, no GPU needed)."""
import itertools

import pytest

from ai2pot_b200 import capi


def _lanes(natoms, ntypes, functions, neurons, umax, is_f64=0, descriptors=0):
    return capi.lib().ai2b_nep_lanes_per_atom(natoms, ntypes, functions, functions, 8, neurons, umax, is_f64, descriptors)


def test_many_atoms_never_lose_the_specialised_kernel():
    """A model that the specialised kernel serves at a few atoms (the most lanes, the least shared memory) keeps it at any
    number of atoms, and the lanes never grow with the number of atoms."""
    for ntypes, functions, neurons, umax, f64, desc in itertools.product((1, 3, 8, 10, 11, 12, 13, 16), (4, 8), (10, 30, 100),
                                                                        (16, 32, 64, 100, 128, 200, 300, 1000), (0, 1), (0, 1)):
        few = _lanes(1, ntypes, functions, neurons, umax, f64, desc)
        assert few in (0, 32)
        row = [_lanes(n, ntypes, functions, neurons, umax, f64, desc) for n in (1000, 1001, 6000, 6001, 49999, 50000, 10 ** 6)]
        if few == 0:
            assert not any(row)
        else:
            assert min(row) > 0 and row == sorted(row, reverse=True)


@pytest.mark.parametrize("natoms,ntypes,neurons,umax,f64,lanes", [
    (60000, 12, 30, 32, 0, 8), (60000, 3, 30, 32, 0, 4), (60000, 3, 30, 36, 0, 8), (20000, 3, 30, 64, 0, 8), (20000, 3, 30, 128, 1, 16),
    (5000, 3, 30, 64, 0, 16), (900, 3, 30, 64, 0, 32), (900, 16, 30, 64, 0, 0), (900, 17, 4, 64, 0, 0), (900, 3, 30, 1025, 0, 0)])
def test_forms_of_single_models(natoms, ntypes, neurons, umax, f64, lanes):
    assert _lanes(natoms, ntypes, 4, neurons, umax, f64) == lanes
    assert _lanes(natoms, ntypes, 9, neurons, umax, f64) == 0
