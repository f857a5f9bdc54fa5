"""Negative net baryon densities with the Chapman-Enskog table (bulk_deltaf_kind
21), whose row index the reference does not bound from below: far negative ones,
which would index before the table, leave the call and the other cells alone."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=2, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=21, turn_on_bulk=1, turn_on_rhob=1, quantum_statistics=1,
              number_of_repeated_sampling=2)


def yields(fo):
    s = iSS(".", inputfile="")
    s.set_params(**PARAMS)
    s.set_surface(fo)
    s.set_random_seed(2)
    s.generate_samples()
    out = s.cell_yields()
    s.close()
    return out


def test_far_negative_densities_stay_inside_the_table():
    fo = S.finite_density_3d(400, seed=5).fo_surf().copy()
    ref = yields(fo)
    some = np.arange(400) % 5 == 2
    fo[some, 15] = np.resize(np.array([-1.0, -50.0, -1e6, -1e30, -np.inf], dtype=np.float32), int(some.sum()))
    got = yields(fo)
    assert np.array_equal(got[:, ~some], ref[:, ~some])
