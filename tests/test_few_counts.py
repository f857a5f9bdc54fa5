"""Counts of up to 32 events of one surface come from one kernel, of more events
(or of a batch, or in a replayed graph) from two: the events both have draw the
same counts, for means on both sides of the inversion table's end and for every
count model."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


def counts(fo, events, batch=False, **extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events, **extra))
    if batch:
        s.set_surface_batch([fo, fo], [events, 1])
    else:
        s.set_surface(fo)
    s.set_random_seed(12)
    s.generate_samples()
    out = s.counts()
    s.close()
    return out


@pytest.mark.parametrize("extra", [{}, dict(local_charge_conservation=1), dict(dN_dy_sampling_model=1),
                                   dict(dN_dy_sampling_model=10, dN_dy_sampling_para1=0.4),
                                   dict(dN_dy_sampling_model=20, dN_dy_sampling_para1=0.4)])
@pytest.mark.parametrize("cells", [60, 2500])
def test_one_kernel_draws_what_two_draw(cells, extra):
    fo = S.viscous_3d(cells, seed=cells).fo_surf()
    many = counts(fo, 65, **extra)
    assert many.sum() > 100
    for events in (64, 33, 32, 1):
        assert np.array_equal(counts(fo, events, **extra), many[:events])
    assert np.array_equal(counts(fo, 30, batch=True, **extra)[:30], many[:30])
