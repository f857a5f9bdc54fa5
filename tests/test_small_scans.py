"""Slot scans, work-item map and report of a call: one kernel up to 8,192
(event, species) segments, separate kernels above.  With 319 species 25 events
are the last of the former and 26 the first of the latter: the events they
share are the same bit for bit, whatever the draws per work item and also on a
handle whose item map was too small for the call."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


def sample(s, events):
    s.set_params(number_of_repeated_sampling=events)
    s.generate_samples()
    had, off = s.all_hadrons()
    cnt = s.counts()
    assert np.array_equal(np.diff(off), cnt.sum(1)) and off[0] == 0 and off[-1] == len(had)
    return had.copy(), off.copy(), cnt


@pytest.mark.parametrize("lcc", [0, 1])
@pytest.mark.parametrize("item_size", [32, 1024])
def test_both_sides_of_the_small_scan(lcc, item_size):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, local_charge_conservation=lcc, number_of_repeated_sampling=1))
    s.set_tuning(item_size=item_size)
    s.set_surface(S.viscous_3d(4000, seed=6).fo_surf())
    s.set_random_seed(17)
    ref, off, cnt = sample(s, 60)
    for events in (1, 25, 26, 2, 0, 60):
        had, o, c = sample(s, events)
        assert np.array_equal(o, off[:events + 1]) and np.array_equal(c, cnt[:events])
        assert had.tobytes() == ref[:off[events]].tobytes(), events
