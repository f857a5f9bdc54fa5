"""Generation 0 of the decays, whose events and particle ids come from the offsets
of the (event, species) segments, 32 segments to a warp: events of one hadron or
none (warps of mostly empty segments, over several events) and of thousands
(segments shared by many warps), with and without charge pairs, against the same
events sampled few at a time; and the time of a call of many small events, whose
segments are nearly all empty."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


def handle(fo, events, **extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, perform_decays=1, number_of_repeated_sampling=events, **extra))
    s.set_surface(fo)
    s.set_random_seed(6)
    return s


def sample(fo, events, **extra):
    s = handle(fo, events, **extra)
    s.generate_samples()
    had, off = s.all_hadrons()
    out = had.copy(), np.asarray(off).copy()
    s.close()
    return out


@pytest.mark.parametrize("lcc", [0, 1])
@pytest.mark.parametrize("cells,events,part", [(3, 1201, 7), (90, 250, 31), (40_000, 3, 1)])
def test_events_do_not_depend_on_their_neighbours(cells, events, part, lcc):
    fo = S.viscous_3d(cells, seed=cells).fo_surf()
    had, off = sample(fo, events, local_charge_conservation=lcc)
    assert len(had) > 100 and ((np.diff(off) == 0).any() or cells > 3)
    for first in (0, part, events - part):
        a, o = sample(fo, part, local_charge_conservation=lcc, gpu_event_offset=first)
        assert np.array_equal(o, off[first:first + part + 1] - off[first])
        assert a.tobytes() == had[off[first]:off[first + part]].tobytes()


def test_time_of_many_small_events():
    """The decays of 100,000 events of nine hadrons take less than the rest of
    the call, whose counts go over the same segments (15 % of it; 170 % with a
    warp for each segment)."""
    fo = S.viscous_3d(40, seed=2).fo_surf()
    ms = []
    for decays in (0, 1):
        s = handle(fo, 100_000)
        s.set_params(perform_decays=decays)
        best = 1e30
        for _ in range(6):
            s.generate_samples()
            t = s.timings()
            best = min(best, t["ms_total"] + t["ms_decays"])
        ms.append(best)
        s.close()
    assert ms[1] < 2.0 * ms[0], ms
