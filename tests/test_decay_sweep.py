"""The decay sweeps: final lists of up to 4,096 events are laid out by one block,
of more by separate kernels, and tiles of 2,048 inputs make up the scans.  An
event's decayed list depends on its seed and number alone, so a run of many
events holds the lists of a run of few; work buffers that are too small cost a
rerun and nothing else; events without a hadron stay empty."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S
from iss_gb300.native import HADRON_DTYPE

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1,
              perform_decays=1)


def sample(fo, events, into=False, **extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events, **extra))
    s.set_surface(fo)
    s.set_random_seed(6)
    if into:
        had, off = s.generate_into(np.zeros(2_000_000, dtype=HADRON_DTYPE))
    else:
        s.generate_samples()
        had, off = s.all_hadrons()
    reruns = s.timings()["decay_reruns"]
    out = had.copy(), np.asarray(off).copy(), reruns
    s.close()
    return out


@pytest.mark.parametrize("into", [False, True])
@pytest.mark.parametrize("cells,few,many", [(40, 4096, 4097), (3, 4095, 9000), (1500, 1, 7)])
def test_lists_do_not_depend_on_the_number_of_events(cells, few, many, into):
    fo = S.viscous_3d(cells, seed=cells).fo_surf()
    a, off_a, _ = sample(fo, few, into)
    b, off_b, _ = sample(fo, many, into)
    assert len(a) > 100 and off_a[-1] == len(a) and off_b[-1] == len(b)
    assert np.array_equal(off_a, off_b[:few + 1])
    assert a.tobytes() == b[:off_b[few]].tobytes()
    if cells == 3:
        assert (np.diff(off_b) == 0).any()


@pytest.mark.parametrize("into", [False, True])
def test_small_buffers_cost_a_rerun_only(into):
    fo = S.viscous_3d(2100, seed=3).fo_surf()
    ref, off, none = sample(fo, 9, into)
    had, o, reruns = sample(fo, 9, into, gpu_decay_arena_factor=0.3, gpu_decay_next_factor=0.01)
    assert none == 0 and reruns >= 1
    assert np.array_equal(o, off) and had.tobytes() == ref.tobytes()


@pytest.mark.parametrize("extra", [{}, dict(local_charge_conservation=1)])
def test_copied_groups_are_the_kept_lists(extra):
    """A host destination takes the lists in groups of events, whose count sweep
    ran beside the sampler; the kept lists are written at once."""
    fo = S.viscous_3d(1300, seed=5).fo_surf()
    ref, off, _ = sample(fo, 2600, False, **extra)
    had, o, _ = sample(fo, 2600, True, **extra)
    assert len(ref) > 400_000
    assert np.array_equal(o, off) and had.tobytes() == ref.tobytes()


def test_abandoned_hadrons_are_kept_without_an_id():
    """Hadrons that the sampler gives up carry no particle id and do not decay."""
    fo = S.viscous_3d(1300, seed=5).fo_surf()
    out = []
    for decays in (0, 1):
        s = iSS(".", inputfile="")
        s.set_params(**dict(PARAMS, number_of_repeated_sampling=40, perform_decays=decays, gpu_max_tries=1,
                            gpu_max_redraws=0))
        s.set_surface(fo)
        s.set_random_seed(6)
        with pytest.raises(Exception, match="abandoned"):
            s.generate_samples()
        had, _ = s.all_hadrons()
        out.append(int((had["pid"] == 0).sum()))
        s.close()
    assert out[0] > 100 and out[0] == out[1]
