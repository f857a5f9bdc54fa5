"""A training call that fails on the way (here: rows that no device memory
holds) leaves the handle as the caller set it: parameters, seed, and the hadrons
it samples next."""
import numpy as np
import pytest

from iss_gb300 import IssError, iSS, surfaces as S

pytestmark = pytest.mark.gpu

SET = dict(number_of_repeated_sampling=3, perform_decays=1, gpu_event_offset=5,
           sample_upto_desired_particle_number=0)


def handle():
    s = iSS(".", inputfile="")
    s.set_params(**dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
                        include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1, **SET))
    s.set_surface(S.viscous_3d(2000, seed=8).fo_surf())
    s.set_random_seed(21)
    return s


def sample(s):
    s.generate_samples()
    had, off = s.all_hadrons()
    return had.copy(), np.asarray(off).copy()


def test_failed_training_leaves_the_handle_alone():
    s = handle()
    ref, off = sample(s)
    with pytest.raises(IssError):
        s.learned_train(n_momenta=1 << 44, n_seeds=1, n_steps=1)
    for key, value in SET.items():
        assert s.getVal(key) == value, key
    assert s.getVal("gpu_sampler", 0) == 0
    had, o = sample(s)
    assert np.array_equal(o, off) and had.tobytes() == ref.tobytes()
    s.close()


def test_failed_training_holds_no_rows():
    """The rows held before went with their buffer: more steps on them, and
    reading them, are refused."""
    s = handle()
    s.set_params(perform_decays=0)
    s.learned_train(n_momenta=4000, n_seeds=1, n_steps=2, batch=256)
    rows, _ = s.learned_rows(0, 4000)
    assert np.abs(rows).max() > 0
    with pytest.raises(IssError):
        s.learned_train(n_momenta=1 << 44, n_seeds=1, n_steps=1)
    with pytest.raises(IssError, match="needs training rows"):
        s.learned_train(n_momenta=0, n_seeds=1, n_steps=1)
    with pytest.raises(IssError, match="0 training rows held"):
        s.learned_rows(0, 1)
    s.learned_train(n_momenta=4000, n_seeds=1, n_steps=2, batch=256)
    again, _ = s.learned_rows(0, 4000)
    assert np.array_equal(again, rows)
    s.close()
