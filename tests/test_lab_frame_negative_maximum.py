"""The lab-frame sampler on bosons whose chemical potential exceeds their mass:
the reference's maximum of the emission function is negative there, and a
proposal above the pole is accepted where its flux through the surface is
negative too.  The bound that rejects proposals in bulk must not apply.  Without
delta f the cap restrict_deltaf changes nothing but that bound, so both settings
give the same hadrons."""
import numpy as np
import pytest

from iss_gb300 import IssError, iSS, surfaces as S

pytestmark = pytest.mark.gpu


def sample(mu_s, restrict):
    c = np.zeros((1, 34), dtype=np.float32)
    c[0, 0], c[0, 4], c[0, 5], c[0, 8] = 10.0, 8.0, 180.0, 1.0   # a space-like normal
    c[0, 12], c[0, 13], c[0, 14], c[0, 17] = 0.25, 0.15, 0.04, mu_s
    s = iSS(".", inputfile="")
    s.set_params(**dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=0,
                        include_deltaf_bulk=0, quantum_statistics=1, number_of_repeated_sampling=4, MC_sampling=2,
                        restrict_deltaf=restrict, deltaf_max_ratio=1.0, sample_pT_up_to=-1,
                        sample_y_minus_eta_s_range=3.0, gpu_max_redraws=1))
    s.set_surface(c)
    s.set_random_seed(77)
    try:
        s.generate_samples()
    except IssError as e:   # hadrons that no proposal fits are given up
        assert "abandoned" in str(e)
    had, off = s.all_hadrons()
    out = had.copy(), np.asarray(off).copy(), s.timings()["n_tries"]
    s.close()
    return out


@pytest.mark.parametrize("mu_s", [0.0, 0.45, 0.55, 0.6])
def test_the_bound_needs_a_positive_maximum(mu_s):
    had, off, tries = sample(mu_s, 1)
    ref, o, t = sample(mu_s, 0)
    assert len(ref) > 50
    assert np.array_equal(off, o) and had.tobytes() == ref.tobytes() and tries == t
