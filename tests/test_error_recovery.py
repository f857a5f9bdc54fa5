"""A call that fails for want of memory is an error of that call alone: the next
calls, on the same handle and on others, work."""
import pytest

from iss_gb300 import IssError, iSS, surfaces as S

pytestmark = pytest.mark.gpu


def handle(**extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
                        include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1,
                        number_of_repeated_sampling=3, **extra))
    s.set_surface(S.viscous_3d(2000, seed=8).fo_surf())
    s.set_random_seed(21)
    return s


def sample(s):
    s.set_random_seed(21)
    s.generate_samples()
    return s.all_hadrons()[0].copy().tobytes()


@pytest.mark.parametrize("graph", [0, 1])
def test_an_allocation_that_fails_fails_once(graph):
    a, b = handle(), handle(gpu_graph=graph)
    ref = sample(b)
    with pytest.raises(IssError, match="out of memory"):
        a.learned_train(n_momenta=1 << 44, n_seeds=1, n_steps=1)   # more rows than any memory holds
    assert sample(b) == ref and sample(b) == ref
    a.set_params(number_of_repeated_sampling=3, perform_decays=0)
    assert sample(a) == ref
