"""gpu_compat_fermion_cdf2 on a handle that sampled without it: the
compatibility sampler takes another path (other hadrons than the plain one) that
reads the 128-byte cell records, and switching it on and off gives on one handle
what fresh handles give."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1,
              number_of_repeated_sampling=3)


def handle(compat, graph):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, gpu_compat_fermion_cdf2=compat, gpu_graph=graph))
    s.set_surface(S.viscous_3d(3000, seed=8).fo_surf())
    return s


def sample(s, compat):
    s.set_params(gpu_compat_fermion_cdf2=compat)
    s.set_random_seed(5)
    s.generate_samples()
    return s.all_hadrons()[0].copy()


@pytest.mark.parametrize("graph", [0, 1])
def test_switching_the_compatibility_sampler(graph):
    plain, compat = sample(handle(0, 0), 0), sample(handle(1, 0), 1)
    assert len(plain) > 500 and plain.tobytes() != compat.tobytes()
    used = handle(0, graph)
    for on in (0, 0, 1, 1, 0, 1, 0):
        assert sample(used, on).tobytes() == (compat if on else plain).tobytes(), on
