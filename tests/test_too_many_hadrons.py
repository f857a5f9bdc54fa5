"""A surface whose yield of a species exceeds what an int32 counts (here a cell of
an enormous normal; a space-time rapidity whose boost cancels in float does the
same) is refused, whatever the count model and whichever kernels count, and the
handle goes on with the next surface."""
import numpy as np
import pytest

from iss_gb300 import IssError, iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=0,
              include_deltaf_bulk=0, quantum_statistics=1)


def cell(da0):
    c = np.zeros((1, 34), dtype=np.float32)
    c[0, 0], c[0, 4], c[0, 8] = 10.0, da0, 1.0
    c[0, 12], c[0, 13], c[0, 14] = 0.25, 0.15, 0.04
    return c


@pytest.mark.parametrize("events,graph", [(1, 0), (3, 1), (40, 0), (700, 0)])
@pytest.mark.parametrize("extra", [{}, dict(dN_dy_sampling_model=1), dict(local_charge_conservation=1),
                                   dict(dN_dy_sampling_model=10, dN_dy_sampling_para1=0.4),
                                   dict(dN_dy_sampling_model=20, dN_dy_sampling_para1=0.4)])
def test_counts_beyond_an_int32_are_refused(extra, events, graph):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events, gpu_graph=graph, **extra))
    s.set_random_seed(3)
    s.set_surface(cell(4.0))
    s.generate_samples()
    ref = s.all_hadrons()[0].copy()
    for da0 in (1e12, 1e18, 1e25, 1e36):
        s.set_surface(cell(da0))
        for _ in range(2):
            with pytest.raises(IssError, match="than an int32 counts"):
                s.generate_samples()
    s.set_surface(cell(4.0))
    s.generate_samples()
    assert s.all_hadrons()[0].tobytes() == ref.tobytes()
    s.close()
