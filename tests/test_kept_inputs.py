"""Small inputs that stay on the device between calls (species, pids, yield
list, surfaces, events): a handle that is taken through species lists, event
numbers, surface sizes and batches, back and forth, samples bit for bit what a
fresh handle samples for each, with and without graph replay."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, include_deltaf_shear=1, include_deltaf_bulk=1,
              bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)
SURF = {n: S.viscous_3d(n, seed=n).fo_surf() for n in (700, 2100)}

# (afterburner, events or per-surface events, cells per surface)
STEPS = [(0, 3, (700,)), (2, 3, (700,)), (2, 5, (700,)), (2, (1, 4), (700, 2100)), (2, (4, 1), (700, 2100)),
         (0, (4, 1), (2100, 700)), (0, 5, (2100,)), (0, 3, (700,))]


def sample(s, afterburner, events, cells, graph):
    s.set_params(**dict(PARAMS, afterburner_type=afterburner, gpu_graph=graph,
                        number_of_repeated_sampling=events if len(cells) == 1 else 1))
    if len(cells) == 1:
        s.set_surface(SURF[cells[0]])
    else:
        s.set_surface_batch([SURF[n] for n in cells], list(events))
    s.set_random_seed(4)
    s.generate_samples()
    had, off = s.all_hadrons()
    return had.copy(), off.copy(), s.species_yields() if len(cells) == 1 else None


@pytest.mark.parametrize("graph", [0, 1])
def test_every_step_is_what_a_fresh_handle_gives(graph):
    used = iSS(".", inputfile="")
    for step in STEPS:
        fresh = iSS(".", inputfile="")
        for repeat in range(2):   # the second is a replay of the first's graph
            a, b = sample(used, *step, graph), sample(fresh, *step, graph)
            assert len(a[0]) > 100 and a[0].tobytes() == b[0].tobytes() and np.array_equal(a[1], b[1])
            if a[2] is not None:
                assert np.array_equal(a[2], b[2])
