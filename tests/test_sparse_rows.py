"""Cell draws on rows whose CDF is not written (few draws expected): they are
searched in the tile and run sums and the yields, and must find the cells the
full CDF rows give.

With sample_upto_desired_particle_number = 1 the number of events is not known
when the rows are made, so every row is written; the same number of events asked
for directly leaves most rows unwritten.  Both runs must agree bit for bit: at
sizes around multiples of a run (32 cells) and of a tile (2,048 cells), with
rows that start at any alignment, for one event and for many, with charge
pairs, in a batch of surfaces, in the lab-frame sampler (whose redrawn cells
take the same search) and in graph replays."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=1, turn_on_bulk=1, quantum_statistics=1,
              dN_dy_sampling_model=30, restrict_deltaf=1, deltaf_max_ratio=1.0, sample_pT_up_to=-1,
              sample_y_minus_eta_s_range=3)


def handle(fo, events, dense, **extra):
    s = iSS(".", inputfile="")
    p = dict(PARAMS, number_of_repeated_sampling=events)
    if dense:   # max(1, min(maximum, as many as 1e15 particles take)) events
        p.update(sample_upto_desired_particle_number=1, number_of_particles_needed=1e9,
                 maximum_sampling_events=events)
    p.update(extra)
    s.set_params(**p)
    s.set_surface(fo)
    s.set_random_seed(21)
    return s


def sample(s):
    s.generate_samples()
    had, off = s.all_hadrons()
    return had.copy(), off.copy()


# 13,056 cells are the smallest surface with unwritten rows (319 x 7 tiles)
@pytest.mark.parametrize("cells,events,extra", [
    (13_056, 1, {}), (14_335, 30, {}), (14_336, 3, {}), (14_337, 30, {}), (20_511, 200, {}),
    (33_001, 7, dict(local_charge_conservation=1)), (16_385, 2, dict(MC_sampling=2, gpu_max_tries=300)),
    (25_000, 900, dict(dN_dy_sampling_model=1)),
])
def test_sparse_rows_give_the_cells_of_the_full_cdf(cells, events, extra):
    fo = S.viscous_3d(cells, seed=cells).fo_surf()
    ref, off = sample(handle(fo, events, True, **extra))
    had, o = sample(handle(fo, events, False, **extra))
    assert len(ref) > 1000 and np.array_equal(off, o)
    assert had.tobytes() == ref.tobytes()


def test_sparse_rows_of_a_batch_and_of_graph_replays():
    sizes, events = (9_001, 2_047, 6_500), (3, 40, 1)
    surfaces = [S.viscous_3d(n, seed=n).fo_surf() for n in sizes]
    b = handle(surfaces[0], 1, False)
    b.set_surface_batch(surfaces, events)
    had, off = sample(b)
    first = 0
    for fo, n in zip(surfaces, events):
        # single surfaces of these sizes have all rows written
        ref, o = sample(handle(fo, n, False, gpu_event_offset=first))
        a = off[first]
        assert had[a:off[first + n]].tobytes() == ref.tobytes()
        assert np.array_equal(off[first:first + n + 1] - a, o)
        first += n
    fo = S.viscous_3d(15_000, seed=5).fo_surf()
    ref, _ = sample(handle(fo, 9, True))
    g = handle(fo, 9, False, gpu_graph=1)
    for _ in range(3):
        assert sample(g)[0].tobytes() == ref.tobytes()
