"""Poisson constants of the counts: a warp per (surface, species) row up to 4,096
rows, a thread per row above.  With 319 species a batch of 12 surfaces is the
last of the former and one of 13 the first of the latter: the surfaces both have
draw the same counts, and those of each surface by itself, for means on both
sides of the inversion table's end; a batch of rows that do not fill the last
block, and one of rows by the ten thousand, likewise."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


def counts(surfaces, events, first=0, **extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events[0], gpu_event_offset=first, **extra))
    if len(surfaces) == 1:
        s.set_surface(surfaces[0])
    else:
        s.set_surface_batch(surfaces, events)
    s.set_random_seed(12)
    s.generate_samples()
    out = s.counts()
    s.close()
    assert out.shape == (sum(events), 319)
    return out


@pytest.mark.parametrize("extra", [{}, dict(local_charge_conservation=1)])
@pytest.mark.parametrize("surfaces", [13, 14, 70])
def test_a_thread_per_row_gives_what_a_warp_gives(surfaces, extra):
    sizes = [(60, 2500, 7, 900)[k % 4] for k in range(surfaces)]
    events = [(2, 40, 1, 5)[k % 3] for k in range(surfaces)]
    fo = [S.viscous_3d(n, seed=k + 1).fo_surf() for k, n in enumerate(sizes)]
    many = counts(fo, events, **extra)
    twelve = counts(fo[:12], events[:12], **extra)
    assert twelve.sum() > 1000 and twelve.max() > 12
    assert np.array_equal(many[:len(twelve)], twelve)
    for k in (0, 1, 11, 12, surfaces - 1):
        first = sum(events[:k])
        assert np.array_equal(many[first:first + events[k]],
                              counts(fo[k:k + 1], events[k:k + 1], first, **extra)), k
