"""Per-cell yields against the FP64 oracle where the yields kernel takes its
different ways: runs of species that share a yield (no strangeness and charge
potential in the warp's cells) and member by member otherwise, both kinds in one
surface, series with arguments off the special-function tables (pions above
0.27 GeV, a second kernel), blocks that are not full, with and without
diffusion; and a batch whose blocks span surfaces."""
import numpy as np
import pytest

import oracle_lib as O
from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

CELL_RTOL = 1e-5   # FP32 against FP64, as for the reference's own yields


def cells(n, potentials, hot):
    rng = np.random.default_rng(n)
    fo = S.finite_density_3d(max(n, 64), seed=n).fo_surf()[:n].copy()
    if hot:
        fo[::3, 13] = rng.uniform(0.2, 0.45, len(fo[::3]))
    if potentials == "none":
        fo[:, 16] = 0.0
    if potentials in ("all", "some"):
        rows = slice(None) if potentials == "all" else slice(n // 3, 2 * n // 3)
        fo[rows, 17] = rng.uniform(-0.05, 0.1, len(fo[rows]))
        fo[rows, 18] = rng.uniform(-0.03, 0.02, len(fo[rows]))
    return fo


@pytest.mark.parametrize("n,potentials,hot,diff", [
    (1, "all", 0, 0), (127, "none", 1, 0), (128, "baryon", 0, 1), (129, "some", 1, 1), (700, "some", 0, 0),
    (700, "all", 1, 0), (257, "baryon", 1, 0), (300, "none", 0, 1),
])
def test_yields_against_the_oracle(n, potentials, hot, diff):
    fo = cells(n, potentials, hot)
    p = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=2, include_deltaf_shear=1,
             include_deltaf_bulk=0, include_deltaf_diffusion=diff, turn_on_rhob=1, turn_on_diff=diff,
             quantum_statistics=1, number_of_repeated_sampling=0)
    s = iSS(".", inputfile="")
    s.set_params(**p)
    s.set_surface(fo)
    s.set_random_seed(1)
    s.generate_samples()
    got = s.cell_yields().astype(np.float64)
    lrf, keep = O.lrf_cells(fo)
    ref = O.yields(O.OracleConfig(p, S.TABLE_DIR, n_events=0), O.chosen_species(S.TABLE_DIR, 2), lrf, keep)
    assert got.shape == ref.shape
    big = ref > 1e-30 * ref.max()
    rel = np.abs(got[big] - ref[big]) / ref[big]
    assert rel.max() < CELL_RTOL
    # the maxima behind the fixed-point sums: the totals are the rows' sums
    tot = s.species_yields()
    assert np.allclose(tot, got.sum(1), rtol=1e-6, atol=0)


def test_blocks_that_span_surfaces():
    sizes, events = (100, 37, 200, 1, 90), (5, 400, 3, 900, 20)
    surfaces = [cells(n, "some" if k % 2 else "baryon", k == 2) for k, n in enumerate(sizes)]
    p = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=2, include_deltaf_shear=0,
             include_deltaf_bulk=0, quantum_statistics=1)
    b = iSS(".", inputfile="")
    b.set_params(**p)
    b.set_surface_batch(surfaces, events)
    b.set_random_seed(9)
    b.generate_samples()
    had, off = b.all_hadrons()
    had, first = had.copy(), 0
    for fo, n in zip(surfaces, events):
        s = iSS(".", inputfile="")
        s.set_params(**dict(p, number_of_repeated_sampling=n, gpu_event_offset=first))
        s.set_surface(fo)
        s.set_random_seed(9)
        s.generate_samples()
        ref, _ = s.all_hadrons()
        assert had[off[first]:off[first + n]].tobytes() == ref.tobytes(), len(fo)
        first += n
