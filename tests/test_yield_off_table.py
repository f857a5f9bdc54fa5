"""Yields whose series leave the special-function tables, which a kernel of its
own evaluates directly, 32 cells of a row of groups at a time: against the FP64
oracle, with hot, cold and very cold cells anywhere among the others, at sizes
around its 32 and 128 cells, with and without diffusion; the same whatever the
order of the cells; and in a time that grows with the cells, not with the turns
of a grid."""
import numpy as np
import pytest

import oracle_lib as O
from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

CELL_RTOL = 1e-5   # FP32 against FP64, as for the reference's own yields


def params(diff):
    return dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=2, include_deltaf_shear=1,
                include_deltaf_bulk=0, include_deltaf_diffusion=diff, turn_on_rhob=1, turn_on_diff=diff,
                quantum_statistics=1, number_of_repeated_sampling=0)


def yields(fo, diff):
    s = iSS(".", inputfile="")
    s.set_params(**params(diff))
    s.set_surface(np.ascontiguousarray(fo))
    s.generate_samples()
    out, ms = s.cell_yields(), s.timings()["ms_yields"]
    s.close()
    return out, ms


@pytest.mark.parametrize("diff", [0, 1])
@pytest.mark.parametrize("n,share", [(1, 1.0), (31, 1.0), (33, 0.1), (127, 0.5), (1025, 0.02), (2600, 0.02)])
def test_direct_evaluation_anywhere(n, share, diff):
    rng = np.random.default_rng(n)
    fo = S.finite_density_3d(max(n, 64), seed=n).fo_surf()[:n].copy()
    some = rng.random(n) < share
    fo[some, 13] = rng.choice([0.3, 0.45, 0.28, 0.004, 0.006], int(some.sum())).astype(np.float32)
    fo[some & (fo[:, 13] < 0.01), 16] = 0.0
    got, _ = yields(fo, diff)
    order = rng.permutation(n)
    assert np.array_equal(yields(fo[order], diff)[0], got[:, order])
    lrf, keep = O.lrf_cells(fo)
    p = params(diff)
    ref = O.yields(O.OracleConfig(p, S.TABLE_DIR, n_events=0), O.chosen_species(S.TABLE_DIR, 2), lrf, keep)
    # FP32 holds nothing below 1e-38 of the scale, nor its relative error near it
    big = ref > 1e-25
    assert big.any()
    assert (np.abs(got.astype(np.float64)[big] - ref[big]) / ref[big]).max() < CELL_RTOL


def test_very_cold_cells_emit_nothing():
    fo = S.viscous_3d(3000, seed=7).fo_surf().copy()
    fo[::2, 13] = 0.0001
    got, _ = yields(fo, 0)
    assert not got[:, ::2].any() and got[:, 1::2].any()


def test_time_grows_with_the_cells():
    """50,000 hot cells are 1.28 times 38,912; a grid of 304 blocks takes two
    turns for the former and one for the latter, twice the time."""
    ms = []
    for n in (38_912, 50_000):
        fo = S.viscous_3d(n, seed=2).fo_surf().copy()
        fo[:, 13] = 0.3
        ms.append(min(yields(fo, 0)[1] for _ in range(2)))
    assert ms[1] < 1.6 * ms[0], ms
