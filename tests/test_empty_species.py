"""A species list that becomes empty and comes back: a user's table folder whose
list for one afterburner names no particle samples no hadron there, and the
handle's next call with the full list is that of a fresh handle, bit for bit, also
with replayed graphs."""
import shutil

import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, include_deltaf_shear=1, include_deltaf_bulk=1,
              bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1, number_of_repeated_sampling=3)


def sample(s, afterburner, fo):
    s.set_params(**dict(PARAMS, afterburner_type=afterburner))
    s.set_surface(fo)
    s.set_random_seed(4)
    s.generate_samples()
    had, off = s.all_hadrons()
    return had.copy(), np.asarray(off).copy(), s.species_yields()


@pytest.mark.parametrize("graph", [0, 1])
def test_the_full_list_after_an_empty_one(tmp_path, graph):
    tables = tmp_path / "iSS_tables"
    shutil.copytree(S.TABLE_DIR, tables)
    (tables / "chosen_particles_SMASH.dat").write_text("")
    fo = S.viscous_3d(700, seed=3).fo_surf()
    ref = sample(iSS(".", inputfile="", table_path=str(tables)), 0, fo)
    assert len(ref[0]) > 100
    used = iSS(".", inputfile="", table_path=str(tables))
    used.set_params(gpu_graph=graph)
    for afterburner in (0, 2, 0, 0, 2, 2, 0):
        had, off, totals = sample(used, afterburner, fo)
        if afterburner == 2:
            assert len(had) == 0 and not off.any() and len(totals) == 0
        else:
            assert had.tobytes() == ref[0].tobytes() and np.array_equal(off, ref[1])
            assert np.array_equal(totals, ref[2])
