"""iss_gpu_generate_into samples groups of event chunks in launches that
alternate between two streams: whatever the number of chunks and groups, the
hadrons are those of iss_gpu_generate followed by a copy, bit for bit, call
after call on one handle."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


# one event; less than one group; several groups (262,144 hadrons each)
@pytest.mark.parametrize("cells,events", [(3000, 1), (3000, 7), (20_000, 250)])
def test_groups_give_the_hadrons_of_generate(cells, events):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events))
    s.set_surface(S.viscous_3d(cells, seed=12).fo_surf())
    s.set_random_seed(3)
    s.generate_samples()
    ref, ref_off = s.all_hadrons()
    ref, cnt, tries = ref.copy(), s.counts(), s.timings()["n_tries"]
    out = np.zeros(len(ref) + 100, dtype=ref.dtype)
    for chunks in (1, 2, 3, 16, 64):
        s.set_tuning(copy_chunks=chunks)
        out[:] = 0
        had, off = s.generate_into(out)
        assert had.tobytes() == ref.tobytes() and np.array_equal(off, ref_off), chunks
        assert np.array_equal(s.counts(), cnt) and s.timings()["n_tries"] == tries, chunks
