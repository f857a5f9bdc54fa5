"""Launch shapes tuned for one sampler are not handed to another: handles of one
surface and event number that differ in the sampler, the diffusion or the bulk
form tune for themselves, and the lab-frame sampler, which takes neither the
draws per work item nor the sampler blocks per SM, leaves both alone."""
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

BASE = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
            include_deltaf_bulk=1, bulk_deltaf_kind=1, turn_on_bulk=1, quantum_statistics=1,
            number_of_repeated_sampling=4, restrict_deltaf=1, deltaf_max_ratio=1.0, sample_pT_up_to=-1,
            sample_y_minus_eta_s_range=3)
CELLS = 731


def handle(**extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(BASE, **extra))
    s.set_surface(S.viscous_3d(CELLS, seed=8).fo_surf())
    s.set_random_seed(21)
    return s


def test_shapes_stay_with_their_kernels():
    a = handle(MC_sampling=4)
    a.set_tuning(copy_chunks=7)   # not tuned: marks the shape that a's tuning keeps
    a.autotune()
    same = handle(MC_sampling=4, gpu_autotune=1)
    same.generate_samples()
    assert same.get_tuning() == a.get_tuning() and same.get_tuning()["copy_chunks"] == 7
    for other in (dict(MC_sampling=2), dict(include_deltaf_bulk=0), dict(bulk_deltaf_kind=11),
                  dict(include_deltaf_diffusion=1, turn_on_diff=1)):
        s = handle(**dict(dict(MC_sampling=4), gpu_autotune=1, **other))
        s.generate_samples()
        assert s.get_tuning()["copy_chunks"] == 16, other


def test_the_lab_frame_sampler_keeps_what_it_does_not_take():
    s = handle(MC_sampling=2)
    for item_size, ctas in ((1024, 1), (32, 3)):
        s.set_tuning(item_size=item_size, sampler_ctas=ctas)
        t, _, _ = s.autotune()
        assert (t["item_size"], t["sampler_ctas"]) == (item_size, ctas)
