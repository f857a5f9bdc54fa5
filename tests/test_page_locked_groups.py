"""iss_gpu_generate_into with a page-locked destination, where the sampler
launches of the two streams, the decays and the copies really run beside one
another (a copy to pageable memory keeps the host from enqueueing the next
launch): several groups of events, call after call with other seeds on one
handle, are bit for bit what generate followed by a copy gives."""
import numpy as np
import pytest
import torch

from iss_gb300 import HADRON_DTYPE, iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)
LAB = dict(MC_sampling=2, bulk_deltaf_kind=1, restrict_deltaf=1, deltaf_max_ratio=1.0, sample_pT_up_to=-1,
           sample_y_minus_eta_s_range=3)


def page_locked(n):
    return torch.zeros(n * HADRON_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(HADRON_DTYPE)


def handle(fo, events, extra):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=events, **extra))
    s.set_surface(fo)
    if extra.get("gpu_sampler"):
        s.learned_init_weights(3)
    return s


@pytest.mark.parametrize("cells,events,groups,extra", [
    (20_000, 250, 4, {}),
    (20_000, 16, 2, {}),
    (3000, 1700, 4, dict(perform_decays=1)),
    (20_000, 250, 4, dict(local_charge_conservation=1)),
    (20_000, 250, 4, dict(local_charge_conservation=1, perform_decays=1)),
    (6000, 1200, 2, dict(gpu_sampler=1)),
    (3000, 40, 2, LAB),
    (3000, 40, 2, dict(LAB, local_charge_conservation=1, perform_decays=1)),
], ids=["plain", "small", "decays", "pairs", "pairs_decays", "learned", "lab", "lab_pairs_decays"])
def test_page_locked_groups_are_the_kept_lists(cells, events, groups, extra):
    fo = S.viscous_3d(cells, seed=cells).fo_surf()
    kept, into = handle(fo, events, extra), handle(fo, events, extra)
    ref = []
    for seed in (3, 4, 5):
        kept.set_random_seed(seed)
        kept.generate_samples()
        had, off = kept.all_hadrons()
        ref.append((had.copy(), np.asarray(off).copy(), kept.counts()))
    sampled = kept.timings()["n_sampled"]
    assert sampled > 5000 and (groups < 3 or sampled > (groups - 1) * 262_144)
    out = [page_locked(max(len(r[0]) for r in ref) + 100) for _ in range(2)]
    for k in (0, 1, 2, 1, 0):
        into.set_random_seed(3 + k)
        out[k & 1][:] = 0
        had, off = into.generate_into(out[k & 1])
        assert had.tobytes() == ref[k][0].tobytes() and np.array_equal(off, ref[k][1]), k
        assert np.array_equal(into.counts(), ref[k][2]), k
    kept.close()
    into.close()
