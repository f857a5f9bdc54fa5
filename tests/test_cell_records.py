"""The 128-byte cell records are written by the prologue only for the calls
whose kernels read them.  A handle that sampled without them trains on the same
rows as a fresh one, samples the same hadrons afterwards, and takes the learned
proposal as a handle that never sampled without it; with and without replayed
graphs.  All comparisons are exact."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1,
              number_of_repeated_sampling=3)


def handle(**kw):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, **kw))
    s.set_surface(S.viscous_3d(3000, seed=8).fo_surf())
    return s


def sample(s, seed, **kw):
    s.set_params(**kw)
    s.set_random_seed(seed)
    s.generate_samples()
    return s.all_hadrons()[0].copy()


def train(s):
    s.learned_train(n_momenta=60_000, first_seed=10, n_seeds=2, n_steps=20, batch=4096,
                    learning_rate=2e-3, init_seed=1)
    return s.learned_rows(0, 60_000)


@pytest.mark.parametrize("graph", [0, 1])
def test_records_follow_the_call(graph):
    fresh, used = handle(gpu_graph=graph), handle(gpu_graph=graph)
    before = [sample(used, 3), sample(used, 3)]
    rows_used, rows_fresh = train(used), train(fresh)
    for a, b in zip(rows_used, rows_fresh):
        assert np.array_equal(a, b)
    assert np.abs(rows_used[0]).max() > 0
    after = [sample(used, 3), sample(used, 3)]
    for had in before[1:] + after:
        assert had.tobytes() == before[0].tobytes()


def test_fermion_compatibility_after_a_plain_call():
    """The compatibility sampler reads the records; the lean one does not."""
    fresh, used = handle(gpu_compat_fermion_cdf2=1), handle(gpu_compat_fermion=0)
    plain = sample(used, 5)
    a, b = sample(fresh, 5), sample(used, 5, gpu_compat_fermion_cdf2=1)
    assert a.tobytes() == b.tobytes()
    assert sample(used, 5, gpu_compat_fermion_cdf2=0).tobytes() == plain.tobytes()
