"""Rows of the network's loss without a target (K not above 0, NaN included)
contribute nothing, whatever stands in their direction: the loss and the
gradient of a batch with such rows are finite, and those of the same batch with
finite directions in them.

A boost-invariant surface sampled over a wide rapidity range makes such rows
itself: |z / t| of a hadron rounds to 1 beyond a space-time rapidity of 9, where
the row's target is not a number.  Training on them leaves finite weights."""
import os
import sys

import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as M  # noqa: E402

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")


def batch(n, seed):
    rng = np.random.default_rng(seed)
    f = rng.normal(0.0, 0.5, (n, M.N_FEAT)).astype(np.float32)
    t = np.zeros((n, 4), dtype=np.float32)
    t[:, 0] = rng.gamma(2.5, 1.0, n) + 1e-2
    v = rng.normal(size=(n, 3))
    t[:, 1:] = v / np.linalg.norm(v, axis=1, keepdims=True)
    return f, t


@pytest.mark.parametrize("K", [0.0, -0.0, -1.5, NAN, -INF])
@pytest.mark.parametrize("direction", [(NAN, NAN, NAN), (INF, 0.0, 0.0), (0.0, -INF, 0.0), (0.0, 0.0, NAN)])
def test_dead_rows_count_nothing(K, direction):
    f, t = batch(260, 3)
    dead = np.zeros(260, dtype=bool)
    dead[[0, 7, 127, 128, 200, 259]] = True
    clean = t.copy()
    clean[dead, 0] = 0.0
    t[dead, 0] = K
    t[dead, 1:] = direction
    s = iSS(".", inputfile="")
    s.learned_set_weights(M.initial_like(4))
    loss, grad = s.learned_loss_grad(f, t)
    ref, gref = s.learned_loss_grad(f, clean)
    s.close()
    # the same live rows: only the order of the FP32 atomic sums differs, as
    # between two runs of one batch (a few 1e-7 of each layer's gradient)
    assert np.isfinite(loss) and np.isfinite(grad).all()
    assert abs(loss - ref) <= 1e-6 * abs(ref)
    for w, b in M.OFFSETS:
        assert np.linalg.norm(grad[w:b] - gref[w:b]) <= 1e-5 * np.linalg.norm(gref[w:b])


def test_training_rows_beyond_the_rapidity_of_one():
    s = iSS(".", inputfile="")
    s.set_params(**dict(S.DEFAULT_PARAMETERS, hydro_mode=1, afterburner_type=0, include_deltaf_shear=0,
                        include_deltaf_bulk=0, quantum_statistics=1, number_of_repeated_sampling=2,
                        y_LB=-12, y_RB=12))
    s.set_surface(S.ideal_boost_invariant(dx=2.0).fo_surf())
    curve = s.learned_train(n_momenta=20_000, first_seed=10, n_seeds=1, n_steps=20, batch=4096,
                            learning_rate=1e-3, init_seed=1)
    _, t = s.learned_rows(0, 20_000)
    w = s.learned_get_weights()
    s.close()
    assert (~np.isfinite(t)).any()
    assert np.isfinite(w).all() and np.isfinite(curve).all()
