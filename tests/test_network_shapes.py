"""The network's loss and gradient at the edges of the kernels' tiles: rows
around 128 (a tile), one row, more tiles than SMs, against the FP64 oracle with
the same bf16 rounding points and the bounds of test_learned_network.py: the
loss to 1e-4, the gradient of every layer to 1e-2 (relative Frobenius norm).
Rows without a target (K <= 0) count nothing: with as many of them as live rows
the gradient is half that of the live rows alone, a factor that no bf16 rounding
sees, so that only the order of FP32 sums is left (1e-5)."""
import os
import sys

import numpy as np
import pytest

from iss_gb300 import iSS

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as M  # noqa: E402

pytestmark = pytest.mark.gpu


def batch(n, seed):
    rng = np.random.default_rng(seed)
    f = rng.normal(0.0, 0.5, (n, M.N_FEAT)).astype(np.float32)
    t = np.zeros((n, 4), dtype=np.float32)
    t[:, 0] = rng.gamma(2.5, 1.0, n) + 1e-2
    v = rng.normal(size=(n, 3))
    t[:, 1:] = v / np.linalg.norm(v, axis=1, keepdims=True)
    return f, t


def handle():
    s = iSS(".", inputfile="")
    s.learned_set_weights(M.initial_like(4))
    return s


@pytest.mark.parametrize("n", [1, 31, 128, 19_500])
def test_loss_and_gradient(n):
    params = M.initial_like(4).astype(np.float64)
    f, t = batch(n, n)
    loss, grad = handle().learned_loss_grad(f, t)
    rloss, rgrad = M.loss_grad(params, f.astype(np.float64), t.astype(np.float64))
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    for layer, (w, b) in enumerate(M.OFFSETS):
        for a, end in ((w, b), (b, b + M.DIM_OUT[layer])):
            ref = rgrad[a:end]
            assert np.linalg.norm(grad[a:end] - ref) <= 1e-2 * np.linalg.norm(ref) + 1e-7, (n, layer, a)


@pytest.mark.parametrize("n", [1, 64, 127, 1000])
def test_rows_without_a_target(n):
    f, t = batch(2 * n, n)
    live = np.zeros(2 * n, dtype=bool)
    live[np.random.default_rng(n).permutation(2 * n)[:n]] = True
    t[~live, 0] = 0.0
    s = handle()
    loss, grad = s.learned_loss_grad(f, t)
    alone, g1 = s.learned_loss_grad(f[live], t[live])
    assert abs(loss - 0.5 * alone) < 1e-5 * abs(alone)
    assert np.linalg.norm(grad - 0.5 * g1) <= 1e-5 * np.linalg.norm(g1)
