"""The yields kernel with diffusion: the loop over runs (warps whose cells have
no strangeness and charge potential and lie in a block of one surface), the
general loop (blocks of several surfaces, blocks that are not full, the other
warps) and the kernel of arguments off the special-function tables must round
alike, since the yields feed integer sums: a surface's yields are those of its
pieces and of its place in a batch, bit for bit."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

BASE = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, include_deltaf_shear=1, quantum_statistics=1, afterburner_type=2,
            include_deltaf_diffusion=1, turn_on_diff=1, turn_on_rhob=1, number_of_repeated_sampling=0)
KINDS = {
    "none": dict(include_deltaf_bulk=0),
    "ce": dict(include_deltaf_bulk=1, bulk_deltaf_kind=1, turn_on_bulk=1),
    "14": dict(include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1),
}


def yields(kind, *pieces):
    s = iSS(".", inputfile="")
    s.set_params(**dict(BASE, **KINDS[kind]))
    if len(pieces) == 1:
        s.set_surface(np.ascontiguousarray(pieces[0]))
    else:
        s.set_surface_batch([np.ascontiguousarray(p) for p in pieces], [0] * len(pieces))
    s.generate_samples()
    out = s.cell_yields()
    s.close()
    return out


@pytest.mark.parametrize("kind", ["none", "ce", "14"])
@pytest.mark.parametrize("n,hot", [(127, 0), (1280, 0), (1281, 1), (3001, 0), (6400, 1)])
def test_every_way_through_the_kernel_rounds_alike(n, hot, kind):
    rng = np.random.default_rng(n)
    fo = S.finite_density_3d(n, seed=n).fo_surf().copy()
    if hot:
        some = rng.random(n) < 0.05
        fo[some, 13] = rng.uniform(0.2, 0.45, int(some.sum())).astype(np.float32)
    whole = yields(kind, fo)
    assert whole.max() > 0
    # no piece fills a block, and no block of the batch lies on one surface
    pieces = np.array_split(fo, n // 50)
    assert yields(kind, *pieces).tobytes() == whole.tobytes()
    halves = [yields(kind, fo[:n // 2 + 3]), yields(kind, fo[n // 2 + 3:])]
    assert np.concatenate(halves, axis=1).tobytes() == whole.tobytes()
    # the last cell of every warp takes the warp to the general loop
    mixed = fo.copy()
    mixed[31::32, 17] = 0.02
    keep = np.ones(n, dtype=bool)
    keep[31::32] = False
    assert np.array_equal(yields(kind, mixed)[:, keep], whole[:, keep])
