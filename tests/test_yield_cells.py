"""One and two cells per thread of the yields kernel (two from 2,500 cells on
without diffusion), and the loop over runs against the general one: the yields
of a surface are those of its pieces, bit for bit, at sizes around a warp's 64
and a block's 256 cells, with cells that have a strangeness or charge potential
among the others, with cells that are dropped, and in a batch."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

BASE = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, include_deltaf_shear=1, quantum_statistics=1,
            number_of_repeated_sampling=0)
KINDS = {
    "none": dict(include_deltaf_bulk=0, afterburner_type=0),
    "ce": dict(include_deltaf_bulk=1, bulk_deltaf_kind=1, turn_on_bulk=1, afterburner_type=2),
    "14": dict(include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, afterburner_type=2),
}


def yields(fo, kind, batch=None):
    s = iSS(".", inputfile="")
    s.set_params(**dict(BASE, **KINDS[kind]))
    if batch is None:
        s.set_surface(fo)
    else:
        s.set_surface_batch(batch, [0] * len(batch))
    s.generate_samples()
    out = s.cell_yields()
    s.close()
    return out


@pytest.mark.parametrize("kind", ["none", "ce", "14"])
@pytest.mark.parametrize("n", [2499, 2500, 2560, 2561, 2816, 4001])
def test_yields_do_not_depend_on_the_cells_per_thread(n, kind):
    rng = np.random.default_rng(n)
    fo = S.finite_density_3d(n, seed=n).fo_surf().copy()
    fo[:700, 16] = 0.0                                    # no baryon potential
    some = rng.random(n) < 0.004                          # a few warps take the general loop
    some[:1200] = False
    fo[some, 17] = 0.03
    fo[some & (rng.random(n) < 0.5), 18] = -0.02
    dropped = rng.random(n) < 0.01
    fo[dropped, 4:8] *= -1.0
    whole = yields(fo, kind)
    pieces = np.concatenate([yields(np.ascontiguousarray(fo[a:a + 1000]), kind) for a in range(0, n, 1000)], axis=1)
    assert whole.max() > 0 and whole.tobytes() == np.ascontiguousarray(pieces).tobytes()
    cut = n // 2 + 3
    both = yields(None, kind, [np.ascontiguousarray(fo[:cut]), np.ascontiguousarray(fo[cut:])])
    assert both.tobytes() == whole.tobytes()


@pytest.mark.parametrize("kind", ["none", "ce", "14"])
@pytest.mark.parametrize("T", [(0.1, 0.6), (0.0005, 0.2)])
def test_arguments_off_the_tables(T, kind):
    """Pions above 0.27 GeV and every species in very cold cells leave the
    special-function tables; they are evaluated by a kernel of their own."""
    n = 3000
    fo = S.viscous_3d(n, seed=7).fo_surf().copy()
    fo[:, 13] = np.linspace(*T, n).astype(np.float32)
    whole = yields(fo, kind)
    pieces = np.concatenate([yields(np.ascontiguousarray(fo[a:a + 1000]), kind) for a in range(0, n, 1000)], axis=1)
    assert whole.max() > 0 and whole.tobytes() == np.ascontiguousarray(pieces).tobytes()
