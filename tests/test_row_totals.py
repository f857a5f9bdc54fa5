"""Row totals of the fixed-point CDF: every yield y of a row is cut to
floor(y 2^s), s = 188 - L - exponent of the row's largest yield, L = ceil(log2 n),
and the total is the exact integer sum times 2^-s.  Restated here in integers
from the cells' yields, for sizes at the edges of a run (32 cells), a warp, a
tile (2,048 cells) and of the two splits of the sum (L below 16 and from 16 on),
and for yields so small or so large that one float does not hold the scale.
The comparison is exact."""
import numpy as np
import pytest

from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1,
              number_of_repeated_sampling=0)


def restated(y):
    n = y.size
    L = int(n - 1).bit_length()
    b = np.ascontiguousarray(y, dtype=np.float32).view(np.uint32).astype(np.int64)
    ex = max(int(b.max() >> 23), 1)
    base = 38 - L - ex
    e = b >> 23
    m = np.where(e > 0, (b & 0x7FFFFF) | 0x800000, b & 0x7FFFFF)
    sh = np.maximum(e, 1) + base
    q = np.where(sh >= 0, m << np.clip(sh, 0, 62), m >> np.clip(-sh, 0, 63))
    Q = sum(int(v) for v in np.add.reduceat(q, np.arange(0, n, 1024)))
    return float(np.ldexp(np.float64(Q), -(150 + base)))


@pytest.mark.parametrize("scale", [1.0, 1e-33, 1e33])
@pytest.mark.parametrize("n", [1, 31, 33, 512, 2047, 2048, 2049, 6001, 32768, 32769, 70003])
def test_totals_are_the_integer_sums(n, scale):
    fo = S.viscous_3d(n, seed=n).fo_surf().copy()
    fo[:, 4:8] *= np.float32(scale)
    s = iSS(".", inputfile="")
    s.set_params(**PARAMS)
    s.set_surface(fo)
    s.generate_samples()
    totals = s.species_yields()
    some = 0
    for k in range(len(totals)):
        y = s.cell_yields(k)
        if not y.any():
            assert totals[k] == 0.0
            continue
        some += 1
        assert totals[k] == restated(y), k
    assert some or n < 100
