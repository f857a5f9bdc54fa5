"""The lab-frame sampler (MC_sampling = 2) gives each hadron to a warp, whose
32 lanes make 32 consecutive proposals: the hadron must be the first accepted
proposal of its stream, whatever the number of proposals per cell.

One static cell without delta f, where the emission function is E f0(E):
* against a FP64 restatement of the proposals on the same Philox counters;
* a redrawn hadron of a one-cell surface gets the same cell again and its
  proposal counter runs on, so caps below, at and above a warp's width and the
  default give the same hadrons bit for bit, pairs of local charge
  conservation included."""
import numpy as np
import pytest

import oracle_lib as O
from iss_gb300 import iSS, surfaces as S

pytestmark = pytest.mark.gpu

T, PT_MAX, Y_RANGE, SEED = 0.150, 3.6943142, 3.0, 77
TAG_EFA = 8


def cell():
    c = np.zeros((1, 34), dtype=np.float32)
    c[0, 0], c[0, 4], c[0, 8] = 10.0, 40.0, 1.0
    c[0, 12], c[0, 13], c[0, 14] = 0.25, T, 0.04
    return c


def sample(**extra):
    s = iSS(".", inputfile="")
    p = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=0,
             include_deltaf_bulk=0, quantum_statistics=1, number_of_repeated_sampling=6, MC_sampling=2,
             restrict_deltaf=1, deltaf_max_ratio=1.0, sample_pT_up_to=-1, sample_y_minus_eta_s_range=Y_RANGE,
             gpu_max_redraws=1000000)
    p.update(extra)
    s.set_params(**p)
    s.set_surface(cell())
    s.set_random_seed(SEED)
    s.generate_samples()
    had, off = s.all_hadrons()
    return s, had, off


def philox(c0, c1, c2, c3, k0, k1):
    c = [np.broadcast_to(np.asarray(v, dtype=np.uint64), np.shape(c0)).copy() for v in (c0, c1, c2, c3)]
    m = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [(v >> np.uint64(9)).astype(np.float64) / 2.0 ** 23 for v in c]


def first_accepted(m, sign, s, e, i):
    """pT, phi, y of the hadron i of species s (sorted order) in event e."""
    E = np.linspace(m, m + 30 * T, 200001)
    top = (E / (np.exp(E / T) + sign)).max()
    for t0 in range(0, 4_000_000, 16384):
        t = np.arange(t0, t0 + 16384)
        a, b, c, d = philox(t, i, e, s | (TAG_EFA << 16), SEED, 0)
        pT, phi, y = PT_MAX * np.sqrt(a), 2 * np.pi * b, (1 - 2 * c) * Y_RANGE
        p0 = np.sqrt(m * m + pT * pT) * np.cosh(y)
        ok = np.flatnonzero(d < p0 / (np.exp(p0 / T) + sign) / top)
        if len(ok):
            return pT[ok[0]], phi[ok[0]], y[ok[0]]
    raise AssertionError("no proposal accepted")


def test_first_accepted_proposal():
    s, had, off = sample()
    cnt = s.counts()
    sp = O.chosen_species(S.TABLE_DIR, 0)
    at, n = 0, 0
    for e in range(cnt.shape[0]):
        for k in range(cnt.shape[1]):
            for i in range(cnt[e, k]):
                h = had[at]
                at += 1
                if e >= 3 and i == 0:
                    continue
                n += 1
                m = float(h["mass"])
                pT, phi, y = first_accepted(m, int(sp["sign"][k]), k, e, i)
                mT = np.hypot(m, pT)
                want = np.array([mT * np.cosh(y), pT * np.cos(phi), pT * np.sin(phi), mT * np.sinh(y)])
                got = np.array([h["E"], h["px"], h["py"], h["pz"]], dtype=np.float64)
                # the sine of an angle up to 2 pi in FP32 is good to about
                # 1e-6, the hyperbolic functions to a few 1e-7; FP32 rounding
                # of the acceptance (some 1e-6) flips about one decision in
                # 1e5 hadrons
                assert np.abs(got - want).max() < 2e-5 * want[0], (e, k, i)
    assert n >= 100


@pytest.mark.parametrize("lcc", [0, 1])
def test_any_cap_gives_the_same_hadrons(lcc):
    s, ref, off = sample(local_charge_conservation=lcc)
    tries = s.timings()["n_tries"]
    assert len(ref) > 100
    for cap in (1, 31, 32, 33, 127, 128, 129, 1000):
        s, had, o = sample(local_charge_conservation=lcc, gpu_max_tries=cap)
        assert had.tobytes() == ref.tobytes() and np.array_equal(o, off), cap
        assert s.timings()["n_tries"] == tries
        assert cap > 1000 or s.timings()["n_cell_redraws"] > 0


@pytest.mark.parametrize("density,bulk", [(0, 0), (1, 0), (0, 1)])
def test_bulk_rejection_changes_nothing(density, bulk):
    """The bound that rejects proposals in bulk scales with the cap of delta f: a
    cap of 1e6 rejects none.  Where |delta f| stays below 1 anyway (shear and
    bulk scaled down a thousandfold) the cap itself changes nothing, so both
    must sample the same hadrons: moving and space-like cells, bosons and
    fermions, with and without chemical potentials."""
    make = S.finite_density_3d if density else S.viscous_3d
    fo = make(700, seed=14).fo_surf()
    fo[:, 19:30] *= 1e-3
    ref = None
    for cap in (1.0, 1e6):
        s = iSS(".", inputfile="")
        s.set_params(**dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=2 if density else 0,
                            include_deltaf_shear=1, include_deltaf_bulk=bulk, bulk_deltaf_kind=1,
                            quantum_statistics=1, number_of_repeated_sampling=20, MC_sampling=2,
                            restrict_deltaf=1, deltaf_max_ratio=cap, sample_pT_up_to=-1,
                            sample_y_minus_eta_s_range=Y_RANGE))
        s.set_surface(fo)
        s.set_random_seed(8)
        s.generate_samples()
        had = s.all_hadrons()[0].copy()
        tries = s.timings()["n_tries"]
        assert len(had) > 500
        if ref is None:
            ref, ref_tries = had, tries
    assert had.tobytes() == ref.tobytes() and tries == ref_tries
