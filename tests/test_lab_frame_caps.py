"""Caps of the lab-frame sampler's proposals at the top of their range: within
128 of 2^31 the proposals of a cell must still be counted in integers that hold
them.  A hadron of one static cell is the first accepted proposal of its stream
whatever the cap, so the largest caps give the hadrons of a small one."""
import numpy as np
import pytest

from test_lab_frame_warp import sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lcc", [0, 1])
def test_largest_caps(lcc):
    s, ref, off = sample(local_charge_conservation=lcc, gpu_max_tries=1000)
    tries = s.timings()["n_tries"]
    assert len(ref) > 100 and s.timings()["n_cell_redraws"] > 0
    for cap in (2**31 - 1, 2**31 - 2, 2**31 - 127, 2**31 - 128, 2**31 - 129):
        s, had, o = sample(local_charge_conservation=lcc, gpu_max_tries=cap)
        assert had.tobytes() == ref.tobytes() and np.array_equal(o, off), cap
        assert s.timings()["n_tries"] == tries and s.timings()["n_cell_redraws"] == 0
