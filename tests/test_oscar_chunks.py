"""OSCAR text made on the GPU in 8 MB chunks of lines (32,640 lines): chunks that
end inside an event, events longer than a chunk, events without hadrons, blocks
of 32 lines that span events; the bytes are those of the host's printf writer,
also when a handle writes again, longer or shorter."""
import numpy as np
import pytest

from iss_gb300 import iSS, native, surfaces as S

pytestmark = pytest.mark.gpu

PARAMS = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, include_deltaf_shear=1,
              include_deltaf_bulk=1, bulk_deltaf_kind=11, turn_on_bulk=1, quantum_statistics=1)


def written(s, path, host):
    s.setVal("gpu_oscar_on_host", int(host))
    s.write_output(native.OUTPUT_OSCAR, str(path))
    return path.read_bytes()


def test_chunks_of_lines_equal_the_host_writer(tmp_path):
    s = iSS(".", inputfile="")
    s.set_params(**dict(PARAMS, number_of_repeated_sampling=1))
    # events of some 35,000 hadrons; hundreds of events of a few; events of which
    # most are empty; a short file again
    for cells, events in ((160_000, 3), (60, 700), (1, 900), (160_000, 1), (900, 5)):
        s.set_params(number_of_repeated_sampling=events)
        s.set_surface(S.viscous_3d(cells, seed=cells).fo_surf())
        s.set_random_seed(events)
        s.generate_samples()
        n = np.diff(s.event_offsets())
        assert n.max() > 32_640 or events != 3
        assert (n == 0).any() or cells != 1
        assert written(s, tmp_path / "gpu", False) == written(s, tmp_path / "host", True), (cells, events)
