"""The inspection calls around a change of the job: before any integration, for
a stream that the last integration did not have, and with more streams or
input in place than that integration had."""
import numpy as np
import pytest

from sfxc_gpu import correlator, lib, scenario

pytestmark = pytest.mark.gpu

RATE, NCHAN, ROWS = 32_000_000, 256, 20


def make_job(stations, rows=ROWS):
    sc = scenario.Scenario(stations=scenario.cubic_stations(stations, seed=4, max_delay=1e-4, max_rate=1e-6),
                           sample_rate=RATE, bandwidth=RATE // 2, nchan=NCHAN,
                           integration_us=rows * NCHAN * 1_000_000 // RATE, n_integrations=1, lead_us=1000, seed=9,
                           block_bytes=2000)
    return scenario.build_job_bulk(sc)


def refused(node, stream):
    for call in (node.spectra, node.spectra_noalloc):
        with pytest.raises(lib.SfxcError) as e:
            call(stream, ROWS, NCHAN)
        assert e.value.code == lib.ESTATE
    with pytest.raises(lib.SfxcError) as e:
        node.unpacked(stream, ROWS * NCHAN)
    assert e.value.code == lib.ESTATE


def test_streams_of_another_job(sfxc_lib):
    small, large = make_job(2), make_job(40)
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        node.set_parameters(small)
        refused(node, 0)  # nothing has run
        node.correlate(small)
        want = node.spectra(1, ROWS - 1, NCHAN)
        assert np.abs(want).max() > 0
        # the job of many streams is set, the last integration is still the small one's
        node.set_parameters(large)
        refused(node, 2)
        refused(node, 39)
        for k in range(3):  # (its kernels' error flag included: the calls clear and read it)
            assert np.array_equal(node.spectra(1, ROWS - 1, NCHAN), want)
            assert np.array_equal(node.spectra_noalloc(1, ROWS - 1, NCHAN), want)
        node.correlate(large)
        assert np.abs(node.spectra(39, ROWS - 1, NCHAN)).max() > 0
    finally:
        node.close()


def test_input_moved_by_the_next_push(sfxc_lib):
    job, longer = make_job(2), make_job(2, rows=40 * ROWS)
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        node.correlate(job)
        want, samples = node.spectra(0, ROWS - 1, NCHAN), node.unpacked(0, ROWS * NCHAN)
        assert np.abs(want).max() > 0 and np.abs(samples).max() == 7
        node.push_protocol(0, longer["protocols"][0][0])  # does not fit behind the first: the stream's buffer grows
        assert np.array_equal(node.spectra(0, ROWS - 1, NCHAN), want)
        assert np.array_equal(node.unpacked(0, ROWS * NCHAN), samples)
    finally:
        node.close()
