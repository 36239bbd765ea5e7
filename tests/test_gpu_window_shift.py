"""The windowed FFT of streams whose channels are shifted against the job's or cover
part of its band (stations at twice or half the job's rate), at the lengths of one
pair (8192 points) and of one stream (16384 points) a CTA and the one below, in
both spectra layouts, against the FP64 restatement.  Tolerances as in
test_gpu_window_fft."""
import numpy as np
import pytest

from sfxc_gpu import scenario
from test_gpu_window_fft import check

RATE = 32_000_000


def make_job(nchan, modes, rows=8, seed=5):
    """Five stations; modes: {station: (rate factor, bits, band start - the job's, in job bandwidths)}."""
    bw = RATE // 2
    st = scenario.cubic_stations(5, seed=seed, max_delay=2e-4, max_rate=3e-6)
    sc = scenario.Scenario(stations=st, sample_rate=RATE, bandwidth=bw, nchan=nchan,
                           integration_us=rows * nchan * 1_000_000 // RATE, n_integrations=1, lead_us=1000, seed=seed,
                           block_bytes=2000,
                           station_modes={k: (int(f * RATE), bits, int(off * bw)) for k, (f, bits, off) in modes.items()})
    return scenario.build_job_bulk(sc)


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,modes", [
    # 4096 channels: 8192 points with the job's band in the lower, upper or middle half of the station's
    (4096, {1: (2, 2, 0), 2: (2, 2, -1), 4: (2, 2, -0.5)}),
    # 8192 channels: 16384 points likewise, and 4096 over half of the band
    (8192, {0: (2, 2, -1), 1: (2, 2, 0), 3: (2, 2, -0.25), 4: (0.5, 1, 0.5)}),
    # 16384 channels: 8192 points over half of the band
    (16384, {1: (0.5, 2, 0), 2: (0.5, 2, 0.5), 4: (0.5, 1, 0.25)}),
])
def test_shifted_streams(nchan, modes):
    check(make_job(nchan, modes))
