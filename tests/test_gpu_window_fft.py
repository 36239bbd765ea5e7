"""The windowed FFT at the edges of its dispatch: every transform length, both
spectra layouts, stream counts that leave groups of two or four part empty,
rows that leave the last group or run part empty, every window and a
lower-sideband station, against the FP64 restatement.

Tolerances (relative L2 over all visibilities of a job): FP32 rounding in
transforms of 8 + 15 radix-2 levels, each adding about half a unit (6e-8) in
quadrature, and FP32 phases of up to 2 pi (2.4e-7) stay below 1e-6; twice that
is allowed.  The FP16 hi + lo form carries 22 bits of each spectrum value and
sums a run of rows in the tensor cores' FP32 accumulators, 1e-5."""
import numpy as np
import pytest

from oracle import jobs
from sfxc_gpu import correlator, lib, scenario

NONE, RECT, COS, HAMMING, HANN = range(5)


def make_job(nchan, stations, pols, rows, window=HANN, lsb=False, seed=3):
    rate = 32_000_000
    st = scenario.cubic_stations(stations, seed=seed, max_delay=2e-4, max_rate=3e-6)
    sc = scenario.Scenario(stations=st, pols=("R", "L")[:pols], sample_rate=rate, bandwidth=rate // 2, nchan=nchan,
                           window=window, integration_us=rows * nchan * 1_000_000 // rate, n_integrations=1,
                           lead_us=1000, seed=seed, block_bytes=2000,
                           station_sidebands={st[-1].number: "L"} if lsb else {})
    j = scenario.build_job_bulk(sc)
    if lsb:  # the same sky band recorded from its upper edge down
        j["streams"] = [s[:3] + (s[3] + sc.bandwidth,) + s[4:5] + ("L",) + s[6:] if s[0] == st[-1].number else s
                        for s in j["streams"]]
    return j


def vis(j, cor):
    _, v = correlator.split_output(cor, j["number_channels"])
    return np.array(v).astype(np.complex128)


def check(j, modes=(lib.X_FP32, lib.X_TC_HILO)):
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    ref = vis(j, jobs.correlate(jj, impl="oracle", precision=64)["cor"])
    for mode in modes:
        node = correlator.CorrelatorNode(0, mode)
        try:
            got = vis(j, node.correlate(j)[0])
        finally:
            node.close()
        err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
        assert err < (2e-6 if mode == lib.X_FP32 else 1e-5), (mode, err)


@pytest.mark.gpu
@pytest.mark.parametrize("nchan", [256, 512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("stations,pols,rows", [(2, 1, 3), (5, 1, 18), (3, 2, 33)])
def test_lengths_and_ragged_groups(nchan, stations, pols, rows):
    check(make_job(nchan, stations, pols, rows))


@pytest.mark.gpu
@pytest.mark.parametrize("nchan", [256, 2048, 4096])
@pytest.mark.parametrize("window,lsb", [(NONE, False), (RECT, False), (COS, True), (HAMMING, True)])
def test_windows_and_sidebands(nchan, window, lsb):
    check(make_job(nchan, 3, 1, 21, window=window, lsb=lsb))
