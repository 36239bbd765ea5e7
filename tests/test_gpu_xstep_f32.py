"""The unbinned FP32 X-step where its work split changes: stream counts around
the 8-stream tiles (one unit with eight row groups, two with four, several
units, several parts), rows fewer than a step and more than a run, a
reference station (tiles without baselines), against the FP64 restatement.

Tolerance (relative L2 over all visibilities): as the block stage and windowed
FFT feeding it, FP32 rounding below 1e-6 (sums of at most 256 rows in
registers, then of those sums); twice that is allowed."""
import numpy as np
import pytest

from oracle import jobs
from sfxc_gpu import correlator, lib, scenario, synth


def make_job(streams, rows, ref=-1, pols=1, seed=7):
    rate, nchan = 32_000_000, 256
    st = scenario.cubic_stations(streams // pols, seed=seed, max_delay=1e-4, max_rate=1e-6)
    sc = scenario.Scenario(stations=st, pols=("R", "L")[:pols], sample_rate=rate, bandwidth=rate // 2, nchan=nchan,
                           integration_us=rows * nchan * 1_000_000 // rate, n_integrations=1, lead_us=1000, seed=seed,
                           block_bytes=2000, reference_station=ref)
    return scenario.build_job_bulk(sc)


@pytest.mark.gpu
@pytest.mark.parametrize("streams,rows,ref,pols", [(1, 5, -1, 1), (2, 700, -1, 1), (7, 33, -1, 1), (8, 300, -1, 1),
                                                   (9, 40, -1, 1), (16, 1100, -1, 2), (17, 64, -1, 1),
                                                   (24, 90, 3, 2), (33, 600, -1, 1), (42, 50, 20, 2)])
def test_fp32_xstep_shapes(streams, rows, ref, pols):
    j = make_job(streams, rows, ref, pols)
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    want = jobs.correlate(jj, impl="oracle", precision=64)["cor"]
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        got, _ = node.correlate(j)
    finally:
        node.close()
    (h0, v0), (h1, v1) = (correlator.split_output(x, j["number_channels"]) for x in (got, want))
    assert h0 == h1
    a, b = np.array(v0).astype(np.complex128), np.array(v1).astype(np.complex128)
    assert np.linalg.norm(a - b) < 2e-6 * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("streams,rows,ref", [(20, 600, -1), (35, 40, -1), (48, 300, -1), (65, 12, -1), (72, 300, 1),
                                              (100, 9, -1), (128, 5, 2)])
def test_fp32_xstep_wide(streams, rows, ref):
    """Five and six units in two row groups, parts that leave warps without a
    unit, steps of a single row (from 65 streams), up to 128 streams."""
    test_fp32_xstep_shapes(streams, rows, ref, 1)


@pytest.mark.gpu
def test_fp32_xstep_sum_rounding():
    """Rounding of long sums: autocorrelations of 1952 rows against FP64, root
    mean square over streams and channels.

    Two roundings a row of a partial sum that grows evenly, each 2.4e-8 of it in
    the root mean square: sqrt(2 x 128 / 3) of them in a run of 128 rows, averaged
    over 15 runs, 5.8e-8; the 15 runs' sums, sqrt(15 / 3) of them, 5.4e-8;
    accumulator and normalisation 4e-8; the transforms' fixed factors up to 7e-8:
    1.2e-7 in quadrature.  (Runs of 256 rows: 1.2e-7 by themselves.)"""
    rate, nchan = 32_000_000, 1024
    sc = scenario.Scenario(stations=scenario.cubic_stations(33, seed=2, max_delay=1e-4, max_rate=1e-6), sample_rate=rate,
                           bandwidth=rate // 2, nchan=nchan, integration_us=62500, n_integrations=1, lead_us=1000, seed=11,
                           block_bytes=2000)
    j = scenario.build_job_bulk(sc)
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    want = jobs.correlate(jj, impl="oracle", precision=64)["cor"]
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        got, _ = node.correlate(j)
    finally:
        node.close()
    a, b = (np.array(correlator.split_output(x, nchan)[1])[:33, 1:-1].real.astype(np.float64) for x in (got, want))
    rms = np.sqrt((((a - b) / b)**2).mean())
    assert rms < 1.2e-7


@pytest.mark.gpu
@pytest.mark.parametrize("streams,period", [(2, 8), (2, 3), (7, 4), (16, 4), (20, 2), (24, 5), (34, 2)])
def test_fp32_xstep_turning_products(streams, period):
    """A tone in every station, half of them at a fringe rate that turns its
    products with the others by 1 / period from row to row: they cancel, and the
    rounding of their sum has to be that of consecutive rows, whose partial sums
    stay at a few terms, whatever the work split.

    Relative to the sum of the terms' moduli: the transforms' 2e-7 a row, which
    differs from row to row, over 1950 rows 5e-9; two roundings a row of sums of
    up to period / pi terms, below 2e-9; 2e-8 is allowed.  (Sums over every
    period-th row grow to all their terms: 5e-8.)"""
    rate, nchan, rows, sky, tone = 32_000_000, 256, 1953, 1_600_000_000, 3_968_750
    r = rate / nchan / period / (sky + tone)  # seconds a second
    st = [scenario.Station("S%d" % k, k, synth.DelayPoly(coeffs=(0.0, r if k % 2 else 0.0), t0=36000.0))
          for k in range(streams)]
    sc = scenario.Scenario(stations=st, sample_rate=rate, bandwidth=rate // 2, nchan=nchan, channel_freq=sky,
                           integration_us=rows * nchan * 1_000_000 // rate, n_integrations=1, lead_us=1000, seed=1,
                           block_bytes=2000)

    def codes(k, nbytes):
        n = 4 * nbytes
        x = np.cos(2 * np.pi * tone / rate * np.arange(n)) + np.random.Generator(np.random.PCG64(k)).normal(size=n)
        return synth.pack_codes(synth.quantise(x, 2), 2)

    j = scenario.build_job_bulk(sc, codes=codes)
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    want = jobs.correlate(jj, impl="oracle", precision=64)["cor"]
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        got, _ = node.correlate(j)
    finally:
        node.close()
    a, b = (np.array(correlator.split_output(x, nchan)[1]).astype(np.complex128) for x in (got, want))
    ch = round(tone / (rate / 2 / nchan))
    assert np.argmax(b[0].real) in (ch - 1, ch, ch + 1)
    pairs = [(p, q) for p in range(streams) for q in range(p + 1, streams)]
    worst = 0.0
    for v, w, (p, q) in zip(a[streams:], b[streams:], pairs):
        if (p + q) % 2:
            moduli = np.sqrt(b[p].real * b[q].real)
            assert abs(w[ch]) < 0.05 * moduli[ch]  # the terms cancel
            worst = max(worst, abs(v[ch] - w[ch]) / moduli[ch])
    assert worst < 2e-8, worst
