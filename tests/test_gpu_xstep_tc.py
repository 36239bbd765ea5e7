"""The tensor-core X-step kernels where their work changes shape: the TMA-fed one
over every number of slot quads; the row-gathered one with runs of rows shorter
and longer than a tile, empty bins, bins dealt in one and in several parts,
channel counts that leave a group of four part empty, both slot counts, and
unbinned from 33 to 64 streams, against the FP64 restatement.

Tolerance (relative L2 over all visibilities): the FP16 hi + lo form carries 22
bits of each spectrum value (relative error up to 2.4e-7) over FP32 transforms
(below 1e-6) and sums in the tensor cores' FP32 accumulators, 1e-5."""
import numpy as np
import pytest

from oracle import jobs
from sfxc_gpu import correlator, lib, scenario


def check(streams, rows, nbins=0, gate=(0.0, 1.0), nchan=256):
    rate = 32_000_000
    pols = 1 if streams % 2 else 2
    st = scenario.cubic_stations(streams // pols, seed=streams, max_delay=1e-4, max_rate=1e-6)
    sc = scenario.Scenario(stations=st, pols=("R", "L")[:pols], sample_rate=rate, bandwidth=rate // 2, nchan=nchan,
                           integration_us=rows * nchan * 1_000_000 // rate, n_integrations=1, lead_us=1000,
                           seed=streams, block_bytes=2000)
    j = scenario.build_job_bulk(sc)
    if nbins:
        j.update(scenario.pulsar_params(sc, nbins=nbins, gate=gate, period=2e-3, obs_freq=4800.0))
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    want = jobs.correlate(jj, impl="oracle", precision=64)["cor"]
    node = correlator.CorrelatorNode(0, lib.X_TC_HILO)
    try:
        got, _ = node.correlate(j)
    finally:
        node.close()
    (h0, v0), (h1, v1) = (correlator.split_output(x, j["number_channels"]) for x in (got, want))
    assert h0 == h1
    a, b = np.array(v0).astype(np.complex128), np.array(v1).astype(np.complex128)
    assert np.isfinite(a).all()
    assert np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("streams,rows", [(1, 5), (3, 64), (6, 65), (12, 40), (17, 200), (24, 33), (27, 130), (32, 71)])
def test_tma_fed(streams, rows):
    check(streams, rows)


@pytest.mark.gpu
@pytest.mark.parametrize("streams,rows", [(33, 7), (36, 300), (45, 33), (49, 64), (64, 97)])
def test_unbinned_rows_in_order(streams, rows):
    check(streams, rows)


@pytest.mark.gpu
@pytest.mark.parametrize("streams,rows,nbins,gate", [(1, 40, 3, (0.0, 1.0)), (6, 700, 2, (0.2, 0.9)),
                                                     (18, 500, 60, (0.0, 1.0)), (32, 260, 17, (0.3, 0.4)),
                                                     (33, 300, 9, (0.0, 1.0)), (40, 200, 70, (0.0, 0.5)),
                                                     (64, 90, 4, (0.0, 1.0))])
def test_binned(streams, rows, nbins, gate):
    check(streams, rows, nbins, gate)
