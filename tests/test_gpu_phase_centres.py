"""Extra phase centres where the work of a sub-integration's dump splits: centres
around a batch of five, channels below and past a CTA's 2048.  With one
sub-integration per integration a centre's cross visibilities are the first
centre's times one amplitude and a phase linear in the channel (its value is
checked against the reference's output in the fixture tests), and its
autocorrelations are the first centre's.

Tolerance: both visibilities and the factor are rounded to FP32, products and
their sum add four more roundings of 6e-8, so a ratio departs from the line by
at most 5e-7; twice that is allowed for the line's fit."""
import numpy as np
import pytest

from sfxc_gpu import correlator, lib, scenario


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,centres", [(256, 2), (2048, 6), (2048, 7), (4096, 12)])
def test_linear_phase(nchan, centres):
    rate, rows = 32_000_000, 24
    us = rows * nchan * 1_000_000 // rate
    st = scenario.cubic_stations(3, seed=centres, max_delay=1e-4, max_rate=1e-6)
    rng = np.random.Generator(np.random.PCG64(nchan))
    extra = [("PC%d" % k, list(rng.uniform(-3e-7, 3e-7, size=3))) for k in range(1, centres)]
    sc = scenario.Scenario(stations=st, pols=("R",), sample_rate=rate, bandwidth=rate // 2, nchan=nchan,
                           integration_us=us, n_integrations=1, sub_integration_us=us, lead_us=1000, seed=1,
                           block_bytes=2000, rho=0.3, extra_centers=extra)
    j = scenario.build_job_bulk(sc)
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        outs, _ = node.correlate(j)
    finally:
        node.close()
    _, v = correlator.split_output(outs, nchan)
    v = np.array(v).astype(np.complex128).reshape(centres, -1, nchan + 1)
    assert v.shape[1] == 6
    k = np.arange(nchan + 1)
    for c in range(1, centres):
        for b in range(6):
            r = v[c, b, 1:-1] / v[0, b, 1:-1]
            if np.array_equal(v[c, b], v[0, b]):
                continue  # an autocorrelation
            line = np.polyfit(k[1:-1], np.unwrap(np.angle(r)), 1)
            fit = np.abs(r).mean() * np.exp(1j * np.polyval(line, k[1:-1]))
            assert np.abs(r - fit).max() < 1e-6 * np.abs(fit).max()
        assert sum(np.array_equal(v[c, b], v[0, b]) for b in range(6)) == 3
