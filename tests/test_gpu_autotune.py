"""The autotuner's plans are kept per job shape and spectra layout: the windowed FFT's
kernels for the FP32 and the tensor-core layout take different numbers of streams
and rows per CTA, so a plan timed on one says nothing of the other."""
import pytest

from sfxc_gpu import correlator, lib, scenario


@pytest.mark.gpu
def test_plans_of_both_layouts(sfxc_lib):
    rate, nchan, streams = 32_000_000, 1024, 11
    sc = scenario.Scenario(stations=scenario.cubic_stations(streams, seed=3, max_delay=1e-4, max_rate=1e-6),
                           sample_rate=rate, bandwidth=rate // 2, nchan=nchan, integration_us=50 * nchan * 1_000_000 // rate,
                           n_integrations=1, lead_us=1000, seed=2, block_bytes=2000)
    j = scenario.build_job_bulk(sc)
    plans = []
    for mode in (lib.X_FP32, lib.X_TC_HILO):
        node = correlator.CorrelatorNode(0, mode)
        try:
            node.correlate(j)
            node.autotune(1)
        finally:
            node.close()
        plans.append({e[:4] for e in correlator.plan_cache() if e[0] == 1 and e[1:3] == (2 * nchan, streams)})
    assert len(plans[0]) == 1 and plans[0] < plans[1] and len(plans[1]) == 2
