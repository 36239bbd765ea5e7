"""Every extra phase centre's visibilities against the FP64 restatement, each over
several sub-integrations: centre counts around the dump's batches of five,
channels below and past a CTA's 2048, and residual delays whose rates turn a
centre's phase by a good part of a turn from one sub-integration to the next, so
that another centre's or another sub-integration's phase, slope or amplitude
shows.

Tolerance (relative L2 over a centre's cross visibilities): the block stage's
FP32 phases of at most pi (2.4e-7) and FP32 rounding in transforms of 8 + 9 or
more radix-2 levels, for two streams, and the centre's FP32 factor and product
stay below 1e-6; twice that is allowed.  A phase that is wrong by 1e-5 turns
exceeds it."""
import numpy as np
import pytest

from oracle import jobs
from sfxc_gpu import correlator, lib, scenario, synth


def make_job(nchan, centres, subs, seed):
    rate, rows = 32_000_000, 16  # FFT rows of a sub-integration
    us = rows * nchan * 1_000_000 // rate
    st = scenario.cubic_stations(3, seed=seed, max_delay=1e-4, max_rate=1e-6)
    sc = scenario.Scenario(stations=st, pols=("R",), sample_rate=rate, bandwidth=rate // 2, nchan=nchan,
                           integration_us=subs * us, n_integrations=1, sub_integration_us=us, lead_us=1000, seed=seed,
                           block_bytes=2000, extra_centers=[("PC%d" % k, [0.0] * 3) for k in range(1, centres)])
    j = scenario.build_job_bulk(sc)
    rng = np.random.Generator(np.random.PCG64(seed))
    tables = []
    for s in st:
        scans = [("SRC", sc.mjd, sc.sec0 - 20, 140, s.poly)]
        for k in range(1, centres):
            c = list(s.poly.coeffs)
            c[0] += rng.uniform(-2e-6, 2e-6)
            c[1] += rng.uniform(-1.0, 1.0) / (sc.channel_freq * us * 1e-6)  # up to a turn a sub-integration
            scans.append(("PC%d" % k, sc.mjd, sc.sec0 - 20, 140, synth.DelayPoly(coeffs=tuple(c), t0=s.poly.t0)))
        tables.append(synth.del_file_bytes(s.name[:2], scans))
    j["del_bytes"] = tables
    return j


def vis(j, cor, centres):
    _, v = correlator.split_output(cor, j["number_channels"])
    return np.array(v).astype(np.complex128).reshape(centres, 6, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,centres,subs", [(256, 2, 3), (256, 6, 5), (512, 7, 3), (2048, 11, 3), (4096, 12, 2)])
def test_centres_against_restatement(nchan, centres, subs):
    j = make_job(nchan, centres, subs, seed=centres)
    jj = dict(j, protocols=[[bytes(p) for p in s] for s in j["protocols"]])
    want = vis(j, jobs.correlate(jj, impl="oracle", precision=64)["cor"], centres)
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        got = vis(j, node.correlate(j)[0], centres)
    finally:
        node.close()
    for c in range(centres):
        assert np.linalg.norm(got[c, :3] - want[c, :3]) < 2e-6 * np.linalg.norm(want[c, :3]), c
        for b in range(3, 6):
            n = np.linalg.norm(want[c, b])
            assert np.linalg.norm(got[c, b] - want[c, b]) < 2e-6 * n, (c, b)
            # (a centre's own: none of the other centres' comes near)
            assert min([np.linalg.norm(want[o, b] - want[c, b]) for o in range(centres) if o != c]) > 1e-3 * n
