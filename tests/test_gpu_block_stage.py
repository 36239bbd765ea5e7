"""The block stage's unpacking where it can go wrong: pairs of 256-sample
blocks that span several records of the input protocol, invalid runs inside
them, integer-delay changes, block counts that leave the last group of four
part empty, 1- and 2-bit samples; visibilities against the FP64 restatement.

Tolerance (relative L2 over all visibilities): FP32 rounding in transforms of
8 + 9 or more radix-2 levels and FP32 phases of at most pi stay below 1e-6;
twice that is allowed."""
import numpy as np
import pytest

from oracle import jobs
from sfxc_gpu import correlator, lib, scenario, timebase


def make_job(bits, block_bytes, rows, invalid, nchan=256, seed=5):
    rate = 32_000_000
    st = scenario.cubic_stations(2, seed=seed, max_delay=2e-4, max_rate=3e-6)
    sc = scenario.Scenario(stations=st, pols=("R",), sample_rate=rate, bandwidth=rate // 2, nchan=nchan, bits=bits,
                           integration_us=rows * nchan * 1_000_000 // rate, n_integrations=1, lead_us=1000, seed=seed,
                           block_bytes=block_bytes)
    j = scenario.build_job_bulk(sc)
    rec0, start, tint, slice_samples = scenario.job_timing(sc)
    for k in range(2):
        raw = np.random.Generator(np.random.PCG64(sc.seed * 7919 + k)).integers(
            0, 256, size=scenario.bulk_stream_bytes(sc, k), dtype=np.uint8)
        spb = block_bytes * 8 // bits * timebase.ticks_per_sample(rate)
        blocks = [(rec0 + b * spb, raw[b * block_bytes:(b + 1) * block_bytes].tobytes(),
                   invalid if k == 0 and b % 5 == 2 else []) for b in range(len(raw) // block_bytes)]
        sl = [(start, start + tint, slice_samples, correlator.delay_list(j["del_bytes"][k], start, start + tint, rate, bits))]
        j["protocols"][k] = correlator.write_protocol(blocks, sl, rate, bits, sc.integration_us)
    return j


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [1, 2])
@pytest.mark.parametrize("block_bytes,rows,invalid", [(2000, 9, []), (64, 11, []), (40, 34, [(7, 9)]),
                                                      (2000, 131, [(100, 700), (900, 1)])])
def test_block_stage_unpacking(bits, block_bytes, rows, invalid):
    j = make_job(bits, block_bytes, rows, invalid)
    ref = jobs.correlate(j, impl="oracle", precision=64)["cor"]
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        cor, _ = node.correlate(j)
    finally:
        node.close()
    (h0, v0), (h1, v1) = (correlator.split_output(x, j["number_channels"]) for x in (cor, ref))
    assert h0 == h1
    a, b = np.array(v0).astype(np.complex128), np.array(v1).astype(np.complex128)
    assert np.linalg.norm(a - b) < 2e-6 * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [1, 2])
@pytest.mark.parametrize("block_bytes,rows,invalid", [(2000, 9, []), (40, 34, [(7, 9)]), (2000, 131, [(100, 700), (900, 1)])])
def test_unpacked_samples(bits, block_bytes, rows, invalid):
    """The samples themselves, bit for bit: the inspection call runs the block stage's own unpacking."""
    j = make_job(bits, block_bytes, rows, invalid)
    want = jobs.correlate(j, dump=True, impl="oracle")["unpacked"]
    node = correlator.CorrelatorNode(0, lib.X_FP32)
    try:
        node.correlate(j)
        for k in range(2):
            assert np.array_equal(node.unpacked(k, want[(0, k)].size), want[(0, k)])
            assert invalid == [] or k == 1 or (want[(0, k)] == 0).any()
    finally:
        node.close()
