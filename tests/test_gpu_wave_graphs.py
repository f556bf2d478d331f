"""Engines that run in several waves share one graph between runs with other photons,
seeds and buffers, queued without waits: every run uses its own parameters."""
import numpy as np
import pytest

from gpu_optical_photons_b200 import params as P
from gpu_optical_photons_b200.wavefront import WaveConfig, WavefrontEngine

pytestmark = pytest.mark.gpu

TC = P.TallyConfig(100, 50.0, 10)
SEVERAL_WAVES = [dict(cadence=4), dict(wave_quota=300), dict(tail_steps=2)]


@pytest.mark.parametrize("cfg", SEVERAL_WAVES, ids=str)
def test_queued_ranges_add_up(engine, oracle, cfg):
    """Ranges of one batch queued one behind another, no wait between them."""
    events = [P.config2()[0].replace(seed=50 + i, abs_length=300.0 + 100.0 * i) for i in range(5)]
    counts = [4000, 1, 0, 2500, 9999]
    n = sum(counts)
    eng = WavefrontEngine(TC, 5, n, WaveConfig(math="exact", **cfg))
    eng.set_events(events, counts, first_id=3)
    for lo, hi in ((0, 1), (1, 4001), (4001, 4001), (4001, 12000), (12000, n)):
        eng.run_tally_range(lo, hi, accumulate=lo > 0)
    got = eng.tallies()
    eng.close()
    arr = (P.CSimParams * 5)(*[e.to_c() for e in events])
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    assert np.array_equal(got, oracle.batch_tally(arr, offs + np.uint64(3), TC, mode=oracle.PORTABLE))


@pytest.mark.parametrize("cfg", SEVERAL_WAVES, ids=str)
def test_new_photons_and_seeds_on_every_run(engine, oracle, cfg):
    eng = WavefrontEngine(TC, 1, 6000, WaveConfig(math="exact", **cfg))
    for i in range(4):
        p, n = P.config2()[0].replace(seed=i + 1, scat_length=300.0 + 50.0 * i), 6000 - 1777 * i
        out, st, _ = eng.run_batch([p], [n], first_id=10**6 * i)
        assert st["launches"] > 1
        assert np.array_equal(out[0], oracle.tally(p, TC, n, 10**6 * i, mode=oracle.PORTABLE)), i
    eng.close()


def test_event_records_of_new_photons(engine, oracle):
    for i in range(3):
        p = P.config2()[0].replace(seed=i + 1)
        rec, _, st = engine.run_gpu_records_event(p, 3000 + i, 3, first_id=10**6 * i, math="exact", chunk=1300)
        ref = oracle.records(p, 3000 + i, 10**6 * i, mode=oracle.PORTABLE)
        for k in oracle.Records.FIELDS:
            assert np.array_equal(np.asarray(rec[k]).view(np.uint8), np.asarray(ref[k]).view(np.uint8)), (i, k)
