"""Runs at the edges of the engine's work distribution (claims of 32 to 256 photons
by the run's size, the last photons of a run finished in place): tallies and records
equal the oracle's exactly, whatever the number of photons per warp."""
import numpy as np
import pytest

from gpu_optical_photons_b200 import params as P
from gpu_optical_photons_b200.wavefront import WaveConfig, WavefrontEngine

pytestmark = pytest.mark.gpu

TC = P.TallyConfig(100, 50.0, 10)
SETUPS = {"cube": P.config1, "lambert": P.config2, "bar": P.config3}


# 8 x 148 x 28 warps x 64 photons = 2,121,728: where claims grow from 32 to 64 photons.
@pytest.mark.parametrize("setup,n", [("cube", 1), ("cube", 31), ("lambert", 33), ("bar", 1000), ("lambert", 40_001),
                                     ("lambert", 2_121_727), ("lambert", 2_121_729)]
                         # one configuration's blocks of 384, 640, 768 and 896 threads (148 SMs)
                         + [("bar", 147), ("bar", 148), ("bar", 170_643), ("bar", 170_644)]
                         + [("bar", 56_979), ("bar", 56_980), ("cube", 227_475), ("cube", 227_476),
                            ("lambert", 568_467), ("lambert", 568_468), ("cube", 1_364_115), ("cube", 1_364_116)])
def test_tally_equals_oracle(engine, oracle, setup, n):
    p = SETUPS[setup]()[0]
    _, flat, _ = engine.run_gpu_tally(p, TC, n, first_id=9, math="exact")
    assert np.array_equal(flat, oracle.tally(p, TC, n, 9, mode=oracle.PORTABLE))


@pytest.mark.parametrize("max_steps", [0, 1, 2, 7, 10_000])
@pytest.mark.parametrize("setup", sorted(SETUPS))
def test_records_equal_oracle(engine, oracle, setup, max_steps):
    p = SETUPS[setup]()[0].replace(max_steps=max_steps)
    rec, _ = engine.run_gpu_records(p, 777, first_id=3, math="exact")
    ref = oracle.records(p, 777, 3, mode=oracle.PORTABLE)
    for k in oracle.Records.FIELDS:
        assert np.array_equal(np.asarray(rec[k]).view(np.uint8), np.asarray(ref[k]).view(np.uint8)), k


@pytest.mark.parametrize("cfg", [dict(), dict(blocks_per_sm=7, threshold=32), dict(tail_steps=3), dict(cadence=4),
                                 dict(chunk=4096), dict(use_graph=False)], ids=str)
def test_small_ragged_batch_equals_oracle(engine, oracle, cfg):
    """Events of 0 to 700 photons, one without steps, seeds that differ per event."""
    rng = np.random.default_rng(4)
    counts = rng.integers(0, 700, 23).astype(np.uint64)
    counts[[3, 7]] = 0, 1
    events = [P.SimParams(n_det=1.5, surface=P.LAMBERTIAN, abs_length=float(np.float32(rng.uniform(200, 3000))),
                          scat_length=float(np.float32(rng.uniform(300, 1000))), source=int(i % 2),
                          max_steps=0 if i == 5 else 10_000, seed=100 + i // 2) for i in range(23)]
    arr = (P.CSimParams * 23)(*[e.to_c() for e in events])
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    eng = WavefrontEngine(TC, 23, int(counts.sum()), WaveConfig(math="exact", **cfg))
    eng.set_events(events, counts)
    eng.run_tally()
    got = eng.tallies()
    eng.close()
    assert np.array_equal(got, oracle.batch_tally(arr, offs, TC, mode=oracle.PORTABLE))


# Device calls from one photon to several per thread (tallies whose histograms leave the
# wave kernel no room: test_gpu_wide_tallies.py).
@pytest.mark.parametrize("n,block,xy", [(1, 256, 10), (33, 32, 10), (9_473, 256, 50), (1, 256, 150), (9_473, 64, 150), (130_000, 256, 50), (152_000, 1024, 10), (152_000, 32, 100),
                                        (400_003, 256, 50), (400_003, 256, 150)])
def test_device_calls_equal_oracle(engine, oracle, n, block, xy):
    import torch
    p = P.config2()[0]
    c = P.TallyConfig(100, 50.0, xy)
    out = torch.ones(c.length, dtype=torch.int64, device="cuda")  # the call adds to it
    engine.tally_device(p, c, n, first_id=2**33 + 5, out=out, block_size=block, math="exact")
    want = oracle.tally(p, c, n, 2**33 + 5, mode=oracle.PORTABLE)
    assert np.array_equal(out.cpu().numpy() - 1, want.astype(np.int64))
    rec = engine.records_to_numpy(engine.records_device(p, n, first_id=2**33 + 5, block_size=block, math="exact"))
    ref = oracle.records(p, n, 2**33 + 5, mode=oracle.PORTABLE)
    for k in oracle.Records.FIELDS:
        assert np.array_equal(np.asarray(rec[k]).view(np.uint8), np.asarray(ref[k]).view(np.uint8)), k


def test_device_calls_overlap_on_streams(engine):
    """Launches in flight together on several streams share nothing."""
    import torch
    p, c = P.config1()[0], TC
    want = engine.run_gpu_tally(p, c, 600_000, first_id=1, math="fast")[1].astype(np.int64)
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [torch.zeros(c.length, dtype=torch.int64, device="cuda") for _ in streams]
    torch.cuda.synchronize()
    for i in range(3):
        for st, o in zip(streams, outs):
            engine.tally_device(p, c, 200_000, first_id=1 + 200_000 * i, out=o, stream=st)
    torch.cuda.synchronize()
    for o in outs:
        assert np.array_equal(o.cpu().numpy(), want)


def test_device_calls_of_different_sizes_from_threads(engine):
    """Launches of one kernel with different shared memory (blocks of 384 to 896 threads,
    different histograms), issued from several threads at once, none refused."""
    from concurrent.futures import ThreadPoolExecutor

    import torch
    p = P.config1()[0]
    jobs = [(n, P.TallyConfig(100, 50.0, xy)) for n in (50_000, 300_000, 900_000, 1_500_000) for xy in (10, 130, 160)]
    want = [engine.run_gpu_tally(p, c, n, first_id=1, math="fast")[1].astype(np.int64) for n, c in jobs]

    def run(job):
        n, c = job
        st, out = torch.cuda.Stream(), torch.zeros(c.length, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(40):
            engine.tally_device(p, c, n, first_id=1, out=out, stream=st)
        st.synchronize()
        return out.cpu().numpy()

    with ThreadPoolExecutor(len(jobs)) as pool:
        for got, w in zip(pool.map(run, jobs), want):
            assert np.array_equal(got, 40 * w)
