"""Tallies that run the history kernel (one thread per photon): histograms that leave
the wave kernel's pantries no room in shared memory (with 100 time bins from 184 x 184
hit-map bins on; tests/cuda/host_check.cpp pins that line), and device calls of more
photons than the wave kernel counts. 183 x 183 bins are the wave kernel's largest."""
import numpy as np
import pytest
import torch

from gpu_optical_photons_b200 import params as P

pytestmark = pytest.mark.gpu

PARITY = {
    "cube": P.config1()[0],
    "lambert": P.config2()[0],
    "bar": P.config3()[0],
    "mixed": P.SimParams(scat_length=600.0, source=P.VOLUME,
                         face_surface=[P.LAMBERTIAN, P.POLISHED, P.SPECULAR, P.BLACK, P.LAMBERTIAN, 0],
                         face_reflectivity=[0.9, 0.95, 0.97, 0.5, 0.85, 0.0]),
    "no_steps": P.config2()[0].replace(max_steps=0),
    "tiny": P.SimParams(hx=1e-20, hy=1e-20, hz=1e-20, scat_length=3e-20, abs_length=1e-19, n_det=1.5,
                        surface=P.LAMBERTIAN),  # outside the branch-free arithmetic's range
}


def both(engine, p, c, n, first_id, math, block):
    """The host call's tally and the device call's, which adds to a buffer of ones."""
    _, flat, _ = engine.run_gpu_tally(p, c, n, first_id=first_id, math=math, block_size=block)
    out = torch.ones(c.length, dtype=torch.int64, device="cuda")
    engine.tally_device(p, c, n, first_id=first_id, out=out, math=math, block_size=block)
    return flat, (out.cpu().numpy() - 1).astype(np.uint64)


# 148 SMs x 256 threads: up to 37,888 photons a thread runs one, beyond it several.
@pytest.mark.parametrize("n,block", [(1, 256), (33, 32), (37_888, 256), (37_889, 256), (9_473, 64), (152_000, 1024),
                                     (400_003, 256)])
@pytest.mark.parametrize("xy", [183, 184, 236])
def test_wide_tally_equals_oracle(engine, oracle, xy, n, block):
    p, c = P.config2()[0], P.TallyConfig(100, 50.0, xy)
    want = oracle.tally(p, c, n, 2**33 + 5, mode=oracle.PORTABLE)
    for got in both(engine, p, c, n, 2**33 + 5, "exact", block):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("name", sorted(PARITY))
def test_wide_tally_of_every_setup_equals_oracle(engine, oracle, name):
    p, c = PARITY[name], P.TallyConfig(500, 50.0, 200)
    want = oracle.tally(p, c, 100_000, 11, mode=oracle.PORTABLE)
    for got in both(engine, p, c, 100_000, 11, "exact", 256):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("math", ["fast", "approx"])
@pytest.mark.parametrize("name", ["cube", "lambert", "bar"])
def test_history_and_wave_kernel_run_the_same_photons(engine, name, math):
    """Fates, arrival times and step sums do not depend on the hit map's bins, so not on
    the kernel either; nor does the tally depend on the block size."""
    p, n = PARITY[name], 300_000
    _, narrow, _ = engine.run_gpu_tally(p, P.TallyConfig(100, 50.0, 10), n, first_id=3, math=math)
    c = P.TallyConfig(100, 50.0, 200)
    wide = [t for block in (32, 64, 256, 512, 1024) for t in both(engine, p, c, n, 3, math, block)]
    for t in wide:
        assert np.array_equal(t, wide[0])
        assert np.array_equal(t[:106], narrow[:106]) and np.array_equal(t[-2:], narrow[-2:])
    assert wide[0][106:-2].sum() == narrow[106:-2].sum()


def test_device_tally_beyond_the_wave_kernels_count(engine):
    """2^32 - 65535 photons in one call (history kernel) are 2^32 - 65536 (wave kernel) and
    the last one."""
    p, c, n = P.config1()[0], P.TallyConfig(100, 50.0, 10), 2**32 - 65536
    whole = engine.tally_device(p, c, n + 1, first_id=17)
    parts = engine.tally_device(p, c, n, first_id=17)
    engine.tally_device(p, c, 1, first_id=17 + n, out=parts)
    assert torch.equal(whole, parts)
    assert int(whole[:5].sum()) == n + 1
