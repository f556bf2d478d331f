"""The branch-free quotients, roots, Fresnel decisions and box exit of the photon
step equal the IEEE operations they replace (tests/cuda/ieee_check.cu, built here
with nvcc, in the contraction of the FAST and of the EXACT kernels), and records
outside their range still take the IEEE path: same records as the oracle."""
import os
import subprocess

import numpy as np
import pytest

from gpu_optical_photons_b200 import build as B
from gpu_optical_photons_b200 import params as P

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("flags", [["-DOPTX_EXACT=0"], ["-DOPTX_EXACT=1", "-fmad=false"]], ids=["fast", "exact"])
def test_step_arithmetic_equals_ieee(engine, tmp_path, flags):
    exe = str(tmp_path / "ieee_check")
    subprocess.run([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "-I", B.CSRC, "-I", B.INCLUDE] + flags
                   + [os.path.join(HERE, "cuda", "ieee_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.count(" 0 mismatches") == 8, out.stdout


@pytest.mark.parametrize("kw", [
    dict(hx=1e-20, hy=1e-20, hz=1e-20, scat_length=3e-20, abs_length=1e-19),  # numerators near the subnormals
    dict(hx=1e16, hy=2e16, hz=1e16, abs_length=1e17),                         # above the ordinary sizes
    dict(n_scint=3000.0, n_det=2500.0),                                       # above the ordinary indices
    dict(src_x=1e15),                                                         # a source far outside the box
], ids=["tiny", "huge", "index", "far"])
def test_records_outside_the_ordinary_range(engine, oracle, kw):
    p = P.SimParams(n_det=1.5, surface=P.LAMBERTIAN).replace(**kw)
    ref = oracle.records(p, 2000, 5, mode=oracle.PORTABLE)
    rec, _ = engine.run_gpu_records(p, 2000, first_id=5, math="exact")
    dev = engine.records_to_numpy(engine.records_device(p, 2000, first_id=5, math="exact"))
    for k in oracle.Records.FIELDS:
        want = np.asarray(ref[k]).view(np.uint8)
        assert np.array_equal(np.asarray(rec[k]).view(np.uint8), want), k
        assert np.array_equal(np.asarray(dev[k]).view(np.uint8), want), k


def test_far_gensteps_equal_on_host_and_device_uploads(engine, oracle):
    from gpu_optical_photons_b200 import gensteps as G
    from gpu_optical_photons_b200.wavefront import WaveConfig, WavefrontEngine
    c = P.TallyConfig(100, 50.0, 10)
    ev = [P.SimParams(n_det=1.5, surface=P.LAMBERTIAN)] * 2
    g = G.as_gensteps([(0, 0, 0, 0, 1, 2, 3, 1, 3000, 0), (3e38, 1e30, 0, 0, 3e38, 1e30, 0, 1, 500, 1),
                       (-3e38, 0, 1, 0, -3e38, 0, 1, 0, 500, 1)])
    eng = WavefrontEngine(c, 2, 4000, WaveConfig(max_gensteps=3, math="exact"))
    eng.set_gensteps(ev, g)
    eng.run_tally()
    host = eng.tallies()
    eng.set_gensteps_device(ev, G.to_device(g))
    eng.run_tally()
    assert np.array_equal(host, eng.tallies())
    eng.close()
    assert np.array_equal(host, oracle.genstep_run(ev, g, c, mode=oracle.PORTABLE)[0])
