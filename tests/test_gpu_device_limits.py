"""The device calls at their limits: they have no error word, so nothing may cut a
run short."""
import numpy as np
import pytest

from gpu_optical_photons_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 40_001])
def test_device_calls_have_no_iteration_cap(engine, oracle, monkeypatch, n):
    """The cap of the calls that can report it (set to one iteration here) does not
    reach the device calls: all photons run to their ends."""
    p, c = P.config2()[0], P.TallyConfig(100, 50.0, 10)
    monkeypatch.setenv("OPTX_TEST_FAULT", "watchdog")
    got = engine.tally_device(p, c, n, first_id=7, math="exact").cpu().numpy().astype(np.uint64)
    rec = engine.records_to_numpy(engine.records_device(p, n, first_id=7, math="exact"))
    assert np.array_equal(got, oracle.tally(p, c, n, 7, mode=oracle.PORTABLE))
    ref = oracle.records(p, n, 7, mode=oracle.PORTABLE)
    for k in oracle.Records.FIELDS:
        assert np.array_equal(np.asarray(rec[k]).view(np.uint8), np.asarray(ref[k]).view(np.uint8)), k
