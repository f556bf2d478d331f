"""Event-records calls of different sizes share an engine: records and statistics are
those of a call with an engine of its own size."""
import numpy as np
import pytest

from gpu_optical_photons_b200 import _lib
from gpu_optical_photons_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 8, 10_000])
def test_event_records_of_several_sizes(engine, oracle, k):
    p = P.config2()[0]
    sizes = [65_537, 300, 65_536, 131_072, 1, 90_001]
    shared = [engine.run_gpu_records_event(p, n, k, first_id=n, math="exact") for n in sizes]
    for n, (rec, st, _) in zip(sizes, shared):
        ref = oracle.records(p, n, n, mode=oracle.PORTABLE)
        for f in oracle.Records.FIELDS:
            assert np.array_equal(np.asarray(rec[f]).view(np.uint8), np.asarray(ref[f]).view(np.uint8)), (n, f)
        steps = ref["n_boundary"].astype(np.int64) + ref["n_scatter"] + (ref["fate"] == P.ABSORBED_BULK)
        assert st["useful_lane_steps"] == int(steps.sum())
        assert _lib.lib().optx_release_cache() == 0  # an engine of its own
        _, alone, _ = engine.run_gpu_records_event(p, n, k, first_id=n, math="exact")
        assert {f: st[f] for f in ("launches", "useful_lane_steps", "spills")} == \
               {f: alone[f] for f in ("launches", "useful_lane_steps", "spills")}, n
