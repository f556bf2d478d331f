"""Replays on engines of one warp per block with arrival-time windows up to the longest
accepted one: the score sums are those of a short window with the same weights."""
import numpy as np
import pytest
import torch

from gpu_optical_photons_b200 import params as P
from gpu_optical_photons_b200.adjoint import ResponseModel
from gpu_optical_photons_b200.wavefront import WaveConfig

pytestmark = pytest.mark.gpu

THETA = (1000.0, 700.0, 0.95, 4.0)
N = 30_001


@pytest.fixture(scope="module")
def short(engine):
    out = {}
    for math in ("fast", "exact"):
        m = ResponseModel(P.config2()[0], N, P.TallyConfig(100, 50.0, 1), config=WaveConfig(math=math))
        out[math] = m.replay(THETA, torch.full((101,), 0.5, dtype=torch.float64), 0.25), *m.score_moments(THETA)
        m.close()
    return out


# 28,529 bins is the longest window that the limit on one warp's shared memory accepts;
# from 28,341 on their weights did not fit there beside the warp's windows and pantry.
@pytest.mark.parametrize("bins,cfg", [(28_000, {}), (28_330, {}), (28_345, {}), (28_529, {}),
                                      (28_400, dict(cadence=5)), (28_400, dict(math="exact"))], ids=str)
def test_long_window_equals_short(engine, short, bins, cfg):
    want_grad, want_hist, want_jac = short[cfg.get("math", "fast")]
    m = ResponseModel(P.config2()[0], N, P.TallyConfig(bins, 50.0, 1), config=WaveConfig(block_size=32, **cfg))
    grad = m.replay(THETA, torch.full((bins + 1,), 0.5, dtype=torch.float64), 0.25)
    hist, jac = m.score_moments(THETA)
    m.close()
    # The same photons; FP64 sums of 3e4 terms in another order.
    assert np.allclose(grad, want_grad, rtol=1e-10, atol=1e-10)
    assert np.allclose(jac.sum(0), want_jac.sum(0), rtol=1e-10, atol=1e-10)
    assert hist.sum() == want_hist.sum()


def test_weights_are_read_bin_by_bin(engine):
    """Weights that differ from bin to bin: long windows against the sum over moments."""
    bins = 28_400
    m = ResponseModel(P.config2()[0], N, P.TallyConfig(bins, 50.0, 1), config=WaveConfig(block_size=32))
    w = torch.linspace(-1.0, 2.0, bins + 1, dtype=torch.float64)
    grad = m.replay(THETA, w, 0.25)
    _, jac = m.score_moments(THETA)
    m.close()
    want = ((w.numpy() + 0.25)[:, None] * np.asarray(jac)).sum(0)
    assert np.allclose(grad, want, rtol=1e-10, atol=1e-10)
