"""The network's calls give large buffers back to the device: training data and prediction buffers do not stay in the
library's pool.  Answers are the same on both sides of the line (64 MB a buffer)."""
import numpy as np
import pytest
import torch

from pramana_b200.mlp import MlpNetwork, TrainOptions

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def net():
    return MlpNetwork([64, 64, 8], max_batch=8192, seed=3)


def test_prediction_gives_memory_back(net):
    x = np.random.default_rng(95).standard_normal((1 << 20, 64)).astype(np.float32)  # 256 MB
    net.forward(x[:100])
    before = _free()
    y = net.forward(x)
    assert before - _free() < 64 * MB
    line = 64 * MB // (64 * 4)  # rows of the largest pooled input
    for rows in (line, line + 1):
        assert np.array_equal(net.forward(x[:rows]), y[:rows])


def test_training_gives_memory_back(net):
    rng = np.random.default_rng(96)
    x = rng.standard_normal((1 << 20, 64)).astype(np.float32)
    t = rng.standard_normal((1 << 20, 8)).astype(np.float32)
    net.train(x[:8192], t[:8192], TrainOptions(epochs=1, batch=8192))
    before = _free()
    losses = net.train(x, t, TrainOptions(epochs=1, batch=8192))
    assert np.isfinite(losses).all() and before - _free() < 64 * MB
