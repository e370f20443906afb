"""The guide gradient of one 128-sample tile inside a large batch (needs a B200).

Samples of weight zero add exact zeros, so with weights in one tile only, a batch of any size must
return that tile's gradient, block by block: whether the tile is a block's first, second or third, or
the partial last one of the call. The weights are chosen so that every sample's weight over the batch
size rounds to the same float in both calls; the weight gradients then come from the same matrix
products and are equal, and the bias gradients differ by the order of four float sums.
"""

import numpy as np
import pytest

from oracle import guide_net as gn
from test_gpu_guiding import BOUNDS, make_samples

pytestmark = pytest.mark.gpu
SHAPES = [("W1", 64 * 80), ("b1", 64), ("W2", 64 * 64), ("b2", 64), ("W3", 64 * 64), ("b3", 64), ("W4", 32 * 64), ("b4", 32)]


@pytest.mark.parametrize("n,tile", [(129, 0), (129, 1), (148 * 128 + 1, 0), (148 * 128 + 1, 147), (148 * 128 + 1, 148),
                                    (2 * 148 * 128 + 77, 0), (2 * 148 * 128 + 77, 160), (2 * 148 * 128 + 77, 296)])
def test_one_tile_of_a_batch(renderer, n, tile):
    renderer.guide_set_params(gn.init_params(seed=6), BOUNDS)
    samples = make_samples(n, 23)
    first, last = 128 * tile, min(n, 128 * tile + 128)
    weights = np.zeros(n, np.float32)
    weights[first:last] = samples[first:last, 9] * np.float32(n)
    samples[:, 9] = weights
    alone = samples[np.resize(np.arange(first, last), 128)].copy()
    alone[:, 9] = 0.0
    alone[: last - first, 9] = (weights[first:last] * (np.float32(1.0) / np.float32(n))) * np.float32(128.0)
    grad, loss = renderer.guide_loss_grad(samples)
    want, want_loss = renderer.guide_loss_grad(alone)
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    at = 0
    for name, size in SHAPES:
        g, w = grad[at:at + size], want[at:at + size]
        at += size
        assert np.linalg.norm(w) > 0.0, name
        if name[0] == "W":
            assert np.array_equal(g, w), name
        else:
            assert np.linalg.norm(g - w) <= 1e-5 * np.linalg.norm(w), name
