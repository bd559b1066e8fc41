"""The network's gradient across the tile edges of its kernels. A block-diagonal union of K
copies of one LP has that LP's loss and gradient (both losses are means over nodes, the
copies' features and activations are the same), and with K a power of two every dz is
scaled exactly, so the bf16 operands round alike: what is left is the order of fp32 sums
over up to 64 x 17 nodes, about sqrt(1088) 2^-24 per sum and eight layers of them: 2e-5.
17 K and 15 K nodes cross the steps of 16, the stages of 64 and the tiles of 128 nodes, and
the heads' 8 rows a warp, at a new remainder for every K."""
import numpy as np
import pytest

import gnn_oracle as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 2, 4, 8, 16, 32, 64])
def test_gradient_of_copies(engine, instances, copies):
    one = instances.lp_uniform(32, 15, 17, 3)
    rng = np.random.default_rng(15)
    xt, yt = rng.uniform(0, 10, 17), rng.standard_normal(15)
    net = engine.Gnn(seed=11, y_scale=1.5)
    ref = G.forward_backward(net.parameters().astype(np.float64), one, xt, yt, ys=1.5)
    union, _, _ = engine.block_diagonal([one] * copies)
    A = engine.Matrix.from_instance(union)
    loss, grad = net.gradient(A, union, np.tile(xt, copies), np.tile(yt, copies))
    assert abs(loss - ref["loss"]) <= 2e-5 * ref["loss"]
    off = 0
    for name, shape in G.param_shapes():
        k = int(np.prod(shape))
        a, b = grad[off:off + k], ref["grad"][off:off + k]
        off += k
        assert np.linalg.norm(a - b) <= 2e-5 * max(np.linalg.norm(b), 1e-6), name
    x, y = net.predict(A, union)
    assert np.array_equal(x, np.tile(x[:17], copies)) and np.array_equal(y, np.tile(y[:15], copies))
