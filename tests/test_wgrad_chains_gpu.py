"""Weight gradients of dense layers whose rows are several chunks of the
tensor-core kernel but only two of its slices (256 x 2304 outputs): no further
from the exact sums than running FP32 sums of the same rows.

The network is set so that the gradient of the first dense layer's output is
known: its weights are zero and its biases one, one unit of each later layer is
connected, and the prediction is zero.  A target then puts a chosen BF16 value
into a sample's output gradient, and the layer's gradients are sums over the
samples of known BF16 values."""
import numpy as np
import pytest

from oracle import nn_oracle as N

pytestmark = pytest.mark.gpu


def running_sums(dz, x):
    """Sums of dz[r][o] x[r][k] in FP32, row after row, in as many slices as a
    kernel of 32 x 32 outputs per CTA spreads 256 x 2304 outputs over."""
    n = len(dz)
    slices = min((n + 255) // 256, 2)
    per = -(-(-(-n // slices)) // 32) * 32
    total = np.zeros((dz.shape[1], x.shape[1]), np.float32)
    for r0 in range(0, n, per):
        part = np.zeros_like(total)
        for r in range(r0, min(n, r0 + per)):
            part += np.outer(dz[r], x[r]).astype(np.float32)   # products of BF16 values are exact in FP32
        total += part
    return total


@pytest.mark.parametrize("n", [64, 100, 129, 192, 256, 300, 512])
def test_sums_of_several_chunks(gpu_lib, n):
    G = gpu_lib
    g = np.random.default_rng(n)
    ctx = G.Context(0, 512, 0)
    ctx.nn_init(1)
    params = np.zeros_like(ctx.nn_params())
    layers = N.split(params)
    c = N.bf16((g.standard_normal(128) * np.exp(g.standard_normal(128))).astype(np.float32))
    layers[4][1][:] = 1.0                        # fc1: every unit is one
    layers[5][0][0, 0::2], layers[5][0][0, 1::2] = c, -c
    layers[5][1][0] = 1.0                        # fc2: unit 0 is one, the others zero
    layers[6][0][0, 0], layers[6][1][0] = 1.0, -1.0
    ctx.nn_set_params(params)
    d = N.bf16((g.standard_normal(n) * np.exp(g.standard_normal(n))).astype(np.float32))
    target = np.zeros((n, 3), np.float32)
    target[:, 0] = -1.5 * n * d                  # d = 2 (0 - target) / (3 n), to the nearest BF16
    x1 = N.bf16(np.maximum(g.standard_normal((n, 256)), 0.0).astype(np.float32))
    _, grads, pred = ctx.nn_forward_backward(x1.astype(np.float32), np.zeros((n, 256, 256), np.float32), target)
    ctx.close()
    assert not pred.any()
    gw, gb = N.split(grads)[4]
    dz = N.bf16(np.outer(d, layers[5][0][0]).astype(np.float32))
    for got, x in ((gw[:, :256], x1), (gb[:, None], np.ones((n, 1)))):
        exact = dz.T @ x
        assert np.linalg.norm(got - exact) <= np.linalg.norm(running_sums(dz, x) - exact), (n, x.shape[1])
