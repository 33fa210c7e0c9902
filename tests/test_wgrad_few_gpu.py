"""Weight gradients of batches below 64 samples, whose dense layers have fewer
rows than one chunk of the tensor-core kernel: every sum is the exact one,
rounded to float32 once.

All weights are zero, so the last hidden layer is its (BF16) bias for every
sample and the prediction zero; the targets put a chosen BF16 value into each
element of the last layer's output gradient.  Its weight gradient is then known
exactly on the host."""
import math

import numpy as np
import pytest

from oracle import nn_oracle as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 17, 33, 48, 63])
def test_sums_of_few_rows_are_rounded_once(gpu_lib, n):
    G = gpu_lib
    g = np.random.default_rng(n)
    ctx = G.Context(0, 512, 0)
    ctx.nn_init(1)
    params = np.zeros_like(ctx.nn_params())
    h2 = N.bf16(np.exp(g.uniform(-3.0, 3.0, 128)).astype(np.float32))
    layers = N.split(params)
    layers[5][1][:] = h2
    ctx.nn_set_params(params)
    dz = N.bf16((g.standard_normal((n, 3)) * np.exp(g.uniform(-4.0, 2.0, (n, 3)))).astype(np.float32))
    target = (-1.5 * n * dz).astype(np.float32)      # dz = 2 (0 - target) / (3 n), to the nearest BF16
    x1, x2 = np.zeros((n, 256), np.float32), np.zeros((n, 256, 256), np.float32)
    _, grads, pred = ctx.nn_forward_backward(x1, x2, target)
    ctx.close()
    assert not pred.any()
    gw, gb = N.split(grads)[6]
    for o in range(3):
        exact = np.array([math.fsum(dz[:, o] * v) for v in h2])    # the products are exact in FP64
        slack = 1e-14 * np.abs(dz[:, o]).sum() * h2
        assert np.all(np.abs(gw[o] - exact) <= 2.0 ** -24 * np.abs(exact) + slack), (n, o)
        b = math.fsum(dz[:, o])
        assert abs(gb[o] - b) <= 2.0 ** -24 * abs(b) + 1e-14 * np.abs(dz[:, o]).sum()
