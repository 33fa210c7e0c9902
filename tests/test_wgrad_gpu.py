"""Weight gradients of ragged batches on the GPU.

The weight-gradient kernel sums chunks of 64 or 256 rows, 32 outputs and 16,
144 or 288 columns per CTA: one sample leaves the dense layers a single row,
33 samples a partial chunk in one slice and the convolutions unequal slices
over the SMs, 130 samples a dense chunk of two rows.  Bars: those of the
gradient check at a batch of 4 (per layer a relative L2 error <= 1e-2 and a
cosine similarity >= 0.9999 against the oracle that rounds to BF16 at the
same points); the sums themselves have no atomics, so a second call returns
the same bits.
"""
import numpy as np
import pytest

from oracle import nn_oracle as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 33, 130])
def test_gradients_of_ragged_batches(gpu_lib, n):
    G = gpu_lib
    ctx = G.Context(0, 512, 0)
    ctx.nn_init(17)
    op = G.make_optics()
    x1, x2, t, _ = ctx.nn_synth_inputs(op, seed=23, first=100, n=n)
    params = ctx.nn_params()
    _, grads, _ = ctx.nn_forward_backward(x1, x2, t)
    _, again, _ = ctx.nn_forward_backward(x1, x2, t)
    ctx.close()
    assert np.array_equal(grads, again)
    _, ograds, _ = N.forward_backward(params, N.bf16(x1), N.bf16(x2), t, emulate_bf16=True)
    for k, ((gw, gb), (ow, ob)) in enumerate(zip(N.split(grads), N.split(ograds))):
        for a, b in ((gw, ow), (gb, ob)):
            a, b = a.ravel().astype(np.float64), b.ravel()
            nb = np.linalg.norm(b)
            if nb == 0:
                assert np.linalg.norm(a) == 0
                continue
            assert np.linalg.norm(a - b) <= 1e-2 * nb, (n, k)
            assert a @ b >= 0.9999 * np.linalg.norm(a) * nb, (n, k)
