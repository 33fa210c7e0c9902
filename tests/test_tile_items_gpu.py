"""The default tile kernel over several work items per cluster: between two
items the column buffer is written plainly (the item's sums on their way out)
and then by the peers' bulk copies (the next item's first tile)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _raw(G, img, shape):
    h, w = img.shape
    ctx = G.Context(0, 512, 0)
    ctx.set_fused_shape(shape)
    ctx.setup(G.make_optics(pixel_size=1.3), w, h)
    out = []
    for _ in range(3):
        ctx.gen_half_spectrum(img)
        out.append(ctx.half_spectrum(raw=True))
    ctx.close()
    return out


@pytest.mark.parametrize("w,h", [(5760, 4092), (11520, 8184), (9001, 9003)])
def test_items_in_a_row_keep_the_bits(gpu_lib, w, h):
    """Frames of up to a hundred items, against the one-line kernel, which
    neither copies in bulk nor stages its sums."""
    import torch
    G = gpu_lib
    g = torch.Generator(device="cuda").manual_seed(w)
    img = torch.poisson(torch.full((h, w), 7.0, device="cuda"), generator=g)
    img += 3.0 * torch.sin(torch.arange(w, device="cuda") * 0.31)   # tiles and columns that differ
    want = _raw(G, img, 816)[0]
    for got in _raw(G, img, 8):
        assert np.array_equal(got, want)
