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


def test_whole_items_where_memory_is_short(gpu_lib):
    """A frame whose tiles are handed out singly keeps a partial spectrum per
    tile (169 of them, 89 MB); with less device memory left it runs on whole
    items, to the same bits."""
    import torch
    G = gpu_lib
    g = torch.Generator(device="cuda").manual_seed(3)
    img = torch.poisson(torch.full((3710, 3838), 5.0, device="cuda"), generator=g)
    other = img[:1024, :1024].contiguous()
    ctx = G.Context(0, 512, 0)

    def raw(x):
        ctx.setup(G.make_optics(pixel_size=1.3), x.shape[1], x.shape[0])
        ctx.gen_half_spectrum(x)
        return ctx.half_spectrum(raw=True)

    raw(other)                                  # all buffers but the larger frame's partials
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (48 << 20), dtype=torch.uint8, device="cuda")
    short = raw(img)
    del hold
    torch.cuda.empty_cache()
    assert np.array_equal(raw(img), short)      # singly
    ctx.close()
