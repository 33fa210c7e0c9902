"""The default tile kernel (two lines per warp, bulk copies between the CTAs of
a cluster) and its cluster-less companion against the one-line kernel: the same
operations in the same order, so the averaged spectra must be the same bits, at
one tile, at ragged sizes, at rows that are only 4-byte aligned (odd offsets,
odd pitch, a base address one float in), and for non-finite pixels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _raw(G, img, w, h, pitch, shape):
    ctx = G.Context(0, 512, 0)
    ctx.set_fused_shape(shape)
    ctx.setup(G.make_optics(pixel_size=1.3), w, h)
    ctx.gen_half_spectrum(img, pitch=pitch)
    out = ctx.half_spectrum(raw=True)
    ctx.close()
    return out


@pytest.mark.parametrize("w,h,pitch,skip", [(512, 512, 512, 0), (513, 767, 513, 0), (1025, 513, 1031, 1),
                                            (1811, 1201, 1811, 0), (2050, 1300, 2052, 2), (6400, 700, 6401, 3)])
@pytest.mark.parametrize("bad", [None, float("inf"), float("nan")])
def test_pair_kernel_equals_one_line_kernel(gpu_lib, w, h, pitch, skip, bad):
    import torch
    G = gpu_lib
    g = torch.Generator().manual_seed(w)
    buf = torch.poisson(torch.full((h * pitch + skip,), 7.0), generator=g)
    if bad is not None:
        buf[skip + (h // 2) * pitch + w // 2] = bad
    img = buf.cuda()[skip:].view(h, pitch)
    a = _raw(G, img, w, h, pitch, 8)
    b = _raw(G, img, w, h, pitch, 816)
    assert np.array_equal(a, b, equal_nan=True)
    assert bad is not None or np.all(np.isfinite(a))


@pytest.mark.parametrize("w,n", [(2561, 24), (1700, 40)])
def test_cluster_less_ctas_equal_the_clusters(gpu_lib, w, n):
    """More items than the cluster-less CTAs leave to the clusters (six per
    cluster), on an odd width: every copy of a micrograph gives the bits of a
    launch with too few items for them."""
    import torch
    G = gpu_lib
    g = torch.Generator().manual_seed(n)
    img = torch.poisson(torch.full((3001, w), 5.0), generator=g).cuda()
    ctx = G.Context(0, 512, 0)
    op = G.make_optics()
    one = ctx.run_batch([img], [1.3], op, mode=G.GCF_SEARCH_BF16)[0]
    many = ctx.run_batch([img] * n, [1.3] * n, op, mode=G.GCF_SEARCH_BF16)
    ctx.close()
    for r in many:
        assert r.as_dict() == one.as_dict()


@pytest.mark.parametrize("w,h", [(512, 512), (1024, 1024), (1500, 2049), (3838, 3710)])
def test_tiles_handed_out_singly_keep_the_bits(gpu_lib, w, h):
    """One small frame alone (its tiles handed out one by one) and the same
    frame in a batch that fills the clusters (whole items): the same result."""
    import torch
    from gctffind_b200 import synth
    G = gpu_lib
    s = synth.MicrographSpec(width=w, height=h, pixel_size=1.4, df_min=13000.0, df_max=13300.0, dose=3.0, seed=w)
    img = synth.make_micrograph(s, device="cuda")
    ctx = G.Context(0, 512, 0)
    op = G.make_optics()
    one = ctx.run_batch([img], [1.4], op)[0]
    n = max(9, 16 * 24 // max(1, ((w - 256) // 256) * ((h - 256) // 256)) + 1)
    many = ctx.run_batch([img] * n, [1.4] * n, op)
    ctx.close()
    for r in many:
        assert r.as_dict() == one.as_dict()
