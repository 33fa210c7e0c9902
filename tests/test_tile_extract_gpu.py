"""Tile extraction of the cuFFT spectrum variant (tiles other than 512): row
slices and one warp per row, at tile edges that are no multiple of a warp, of
the eight rows of a CTA or of the 16 row slices, on odd image sizes and with a
row pitch wider than the image, against the same
definition in FP64 numpy.

Tolerance per pixel 1e-4 |ref| + 1e-5 mean(ref): the accuracy bar of the
averaged spectra (FP32 transforms, relative rounding below 1e-6 each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,w,h,pad", [(16, 101, 67, 0), (18, 64, 64, 3), (100, 333, 251, 0), (250, 777, 640, 1),
                                          (1024, 1601, 2049, 0), (2048, 2048, 3100, 5)])
def test_raw_spectrum_of_other_tiles(gpu_lib, tile, w, h, pad):
    import torch
    G = gpu_lib
    rng = np.random.default_rng(tile)
    buf = rng.poisson(20.0, size=(h, w + pad)).astype(np.float32)
    img = np.ascontiguousarray(buf[:, :w])
    ctx = G.Context(0, tile, 0)
    ctx.setup(G.make_optics(pixel_size=1.3), w, h)
    ctx.gen_half_spectrum(torch.from_numpy(buf).cuda(), pitch=w + pad)
    got = ctx.half_spectrum(raw=True).astype(np.float64)
    ctx.close()
    want = _fp64(img, tile)
    assert np.all(np.abs(got - want) <= 1e-4 * np.abs(want) + 1e-5 * want.mean())


def _fp64(img, tile):
    ov = tile // 2 // 2 * 2
    st = tile - ov
    h, w = img.shape
    nx, ny = (w - ov) // st, (h - ov) // st
    ox, oy = (w - nx * tile + (nx - 1) * ov) // 2, (h - ny * tile + (ny - 1) * ov) // 2
    c = np.abs(np.arange(tile) - 0.5 * tile) * 2.0 / tile
    r = np.sqrt(c[:, None] ** 2 + c[None, :] ** 2)
    taper = np.where(r < 1.0, 1.0 - (0.5 * (1.0 - np.cos(np.pi * r))) ** 3, 0.0)
    acc = np.zeros((tile, tile // 2 + 1))
    for ty in range(ny):
        for tx in range(nx):
            t = img[oy + ty * st:oy + ty * st + tile, ox + tx * st:ox + tx * st + tile].astype(np.float64)
            # the mean that is removed is a float32 (GNormalize2D): its rounding shows at DC
            acc += np.abs(np.fft.rfft2((t - np.float64(np.float32(t.mean()))) * taper))
    return np.roll(acc / (nx * ny), tile // 2, axis=0)
