"""Background removal over tile sizes, edges of its blocks and both spectrum
kinds.

A block covers 8 rows, or 32 or 64 when the call has more blocks than the chip
takes at once, and a strip of columns (one strip up to tile 256, more above), so
the tile sizes below have partial strips and the row and column folds in different
blocks; 16 is the smallest tile and 90 leaves partial blocks of rows.  A faint
image keeps the variance of the result below 1, so that the half spectrum comes
back without the lowpass.  The reference takes the same float32 square roots and
FP64 box sums: what remains is the final rounding to float32 (6e-8 relative) and
FP64 sums in another order, which leave at most 1e-12 of the local background.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def background_removed(raw, log):
    cy, cx = raw.shape
    tile, half = cy, cx - 1
    box = int(np.float32(1.0) / np.float32(15.0) * np.float32(tile))
    box = min(box, int(np.float32(0.3) * np.float32(tile)))
    box = max(box // 2 * 2 + 1, 7)
    hb = box // 2
    a = (raw if log else np.sqrt(raw)).astype(np.float64)
    mirror = a[(-np.arange(tile)) % tile]
    u = np.arange(-hb, cx + hb)
    u = np.where(u >= half, u - 2 * half, u)
    ext = np.where(u >= 0, a[:, np.abs(u)], mirror[:, np.abs(u)])
    v = sum(np.roll(ext, -k, axis=0) for k in range(-hb, hb + 1))
    s = sum(v[:, k:k + cx] for k in range(box))
    b = s / float(box * box)
    if not log:
        b = b * b
    x = np.arange(cx, dtype=np.float32) * np.float32(0.5) / np.float32(half)
    yr = np.arange(tile) - tile // 2
    y2 = (yr * yr).astype(np.float32) / np.float32(tile * tile)
    fr = np.sqrt(x[None] * x[None] + y2[:, None])
    ref = raw.astype(np.float64) - b
    ref[fr.astype(np.float64) < 0.04] = 0.0
    return ref, b


@pytest.mark.parametrize("log", [0, 1])
@pytest.mark.parametrize("tile", [16, 90, 256, 512, 1024, 2048])
def test_background_removed(gpu_lib, tile, log):
    G = gpu_lib
    g = np.random.default_rng(tile + log)
    n = max(2 * tile, 1024)
    img = (g.standard_normal((n, n)) * 1e-3 + 1.0).astype(np.float32)
    ctx = G.Context(0, tile, log)
    ctx.setup(G.make_optics(pixel_size=1.35), n, n)   # no rescale
    ctx.gen_half_spectrum(img)
    raw, got = ctx.half_spectrum(True), ctx.half_spectrum(False)
    ctx.close()
    ref, b = background_removed(raw, log)
    assert ref.var() < 1.0   # no lowpass
    assert np.all(np.abs(got - ref) <= 6.1e-8 * np.abs(ref) + 1e-12 * np.abs(b))


@pytest.mark.parametrize("tile,count", [(90, 46), (512, 9), (1024, 5), (2048, 2)])
def test_blocks_of_32_rows_match_blocks_of_8(gpu_lib, tile, count):
    """Spectra made together (blocks of 32 or 64 rows) against the same spectra made
    one by one, by the per-micrograph cuFFT path, whose raw spectra do not
    depend on the company.  The right half of a full spectrum is the half
    spectrum without its last column."""
    G = gpu_lib
    g = np.random.default_rng(tile)
    n = 2 * tile if tile > 90 else 512
    imgs = [(g.standard_normal((n, n)) * 1e-3 + 1.0).astype(np.float32) for _ in range(count)]
    op = G.make_optics(pixel_size=1.35)
    ctx = G.Context(0, tile, 0)
    ctx.set_spectrum_impl(G.GCF_SPECT_CUFFT)
    full = ctx.run_series(imgs, op, is_tomo=False, want_full=True)[1]
    for k in (0, count // 2, count - 1):
        ctx.setup(op, n, n)
        ctx.gen_half_spectrum(imgs[k])
        raw, one = ctx.half_spectrum(True), ctx.half_spectrum(False)
        assert one.var() < 1.0
        a, b = np.asarray(full[k])[:, tile // 2:], one[:, :-1]
        assert np.all(np.abs(a - b) <= 1.3e-7 * np.abs(b) + 1e-12 * np.abs(raw[:, :-1]).max())
    ctx.close()
