"""Background removal of many spectra in one call, whose blocks are of 64 rows
where the box leaves them wide enough (bg_shape: from 10 spectra of tile 512 and
99 of tile 90; tiles of 1024 and 2048 keep 32), against the host formula: one
that does not know the blocks, so that no rule for them makes a case empty."""
import numpy as np
import pytest

from test_background_gpu import background_removed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log", [0, 1])
@pytest.mark.parametrize("tile,count", [(512, 24), (90, 160), (256, 60), (1024, 12), (2048, 3)])
def test_background_of_many_spectra(gpu_lib, tile, count, log):
    """The right half of a diagnostic spectrum is the half spectrum without its
    last column; faint images keep it without the lowpass.  Bound as for one
    spectrum: the rounding to float32, and 1e-12 of the local background."""
    G = gpu_lib
    g = np.random.default_rng(tile + log)
    n = 2 * tile if tile > 90 else 512
    imgs = [(g.standard_normal((n, n)) * 1e-3 + 1.0).astype(np.float32) for _ in range(count)]
    op = G.make_optics(pixel_size=1.35)
    ctx = G.Context(0, tile, log)
    ctx.set_spectrum_impl(G.GCF_SPECT_CUFFT)   # raw spectra that do not depend on the company
    full = ctx.run_series(imgs, op, is_tomo=False, want_full=True)[1]
    for k in (0, 1, count // 2, count - 1):
        ctx.setup(op, n, n)
        ctx.gen_half_spectrum(imgs[k])
        ref, b = background_removed(ctx.half_spectrum(True), log)
        assert ref.var() < 1.0
        got, ref, b = full[k][:, tile // 2:], ref[:, :-1], b[:, :-1]
        assert np.all(np.abs(got - ref) <= 6.1e-8 * np.abs(ref) + 1e-12 * np.abs(b)), k
    ctx.close()
