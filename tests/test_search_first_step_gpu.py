"""The first step of a refinement-only search follows the kernel that gathers
its band spectrum, with no 1D search between them: the step has to see this
call's spectrum, whatever the buffer held before."""
import pytest

from gctffind_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [256, 512])
def test_refinement_reads_this_calls_spectrum(gpu_lib, tile):
    """Refinements of two spectra in turn, at one set of buffers, against each
    in a context of its own."""
    G = gpu_lib
    op = G.make_optics(pixel_size=1.35)
    imgs = [synth.make_micrograph(synth.MicrographSpec(width=3 * tile, height=3 * tile, pixel_size=1.35,
                                                       df_min=11800.0, df_max=12200.0, azimuth_deg=az, dose=3.0,
                                                       seed=seed), device="cuda")
            for az, seed in ((35.0, 3), (-50.0, 4))]

    def refine(ctx, img):
        ctx.setup(op, img.shape[1], img.shape[0])
        ctx.gen_half_spectrum(img)
        return ctx.refine((12000.0, 800.0), (0.01, 0.02), (0.0, 180.0), (0.0, 0.0)).as_dict()

    want = []
    for img in imgs:
        ctx = G.Context(0, tile, 0)
        want.append(refine(ctx, img))
        ctx.close()
    assert want[0] != want[1]
    ctx = G.Context(0, tile, 0)
    for k in range(40):
        assert refine(ctx, imgs[k % 2]) == want[k % 2], k
    ctx.close()
