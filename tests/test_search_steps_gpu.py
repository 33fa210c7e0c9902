"""Search steps: the 1D search spread over CTAs, and the 2D steps ended by
every CTA of the next step (few searches) or by the last CTA (many).

A search's result must not depend on how many searches run beside it, so a
batch of copies gives the single call's result bit for bit on both sides of
the rule, for plain, contraction and extra-phase searches (a phase range above
61 degrees has more line candidates than any other step).  The extra-phase
results are also compared with the FP64 oracle at the repository's search
bars: one mean-defocus step (60 A here) and 1e-3 in CC, the phase within 2
degrees where the CCs agree."""
import pytest

from gctffind_b200 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("df_min", "df_max", "azimuth", "ext_phase", "score", "ctf_res", "df_1d", "phase_1d", "score_1d")


def _img(tile, phase, seed):
    s = synth.MicrographSpec(width=3 * tile, height=3 * tile, pixel_size=1.35, df_min=11800.0, df_max=12200.0,
                             azimuth_deg=35.0, dose=3.0, seed=seed, ext_phase_deg=phase)
    return synth.make_micrograph(s)


@pytest.mark.parametrize("tile,mode,phase,prange", [(512, 0, 0.0, 0.0), (512, 1, 0.0, 0.0), (256, 0, 60.0, 140.0),
                                                    (512, 0, 30.0, 62.0)])
@pytest.mark.parametrize("n", [2, 4, 13])
def test_result_does_not_depend_on_the_batch(gpu_lib, tile, mode, phase, prange, n):
    G = gpu_lib
    imgs = [_img(tile, phase, 7).cuda(), _img(tile, phase, 8).cuda()]
    op = G.make_optics(pixel_size=1.35, ext_phase_deg=phase, ext_phase_range=prange)
    ctx = G.Context(0, tile, 0)
    one = [ctx.run_batch([a], [1.35], op, mode=mode)[0] for a in imgs]
    many = ctx.run_batch([imgs[k % 2] for k in range(n)], [1.35] * n, op, mode=mode)
    ctx.close()
    for k, r in enumerate(many):
        for f in FIELDS:
            assert getattr(r, f) == getattr(one[k % 2], f), (k, f)


@pytest.mark.parametrize("prange", [5.0, 62.0, 150.0])
def test_phase_search_matches_oracle(gpu_lib, oracle, prange):
    G = gpu_lib
    img = _img(256, 70.0, 9).numpy()
    ctx = G.Context(0, 256, 0)
    ctx.setup(G.make_optics(pixel_size=1.35), img.shape[1], img.shape[0])
    ctx.gen_half_spectrum(img)
    ctx.set_phase(60.0, prange)
    g = ctx.do2d()
    ctx.close()
    p = oracle.params(pixel_size=1.35, tile_size=256, ext_phase_deg=60.0, ext_phase_range=prange)
    o = oracle.find_ctf_image(img, 1.35, p, mode=0)
    o = o[0] if isinstance(o, tuple) else o
    assert abs(g.score - o.score) <= 1e-3
    assert abs(g.df_min - o.df_min) <= 60.0 and abs(g.df_max - o.df_max) <= 60.0
    assert abs(g.ext_phase - o.ext_phase) <= 2.0
