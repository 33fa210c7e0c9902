"""A micrograph's results do not depend on what else is in its call, to the
bit, also where the sums over its pixels are not exact in FP64."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image_at_a_rounding_tie(seed):
    """One 512 x 512 tile of floats of many exponents whose exact mean lies
    halfway between two floats: an FP64 sum of its pixels, off by an ulp or not,
    decides the rounding of the mean, so every order of adding them shows."""
    g = np.random.default_rng(seed)
    a = (g.standard_normal((512, 512)) * np.exp2(g.uniform(-8.0, 2.0, (512, 512))) + 0.3).astype(np.float32)
    a[0, 0] = a[0, 1] = 0.0
    n = a.size
    total = math.fsum(a.ravel().tolist())
    lo = np.float32(total / n)
    hi = np.nextafter(lo, np.float32(np.inf))
    want = 0.5 * (float(lo) + float(hi)) * n
    a[0, 0] = np.float32(want - total)           # to within its rounding
    total = math.fsum(a.ravel().tolist())
    a[0, 1] = np.float32(want - total)           # the rest
    assert math.fsum(a.ravel().tolist()) == want
    return a


def test_mean_of_a_tile_does_not_depend_on_the_call(gpu_lib):
    """Single tiles alone (few block sums per call) and among copies (many)."""
    import torch
    G = gpu_lib
    ctx = G.Context(0, 512, 0)
    op = G.make_optics(pixel_size=1.35)

    def measured(imgs):   # the measured half of the diagnostic spectra
        return ctx.run_series(imgs, op, is_tomo=False, want_full=True)[1][:, :, 256:]

    for seed in range(12):
        img = torch.from_numpy(_image_at_a_rounding_tie(seed)).cuda()
        one, many = measured([img])[0], measured([img] * 160)
        assert all(np.array_equal(m, one) for m in many), seed
    ctx.close()
