"""Bounded waits of the default tile kernel that run out
(gcf_avg_spectrum_gave_up: every CTA waits for bytes that nobody sends)."""
import time

import pytest

pytestmark = pytest.mark.gpu


def _call(L, name, img, out):
    import torch
    st = getattr(L, name)(img.data_ptr(), img.shape[1], img.shape[0], img.shape[1], out.data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
    assert st == 0, L.gcf_strerror(st)
    torch.cuda.synchronize()
    return out.clone()


@pytest.mark.parametrize("w,h", [(512, 512), (3838, 3710), (9001, 9003)])
def test_kernel_ends_soon_after_a_wait_gives_up(gpu_lib, w, h):
    """One tile, several tiles per item and several items per cluster: the call
    ends within a few seconds (one bounded wait of about a second, not one per
    tile), twice in a row, and the next call's spectrum is what it was."""
    import torch
    L = gpu_lib.load_library()
    g = torch.Generator(device="cuda").manual_seed(w)
    img = torch.poisson(torch.full((h, w), 7.0, device="cuda"), generator=g)
    out = torch.empty((512, 257), device="cuda")
    want = _call(L, "gcf_avg_spectrum_noalloc", img, out)
    for _ in range(2):
        t = time.monotonic()
        _call(L, "gcf_avg_spectrum_gave_up", img, out)
        assert 0.5 < time.monotonic() - t < 5.0
        assert torch.equal(_call(L, "gcf_avg_spectrum_noalloc", img, out), want)


def test_spectrum_of_a_wait_that_gave_up_is_nan(gpu_lib):
    """The allocation-free call cannot report it in its status, which it returns
    before the kernels run."""
    import torch
    L = gpu_lib.load_library()
    img = torch.ones((1200, 1100), device="cuda")
    img[::3, ::5] = 4.0
    out = torch.zeros((512, 257), device="cuda")
    assert torch.isnan(_call(L, "gcf_avg_spectrum_gave_up", img, out)).all()
    assert torch.isfinite(_call(L, "gcf_avg_spectrum_noalloc", img, out)).all()
