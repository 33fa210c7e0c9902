"""The two lanes (streams) of a batch's tensor-core rescale (RescaleLanes in
gcf_capi.cpp)."""
import numpy as np
import pytest

from gctffind_b200 import synth

pytestmark = pytest.mark.gpu


def _imgs(n, w, h, seed):
    return [synth.make_micrograph(synth.MicrographSpec(width=w, height=h, pixel_size=0.85, df_min=14000.0,
                                                       df_max=14300.0, dose=2.0, seed=seed + k), device="cuda")
            for k in range(n)]


def _batch(ctx, G, imgs):
    return [r.as_dict() for r in ctx.run_batch(imgs, [0.85] * len(imgs), G.make_optics(), mode=G.GCF_SEARCH_BF16)]


@pytest.mark.parametrize("n", [2, 3, 6])
def test_failed_call_leaves_no_lane_running(gpu_lib, n):
    """A batch that fails after images have been placed on both lanes (its
    last frame, rescaled, holds no tile) and, straight after it, a good one
    on the same buffers: the results of a context that saw no failure."""
    import torch
    G = gpu_lib
    ctx = G.Context(0, 512, 0)
    ctx.set_rescale_impl(G.GCF_RESCALE_GEMM)
    good, other = _imgs(n, 2048, 1900, 100), _imgs(n, 2048, 1900, 500)
    small = torch.ones((540, 540), device="cuda")   # 382 x 382 once rescaled
    want = _batch(ctx, G, good)
    for _ in range(3):
        with pytest.raises(G.GcfError, match="tile"):
            _batch(ctx, G, other + [small])
        assert _batch(ctx, G, good) == want
    ctx.close()


def test_one_lane_where_memory_is_short(gpu_lib):
    """With everything of a call allocated but the second lane's scratch, and
    less device memory left than that takes, the call runs on one lane."""
    import torch
    G = gpu_lib
    ctx = G.Context(0, 512, 0)
    imgs = [img for seed in (100, 500) for img in _imgs(1, 5760, 4092, seed)]
    ctx.set_rescale_impl(G.GCF_RESCALE_LINES)
    _batch(ctx, G, imgs)                        # all but the lanes' scratch
    ctx.set_rescale_impl(G.GCF_RESCALE_GEMM)
    _batch(ctx, G, imgs[:1])                    # the first lane's (about 150 MB)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (64 << 20), dtype=torch.uint8, device="cuda")
    got = _batch(ctx, G, imgs)
    del hold
    torch.cuda.empty_cache()
    assert _batch(ctx, G, imgs) == got          # on two lanes
    ctx.close()
