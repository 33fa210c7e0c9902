"""Contexts of different tile sizes in threads of their own: a kernel's attributes
belong to the process, so no thread may set them to its own call's needs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tile_sizes_in_threads(gpu_lib):
    import torch
    G = gpu_lib
    tiles = (64, 256, 512, 1024, 2048)   # background blocks of 20 to 190 KB of shared memory
    g = torch.Generator(device="cuda").manual_seed(1)
    img = torch.poisson(torch.full((2300, 2300), 6.0, device="cuda"), generator=g)
    torch.cuda.synchronize()

    def spectra(tile, n, out):
        try:
            ctx = G.Context(0, tile, 0)
            ctx.setup(G.make_optics(pixel_size=1.35), img.shape[1], img.shape[0])
            for _ in range(n):
                ctx.gen_half_spectrum(img)
                out.append(ctx.half_spectrum(False))
            ctx.close()
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            out.append(e)

    want = {}
    for t in tiles:
        out = []
        spectra(t, 1, out)
        want[t] = out[0]
    got = {t: [] for t in tiles}
    threads = [threading.Thread(target=spectra, args=(t, 200, got[t])) for t in tiles]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for t in tiles:
        assert not isinstance(got[t][-1], Exception), (t, got[t][-1])
        assert len(got[t]) == 200 and all(np.array_equal(a, want[t]) for a in got[t]), t
