"""The tensor-core product on pairs of CTAs (256 x 256 tiles) at the edges of its
range: the smallest tile count that takes it and just below, ragged rows, columns
and K, a last tile of one row or column, against an FP32 torch product of the
same BF16 operands.  Tolerance per element: 2^-22 x sqrt(K) x max |a| |b| x 8, the
growth of FP32 accumulation in another order (measured spread below a quarter)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(4096, 2560, 1024),     # 160 tiles
                                   (4097, 2305, 1025),     # 170 tiles, ragged everywhere, one-row tile
                                   (2304, 4353, 1087),     # one column over
                                   (4096, 2304, 1023),     # short K: the one-CTA product
                                   (3000, 2900, 4097)])    # 144 tiles: below the rule on 148 SMs
def test_pair_product_matches_torch(gpu_lib, m, n, k):
    import torch
    G = gpu_lib
    L = G.load_library()
    kp = (k + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn((m, kp), generator=g, device="cuda").bfloat16()
    b = torch.randn((n, kp), generator=g, device="cuda").bfloat16()
    d = torch.full((m, n + 3), float("nan"), device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert L.gcf_gemm_bf16_ex(a.data_ptr(), kp, b.data_ptr(), kp, m, n, k, d.data_ptr(), n + 3, 256, 4, 1, st) == 0
    ref = a[:, :k].double() @ b[:, :k].double().t()
    tol = 2.0 ** -22 * k ** 0.5 * 8 * float(a.abs().max() * b.abs().max())
    assert float((d[:, :n].double() - ref).abs().max()) <= tol
    assert bool(torch.isnan(d[:, n:]).all())
    one = torch.empty((m, n), device="cuda")
    assert L.gcf_gemm_bf16(a.data_ptr(), kp, b.data_ptr(), kp, m, n, k, one.data_ptr(), n, 256, 4, st) == 0
    assert torch.equal(one, d[:, :n])


def test_products_on_several_streams(gpu_lib):
    """Products on pairs of CTAs and on single ones, launched on three streams
    so that each starts while another leaves its SMs: every result equals the
    one computed alone."""
    import torch
    L = gpu_lib.load_library()
    shapes = [(4096, 2560, 1024), (3000, 2900, 1088), (2816, 3840, 2048)]
    g = torch.Generator(device="cuda").manual_seed(3)
    ops, ref = [], []
    for m, n, k in shapes:
        a = torch.randn((m, k), generator=g, device="cuda").bfloat16()
        b = torch.randn((n, k), generator=g, device="cuda").bfloat16()
        ops.append((a, b, m, n, k))
    call = lambda o, d, st: L.gcf_gemm_bf16_ex(  # noqa: E731
        o[0].data_ptr(), o[4], o[1].data_ptr(), o[4], o[2], o[3], o[4], d.data_ptr(), o[3], 256, 4, 1, st)
    for o in ops:
        ref.append(torch.empty((o[2], o[3]), device="cuda"))
        assert call(o, ref[-1], torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [[torch.empty_like(r) for r in ref] for _ in streams]
    for i in range(200):
        for s, st in enumerate(streams):
            q = (i + s) % len(ops)
            assert call(ops[q], outs[s][q], st.cuda_stream) == 0
    torch.cuda.synchronize()
    for o in outs:
        for d, r in zip(o, ref):
            assert torch.equal(d, r)
