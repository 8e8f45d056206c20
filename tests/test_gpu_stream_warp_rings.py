"""The streaming product's two forms against float64, every epilogue.  Rings of warps: rows on both sides of 8, every K form (activations in
registers whole, or stages ahead), columns that end inside a unit of 8 or 16 rows, more and fewer units than SMs.  Bulk copies: activations
in shared memory and from L2, the same edges.  Operands that are slices of wider buffers, and norms handed over between two products."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def bound(a, w, k):
    """Exact products, each of k sums rounded once (to float32; the tensor core's own sums of 16 may be cut instead of rounded)."""
    return 2 * k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)


def gated(out, act):
    """The gated activation of alternating gate and up columns, in float64."""
    alpha, limit, offset, cubic = act
    gate, up = out[:, 0::2].double().clamp(max=limit), out[:, 1::2].double().clamp(-limit, limit) + offset
    return gate * torch.sigmoid(alpha * gate + cubic * gate ** 3) * up


def check_every_epilogue(a, w, M, N, K, wide=0):
    """``wide``: that many columns of every output's buffer lie beside the output and stay as they are."""
    from inf_engine_b200 import kernels

    def room(n, dtype=torch.float32):
        return torch.full((M, n + wide), float("nan"), device="cuda", dtype=dtype)

    g = torch.Generator("cuda").manual_seed(1)
    ref, most = a.double() @ w.double().T, bound(a, w, K)
    buffers = [room(N), room(N, BF), torch.randn(M, N + wide, device="cuda", generator=g), room(N, BF), room(N // 2, BF), room(N // 2, BF)]
    out, half, total, squares, silu, gelu = (b[:, wide:] for b in buffers)
    start = buffers[2].clone()
    kernels.gemm_stream(a, w, out, M, "f32")
    assert bool(((out.double() - ref).abs() <= most).all())
    kernels.gemm_stream(a, w, half, M, "bf16")
    assert torch.equal(half, out.to(BF))
    kernels.gemm_stream(a, w, total, M, "residual")
    assert torch.equal(total, start[:, wide:] + out)
    kernels.gemm_stream(a, w, squares, M, "relu2")
    assert torch.equal(squares, (out.clamp(min=0) ** 2).to(BF))
    if N % 2 == 0:
        kernels.gemm_stream(a, w, silu, M, "silu_mul")
        want = gated(out, (1.0, float("inf"), 0.0, 0.0))
        assert bool(((silu.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())
        for act in (kernels.glu_constants("gelu_tanh"), kernels.glu_constants("clamped_swish", 1.7, 3.0, 1.0)):
            gelu.fill_(float("nan"))
            kernels.gemm_stream(a, w, gelu, M, "glu", act=act)
            want = gated(out, act)
            assert bool(((gelu.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())
    if wide:
        assert torch.equal(buffers[2][:, :wide], start[:, :wide])
        assert all(bool(b[:, :wide].isnan().all()) for i, b in enumerate(buffers) if i != 2)
    torch.cuda.synchronize()
    assert kernels.stream_error() == 0


@pytest.mark.parametrize("K", [1024, 2048, 3072, 4096, 6144, 8192])
@pytest.mark.parametrize("M,N", [(1, 5), (8, 1189), (9, 2056), (16, 9490), (7, 19001)])
def test_stores_against_float64(M, N, K):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(BF)
    check_every_epilogue(a, w, M, N, K)


# activations in shared memory up to 100 KB of padded rows, from L2 beyond (5,120 with more than 8 rows, 11,008)
@pytest.mark.parametrize("M,N,K", [(1, 5, 768), (8, 1190, 1280), (8, 520, 5120), (9, 520, 5120), (16, 9490, 5120), (7, 9490, 1280), (16, 19002, 768),
                                   (8, 520, 11008), (8, 9490, 11008), (13, 1002, 11008)])
def test_stores_of_bulk_copies_against_float64(M, N, K):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(BF)
    check_every_epilogue(a, w, M, N, K)


@pytest.mark.parametrize("K", [2048, 4096, 1280, 11008])
@pytest.mark.parametrize("M,N", [(5, 390), (16, 9490)])
def test_operands_that_are_slices(M, N, K):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(M, K + 24, device="cuda", generator=g).to(BF)[:, 8:8 + K]
    w = (torch.randn(N, K + 40, device="cuda", generator=g) * 0.05).to(BF)[:, 16:16 + K]
    for wide in (8, 3):
        check_every_epilogue(a, w, M, N, K, wide)


# the handing product's inner size and the taking product's K: rings of warps and bulk copies on both sides
@pytest.mark.parametrize("N", [1032, 9490])
@pytest.mark.parametrize("M,hidden,inter", [(1, 1024, 2048), (8, 2048, 8192), (9, 3072, 4096), (16, 2048, 1024), (8, 2048, 5632), (13, 1024, 768),
                                            (8, 1280, 11008), (8, 4096, 2048), (3, 6144, 1024)])
def test_norm_handed_over(M, hidden, inter, N):
    from inf_engine_b200 import kernels
    g = torch.Generator("cuda").manual_seed(M + hidden)
    h = torch.randn(M, inter, device="cuda", generator=g).to(BF)
    wd = (torch.randn(hidden, inter, device="cuda", generator=g) * 0.03).to(BF)
    wq = (torch.randn(N, hidden, device="cuda", generator=g) * 0.03).to(BF)
    for gain_dtype in (BF, torch.float32):
        gain = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).to(gain_dtype)
        res = torch.randn(M, hidden, device="cuda", generator=g)
        want = res.double() + h.double() @ wd.double().T
        xg = torch.full((M, hidden), float("nan"), device="cuda", dtype=BF)
        ssq = torch.full((kernels.SSQ_SLOT, kernels.sm_count()), float("nan"), device="cuda")
        kernels.gemm_stream(h, wd, res, M, "residual", normout=(xg, gain, ssq))
        assert bool(((res.double() - want).abs() <= bound(h, wd, inter) + 2.0 ** -23 * want.abs()).all())
        assert torch.equal(xg, (res * gain.float()).to(BF))
        assert torch.allclose(ssq[:M].double().sum(1), (res.double() ** 2).sum(1), rtol=1e-5)
        out = torch.full((M, N), float("nan"), device="cuda")
        kernels.gemm_stream(res, wq, out, M, "f32", eps=1e-5, prenormed=(xg, ssq))
        inv = 1.0 / torch.sqrt((res.double() ** 2).mean(1, keepdim=True) + 1e-5)
        ref = (xg.double() @ wq.double().T) * inv
        assert bool(((out.double() - ref).abs() <= bound(xg, wq, hidden) * inv + 1e-6 * ref.abs()).all())
        half = torch.full((M, N), float("nan"), device="cuda", dtype=BF)
        kernels.gemm_stream(res, wq, half, M, "bf16", eps=1e-5, prenormed=(xg, ssq))
        assert torch.equal(half, out.to(BF))
        act = torch.full((M, N // 2), float("nan"), device="cuda", dtype=BF)
        kernels.gemm_stream(res, wq, act, M, "silu_mul", eps=1e-5, prenormed=(xg, ssq))
        want = gated(out, (1.0, float("inf"), 0.0, 0.0))
        assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())
    torch.cuda.synchronize()
    assert kernels.stream_error() == 0
