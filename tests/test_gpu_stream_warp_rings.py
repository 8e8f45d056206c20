"""The streaming product's rings of warps: rows on both sides of 8, every K form (activations in registers whole, or a stage ahead),
columns that end inside a unit of 8 or 16 rows, more and fewer units than SMs, every epilogue, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def bound(a, w, k):
    """Exact products, each of k sums rounded once (to float32; the tensor core's own sums of 16 may be cut instead of rounded)."""
    return 2 * k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("K", [1024, 2048, 3072, 4096, 6144, 8192])
@pytest.mark.parametrize("M,N", [(1, 5), (8, 1189), (9, 2056), (16, 9490), (7, 19001)])
def test_stores_against_float64(M, N, K):
    from inf_engine_b200 import kernels
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(BF)
    ref, most = a.double() @ w.double().T, bound(a, w, K)
    out = torch.full((M, N), float("nan"), device="cuda")
    kernels.gemm_stream(a, w, out, M, "f32")
    assert bool(((out.double() - ref).abs() <= most).all())
    half = torch.full((M, N), float("nan"), device="cuda", dtype=BF)
    kernels.gemm_stream(a, w, half, M, "bf16")
    assert torch.equal(half, out.to(BF))
    total = torch.randn(M, N, device="cuda", generator=g)
    start = total.clone()
    kernels.gemm_stream(a, w, total, M, "residual")
    assert torch.equal(total, start + out)
    if N % 2 == 0:
        act = torch.full((M, N // 2), float("nan"), device="cuda", dtype=BF)
        kernels.gemm_stream(a, w, act, M, "silu_mul")
        gate, up = out[:, 0::2].double(), out[:, 1::2].double()
        want = gate * torch.sigmoid(gate) * up
        assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())


@pytest.mark.parametrize("M,hidden,inter", [(1, 1024, 2048), (8, 2048, 8192), (9, 3072, 4096), (16, 2048, 1024)])
def test_norm_handed_over(M, hidden, inter):
    from inf_engine_b200 import kernels
    g = torch.Generator("cuda").manual_seed(M + hidden)
    h = torch.randn(M, inter, device="cuda", generator=g).to(BF)
    wd = (torch.randn(hidden, inter, device="cuda", generator=g) * 0.03).to(BF)
    wq = (torch.randn(1031, hidden, device="cuda", generator=g) * 0.03).to(BF)
    gain = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).to(BF)
    res = torch.randn(M, hidden, device="cuda", generator=g)
    want = res.double() + h.double() @ wd.double().T
    xg = torch.full((M, hidden), float("nan"), device="cuda", dtype=BF)
    ssq = torch.full((kernels.SSQ_SLOT, kernels.sm_count()), float("nan"), device="cuda")
    kernels.gemm_stream(h, wd, res, M, "residual", normout=(xg, gain, ssq))
    assert bool(((res.double() - want).abs() <= bound(h, wd, inter) + 2.0 ** -23 * want.abs()).all())
    assert torch.equal(xg, (res * gain.float()).to(BF))
    out = torch.full((M, 1031), float("nan"), device="cuda")
    kernels.gemm_stream(res, wq, out, M, "f32", eps=1e-5, prenormed=(xg, ssq))
    inv = 1.0 / torch.sqrt((res.double() ** 2).mean(1, keepdim=True) + 1e-5)
    ref = (xg.double() @ wq.double().T) * inv
    assert bool(((out.double() - ref).abs() <= bound(xg, wq, hidden) * inv + 1e-6 * ref.abs()).all())
