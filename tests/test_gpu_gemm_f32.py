"""The float32 product's two kernels (rows streamed for up to 16, tiles beyond) against float64, at the edges of their tiles,
and the promise that a row's result depends neither on its neighbours nor on the kernel that took it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around the kernels' limits (4, 8, 16, 32, 64), columns around a group of 32 / 64 and a tile of 128, K from the smallest
# with runs that are short or empty, weights enough for each way of laying the stream out (fewer groups than SMs, more, many)
@pytest.mark.parametrize("M,N,K", [(1, 8, 512), (4, 33, 516), (5, 131, 1028), (8, 4768, 548), (9, 4736, 512), (16, 63, 1028),
                                   (17, 131, 580), (3, 18999, 516), (8, 18976, 512), (13, 18977, 512), (32, 300, 512),
                                   (33, 129, 2048), (65, 257, 900), (64, 128, 8192), (130, 19000, 516), (40, 100, 508)])
def test_rows_and_tiles_follow_one_order_of_sums(M, N, K):
    from inf_engine_b200 import kernels as k
    g = torch.Generator("cuda").manual_seed(M * 1000 + N + K)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    out = torch.full((M, N), float("nan"), device="cuda")
    k.gemm_simt(a, w, out)
    # a run of ceil(K / 8) products in two accumulators, one sum of the two and eight of the runs, each rounded once
    steps = -(-K // 16) + 32 + 1 + 8
    bound = steps * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - a.double() @ w.double().T).abs() <= bound).all())
    for rows in (slice(M // 2, M // 2 + 1), slice(0, min(M, 7)), slice(0, min(M, 40))):
        part = torch.empty(rows.stop - rows.start, N, device="cuda")
        k.gemm_simt(a[rows], w, part)
        assert torch.equal(part, out[rows])
    wide = torch.full((M, N + 3), 2.0, device="cuda")
    k.gemm_simt(a, w, wide[:, 3:])
    assert torch.equal(wide[:, 3:], out) and bool((wide[:, :3] == 2.0).all())
