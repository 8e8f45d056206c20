"""A block per (token, head) for decode tokens in float32 arithmetic gives the tile kernel's bits: head sizes with and without
16-byte rows, pages, windows, score options, key counts around a tile of 32 and around what a block holds at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hk,hd,hdv,ps,window,extras", [(8, 2, 64, 64, 16, None, False), (6, 2, 32, 32, 8, 40, True), (3, 1, 48, 48, 16, None, True),
                                                          (4, 4, 20, 12, 4, None, False), (4, 1, 128, 256, 16, 70, False)])
def test_same_bits_as_the_tile_kernel(dtype, H, Hk, hd, hdv, ps, window, extras):
    from inf_engine_b200 import kernels as k
    g = torch.Generator("cuda").manual_seed(hd + H)
    group = H // Hk
    ctx, lens = [0, 31, 32, 255, 256, 700, 5, 33], [1, 1, 1, 1, 1, 1, 16 // group, 40]
    R, N = len(lens), sum(lens)
    pages = [-(-(c + n) // ps) for c, n in zip(ctx, lens)]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((R, max(pages)), -1, dtype=torch.int32)
    for r, n in enumerate(pages):
        table[r, :n] = torch.tensor([order.pop() for _ in range(n)])
    kp, vp = (torch.randn(sum(pages), Hk, ps, d, device="cuda", generator=g).to(dtype) for d in (hd, hdv))
    q = torch.randn(N, H * hd, device="cuda", generator=g).to(dtype)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    starts = [sum(lens[:r]) for r in range(R + 1)]
    bias = 0.1 * torch.randn(H, 50, device="cuda", generator=g) if extras else None
    scale = 1 + 0.2 * torch.rand(H, device="cuda", generator=g) if extras else None
    work = [(r, p) for r, n in enumerate(lens) for p in range(0, n * group, 32)]
    whole, rows = (torch.full((N, H * hdv), 5.0, device="cuda").to(dtype) for _ in range(2))
    k.attention_general(q, whole, kp, vp, table.cuda(), i32(starts), i32(ctx), i32([w[0] for w in work]), i32([w[1] for w in work]),
                        len(work), H, Hk, hd, ps, window, hd ** -0.5, bias, scale, hdv)
    k.attention_ordered_rows(q, rows, kp, vp, table.cuda(), i32(starts), i32(ctx), R, 16, H, Hk, hd, ps, window, hd ** -0.5, bias, scale, hdv)
    few = starts[-2]                               # the last request brings more rows than 16: it is left alone
    assert torch.equal(rows[:few], whole[:few]) and bool((rows[few:] == 5.0).all())
