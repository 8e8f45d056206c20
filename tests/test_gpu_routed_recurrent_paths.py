"""The forms that recurrent blocks and mixtures of experts take by size: runs of tokens side by side, 16-byte rows, block-diagonal
products, experts of a few tokens through the ring, each against float64 or against the form it stands in for."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(seed, *shape):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(DEV).manual_seed(seed))


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,width", [((64, 1, 7, 8, 9), 40), ((511, 512, 513), 16), ((1100, 3), 33), ((32, 31), 8)])
def test_recurrence_in_runs_of_tokens(dtype, lens, width):
    from inf_engine_b200 import kernels as k
    N, R = sum(lens), len(lens)
    u, y, r, i = rnd(1, N, width).to(dtype), rnd(2, N, width).to(dtype), rnd(3, N, width), rnd(4, N, width)
    gates = torch.cat([r, i], 1)
    rb, ib, lam = (0.1 * rnd(5 + j, width) for j in range(3))
    lam += torch.linspace(-7, 1, width, device=DEV)               # decays from 1 - 1e-3 down to e^-10
    state, cuts = rnd(9, R + 1, width), [sum(lens[:j]) for j in range(R + 1)]
    slots = [R - j for j in range(R)]
    slots[1] = -1
    want, ends = torch.zeros(N, width, dtype=torch.float64, device=DEV), state.double()
    for q in range(R):
        if slots[q] >= 0:
            S = state[slots[q]].double()
            for t in range(cuts[q], cuts[q + 1]):
                log_a = -8.0 * torch.sigmoid(r[t].double() + rb.double()) * torch.nn.functional.softplus(lam.double())
                S = torch.exp(log_a) * S + torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(i[t].double() + ib.double()) * u[t].double()
                want[t] = 0.5 * S * torch.nn.functional.gelu(y[t].double(), approximate="tanh")
            ends[slots[q]] = S

    def run(max_q_len, write=True):
        st, out = state.clone(), torch.full((N, width), 3.0, device=DEV).to(dtype)
        k.linear_recurrence(u, y, gates[:, :width], gates[:, width:], rb, ib, lam, st, out, i32(cuts), i32(slots), R, 8.0, 0.5,
                            write_state=write, max_q_len=max_q_len)
        return out, st

    err = lambda a, b: float((a.double() - b).norm() / b.norm())
    out, st = run(max(lens))
    slow, st_slow = run(0)
    # a rounding or two a token, each shrunk by the decays after it; no further off than token after token, give or take
    assert err(st, ends) < 1e-6 and err(st, ends) < 1.5 * err(st_slow, ends) + 1e-7
    assert err(out, want) < (2e-6 if dtype is torch.float32 else 4e-3)
    again, kept = run(max(lens), write=False)
    assert torch.equal(again, out) and torch.equal(kept, state)


@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps,channels", [(2, 8), (3, 264), (4, 512)])
def test_convolution_of_16_byte_rows_keeps_its_bits(w_dtype, taps, channels):
    from inf_engine_b200 import kernels as k
    lens = (1, 2, 70, 8, 129)
    N, R = sum(lens), len(lens)
    rows = rnd(1, N, channels).bfloat16()
    off = torch.zeros(N, channels + 8, device=DEV, dtype=torch.bfloat16)[:, 7:7 + channels]
    off.copy_(rows)
    w, bias, state = rnd(2, channels, taps).to(w_dtype), rnd(3, channels).to(w_dtype), rnd(4, R + 1, taps - 1, channels).bfloat16()
    cuts, slots = i32([sum(lens[:j]) for j in range(R + 1)]), i32([3, -1, 0, 5, 1])
    got = []
    for x in (rows, off):                                 # rows on 16 bytes, rows off them
        st, out = state.clone(), torch.empty(N, channels, device=DEV, dtype=torch.bfloat16)
        k.causal_conv(x, w, bias, st, out, cuts, slots, R, activation="silu", max_q_len=max(lens), in_runs=True)
        got.append((out, st))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("a_dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("m,blocks,n,kk", [(1, 3, 24, 20), (8, 8, 256, 256), (13, 2, 40, 132), (16, 4, 128, 64), (17, 2, 128, 64),
                                           (128, 4, 128, 128), (200, 2, 256, 64)])
def test_block_diagonal(a_dtype, w_dtype, m, blocks, n, kk):
    from inf_engine_b200 import kernels as k
    a, w = rnd(1, m, blocks * kk).to(a_dtype), rnd(2, blocks, n, kk).to(w_dtype)
    out = torch.zeros(m, blocks * n + 4, device=DEV)
    k.block_diagonal(a, w, out[:, 4:])
    x = a.double().view(m, blocks, kk)
    want = torch.einsum("mbk,bnk->mbn", x, w.double()).reshape(m, -1)
    bound = (kk + 8) * 2.0 ** -24 * torch.einsum("mbk,bnk->mbn", x.abs(), w.double().abs()).reshape(m, -1)
    assert bool(((out[:, 4:].double() - want).abs() <= bound).all()) and float(out[:, :4].abs().sum()) == 0


@pytest.mark.parametrize("m,blocks,n,kk", [(8, 2, 256, 256), (128, 3, 128, 64), (200, 5, 128, 128), (300, 4, 256, 256), (513, 2, 512, 512)])
def test_gates_are_no_further_off_than_float32_multiply_adds(m, blocks, n, kk):
    """Gate products drive a recurrence, and the tensor cores cut bits off at every step of an accumulator: whatever form takes
    them, the error against 64 bits is no larger than the tile kernel's (a relative 2-norm over 32,000 values and more, so
    chance moves it by a few per cent)."""
    from inf_engine_b200 import kernels as k
    a, w = rnd(1, m, blocks * kk).bfloat16(), (0.05 * rnd(2, blocks, n, kk)).bfloat16()
    want = torch.einsum("mbk,bnk->mbn", a.double().view(m, blocks, kk), w.double()).reshape(m, -1)
    got, tiles = torch.empty(m, blocks * n, device=DEV), torch.empty(m, blocks * n, device=DEV)
    k.block_diagonal(a, w, got)
    k.gemm_simt_batched(a, w, tiles)
    err = [float((x.double() - want).norm() / want.norm()) for x in (got, tiles)]
    assert err[0] <= 1.05 * err[1], err


@pytest.mark.parametrize("m,n,kk", [(512, 17, 2048), (515, 3, 1000), (520, 40, 33)])
def test_router_rows_do_not_depend_on_their_number(m, n, kk):
    from inf_engine_b200 import kernels as k
    a, w = rnd(1, m, kk).bfloat16(), rnd(2, n, kk).bfloat16()
    many, few = torch.empty(m, n, device=DEV), torch.empty(9, n, device=DEV)
    k.gemm_rowdot(a, w, many)
    k.gemm_rowdot(a[m - 9:], w, few)
    assert torch.equal(many[m - 9:], few)
    bound = (kk / 32 + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((many.double() - a.double() @ w.double().T).abs() <= bound).all())


@pytest.mark.parametrize("n_pairs,experts,rows", [(1, 1, 16), (40, 33, 16), (300, 70, 64), (4096, 16, 128), (64, 5, 3)])
def test_sort_names_every_pair_once(n_pairs, experts, rows):
    from inf_engine_b200 import kernels as k
    ids = torch.randint(0, experts, (n_pairs, 1), generator=torch.Generator().manual_seed(n_pairs))
    ids[ids == experts // 2] = 0                          # an expert that nobody chose
    dev, order = ids.int().to(DEV), torch.full((n_pairs,), -1, dtype=torch.int32, device=DEV)
    tiles = torch.full((k.moe_max_tiles(n_pairs, experts, rows), 4), 9, dtype=torch.int32, device=DEV)
    k.moe_sort(dev, experts, order, tiles, rows)
    order, tiles, flat = order.cpu().long(), tiles.cpu(), ids.view(-1)
    assert sorted(order.tolist()) == list(range(n_pairs)) and bool((flat[order][1:] >= flat[order][:-1]).all())
    at, used = 0, int(tiles[0, 3])
    for e, pos, n, _ in tiles[:used].tolist():
        assert pos == at and 0 < n <= rows and bool((flat[order[pos:pos + n]] == e).all())
        assert n == rows or pos + n == n_pairs or int(flat[order[pos + n]]) != e      # only an expert's last tile is short
        at += n
    assert at == n_pairs and bool((tiles[used:] == 0).all()) if used > 0 else n_pairs == 0


@pytest.mark.parametrize("epi", ["silu_mul", "relu2"])
@pytest.mark.parametrize("tokens,experts,top,hidden,inter", [(1, 4, 1, 256, 256), (8, 16, 2, 512, 256), (16, 3, 2, 256, 1280), (11, 40, 4, 1024, 512)])
def test_experts_of_a_few_tokens_through_the_ring(epi, tokens, experts, top, hidden, inter):
    from inf_engine_b200 import kernels as k
    x, wide = rnd(1, tokens, hidden).bfloat16(), 2 * inter if epi == "silu_mul" else inter
    first, down = (0.05 * rnd(2, experts, wide, hidden)).bfloat16(), (0.05 * rnd(3, experts, hidden, inter)).bfloat16()
    g = torch.Generator().manual_seed(tokens)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(tokens)])
    ids[:] = ids[0] if experts == 3 else ids              # every token with the same experts: tiles of 16 rows
    dev, n = ids.int().to(DEV), tokens * top
    order = torch.empty(n, dtype=torch.int32, device=DEV)
    tiles = torch.empty(k.moe_max_tiles(n, experts, k.MOE_RING_ROWS), 4, dtype=torch.int32, device=DEV)
    k.moe_sort(dev, experts, order, tiles, k.MOE_RING_ROWS)
    act = k.glu_constants("silu") if epi == "silu_mul" else None
    h, y = torch.empty(n, inter, device=DEV, dtype=torch.bfloat16), torch.full((n, hidden), 9.0, device=DEV)
    assert k.moe_ring_supports(x, hidden, inter)
    k.moe_gemm_ring(x, first, h, order, tiles, top, gather=True, scatter=False, epi=epi, act=act)
    k.moe_gemm_ring(h, down, y, order, tiles, top, gather=False, scatter=True)
    for p, e in enumerate(ids.view(-1).tolist()):
        z = x[p // top].double() @ first[e].double().T
        z = torch.nn.functional.silu(z[0::2]) * z[1::2] if epi == "silu_mul" else torch.relu(z) ** 2
        at = int((order == p).nonzero())
        assert bool(((h[at].double() - z).abs() <= 2.0 ** -8 * z.abs() + 2e-5).all())
        want, size = h[at].double() @ down[e].double().T, h[at].double().abs() @ down[e].double().abs().T
        assert bool(((y[p].double() - want).abs() <= (inter / 16 + 16) * 2.0 ** -24 * size).all())
    assert k.stream_error() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,d,top,shared,gated", [(1, 8, 1, True, True), (3, 2048, 2, True, True), (2, 2056, 3, False, False), (2, 8192, 2, True, True),
                                                  (5, 64, 2, True, True), (3, 256, 3, True, True), (2, 264, 1, False, False)])
def test_mixture_normed_into_the_stream(dtype, n, d, top, shared, gated):
    from inf_engine_b200 import kernels as k
    y, w, res = rnd(1, n * top, d), rnd(2, n, top).abs(), rnd(3, n, d)
    gate, sh = (rnd(4, n).sigmoid() if gated else None), (rnd(5, n, d).to(dtype) if shared else None)
    gain = (1 + 0.1 * rnd(6, d)).to(dtype)
    row = (w[:, :, None].double() * y.view(n, top, d).double()).sum(1) + (gate[:, None].double() * sh.double() if shared else 0)
    want = res.double() + row / torch.sqrt((row * row).mean(-1, keepdim=True) + 1e-5) * gain.double()
    got, nxt = res.clone(), torch.empty(n, d, device=DEV, dtype=dtype)
    k.moe_combine_outnorm(got, y, w, gate, sh, gain, 1e-5, nxt)
    assert bool(((got.double() - want).abs() <= 3e-6 * (1 + want.abs())).all()) and torch.equal(nxt, got.to(dtype))
    plain, out = res.clone(), torch.empty(n, d, device=DEV)
    k.moe_combine(y, w, gate, sh, out)
    k.outnorm_accumulate(plain, out, gain, 1e-5)
    assert torch.equal(plain, got)


@pytest.mark.parametrize("off", [0, 1])
def test_a_gain_that_starts_off_16_bytes(off):
    """A norm's gain may be any piece of a program's memory; the kernel with the mixture's sum in it wants 16-byte rows."""
    from types import SimpleNamespace
    from inf_engine_b200.parts.norms import RMSNorm
    from inf_engine_b200.parts.runtime import Runtime
    n, d, top = 3, 512, 2
    flat = (1 + 0.1 * rnd(6, d + 8)).bfloat16()
    norm = RMSNorm(SimpleNamespace(weight="w", eps=1e-5, size=d), {"w": flat[off:off + d]}, Runtime("cuda:0", torch.bfloat16))
    y, w, res = rnd(1, n * top, d), rnd(2, n, top).abs(), rnd(3, n, d)
    row = (w[:, :, None].double() * y.view(n, top, d).double()).sum(1)
    want = res.double() + row / torch.sqrt((row * row).mean(-1, keepdim=True) + 1e-5) * norm.gain.double()
    got = res.clone()
    norm.accumulate_mixture(got, (y, w, None, None))
    assert bool(((got.double() - want).abs() <= 3e-6 * (1 + want.abs())).all())
