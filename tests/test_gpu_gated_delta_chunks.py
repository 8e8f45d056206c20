"""The gated delta rule in chunks of 64 tokens against float64, token after token: lengths around a chunk's edges, several
requests, a padding row without a slot, a state that is only read; its error beside the token-by-token kernel's.  Key sizes of
every kind: eight and four groups of threads, a last pass over the rows of the state that is part empty, one pass and two."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def plain(q, k, v, b, a, gate, a_log, dt_bias, gain, S, G):
    n, H, dv = v.shape
    dk = q.shape[-1]
    q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5).repeat_interleave(H // G, 1)
    k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    g = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(a + dt_bias))
    out = []
    for t in range(n):
        S = S * g[t, :, None, None]
        u = torch.sigmoid(b[t])[:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        o = torch.einsum("hkv,hk->hv", S, q[t])
        out.append(o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * gain * torch.nn.functional.silu(gate[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dk,dv,H,G,lens", [(64, 64, 4, 2, (1, 64, 65, 7, 200)), (64, 128, 2, 1, (63, 130)), (128, 128, 2, 2, (129, 2)),
                                             (32, 128, 4, 2, (130, 3)), (48, 48, 2, 1, (66, 2)), (80, 32, 3, 3, (129, 5)),
                                             (96, 96, 2, 1, (70, 64))])
def test_chunks_against_the_recurrence(dtype, dk, dv, H, G, lens):
    from inf_engine_b200 import kernels
    g = torch.Generator("cuda").manual_seed(sum(lens) + dk)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    R, N = len(lens), sum(lens)
    cuts = [0]
    for n in lens:
        cuts.append(cuts[-1] + n)
    qk, v, ba, gate = (rnd(N, w).to(dtype) for w in (2 * G * dk, H * dv, 2 * H, H * dv))
    a_log, dt_bias = torch.linspace(-4, 0.5, H, device="cuda").to(dtype), torch.linspace(-3, 1, H, device="cuda").to(dtype)
    gain = (1 + 0.1 * rnd(dv)).to(dtype)
    state = 0.3 * rnd(R + 1, H, dk, dv)
    slots = [R - i for i in range(R)]
    slots[1] = -1                                  # a padding row: zeros come out, no state is touched
    want, ends = torch.zeros(N, H * dv, dtype=torch.float64, device="cuda"), {}
    for r in range(R):
        if slots[r] >= 0:
            x = slice(cuts[r], cuts[r + 1])
            d = lambda t, *s: t[x].double().view(lens[r], *s)
            o, S = plain(d(qk[:, :G * dk], G, dk), d(qk[:, G * dk:], G, dk), d(v, H, dv), d(ba[:, :H], H), d(ba[:, H:], H),
                         d(gate, H, dv), a_log.double(), dt_bias.double(), gain.double(), state[slots[r]].double(), G)
            want[x], ends[slots[r]] = o.reshape(lens[r], -1), S
    starts, slot_ids = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in (cuts, slots))
    floats = kernels.gated_delta_scratch_floats(N, R, H, dk, dv)

    def run(scratch, write=True):
        st, out = state.clone(), torch.full((N, H * dv), 7.0, device="cuda").to(dtype)
        kernels.gated_delta(qk[:, :G * dk], qk[:, G * dk:], v, ba[:, :H], ba[:, H:], gate, a_log, dt_bias, gain, st, out, starts,
                            slot_ids, R, H, G, dk, dv, 1e-6, 1e-5, write_state=write, scratch=scratch, max_q_len=max(lens))
        return out, st

    out, st = run(torch.full((floats,), float("nan"), device="cuda"))
    err = lambda x, y: float((x.double() - y).norm() / y.norm())
    # float32 sums of up to 128 products, three in a row, and a recurrence that shrinks what it carries: a few 2^-24 each
    # (2.6e-7 measured on the outputs, 2.3e-7 on the state; a chunk's term left out shows at 1e-2); bfloat16 rounds the result
    assert err(out, want) < (1.5e-6 if dtype is torch.float32 else 4e-3)
    for s, S in ends.items():
        assert err(st[s], S) < 1.5e-6, s
    for s in set(range(R + 1)) - set(ends):
        assert torch.equal(st[s], state[s])
    other, _ = run(None)
    assert err(out, other.double()) < (3e-6 if dtype is torch.float32 else 6e-3)
    again, kept = run(torch.full((floats,), float("nan"), device="cuda"), write=False)
    assert torch.equal(again, out) and torch.equal(kept, state)


def inputs(H, G, dk, dv, N, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    qk, v, ba, gate = (torch.randn(N, w, device="cuda", generator=g) for w in (2 * G * dk, H * dv, 2 * H, H * dv))
    return {"qk": qk, "v": v, "ba": ba, "gate": gate, "a_log": torch.linspace(-4, 0.5, H, device="cuda"),
            "dt_bias": torch.linspace(-3, 1, H, device="cuda"), "gain": 1 + 0.1 * torch.randn(dv, device="cuda", generator=g),
            "state": 0.3 * torch.randn(1, H, dk, dv, device="cuda", generator=g)}


def both_forms(x, H, G, dk, dv):
    """(outputs [N, H, dv], state) in chunks, and token after token"""
    from inf_engine_b200 import kernels
    N, got = len(x["v"]), []
    for floats in (kernels.gated_delta_scratch_floats(N, 1, H, dk, dv), 0):
        st, out = x["state"].clone(), torch.empty(N, H * dv, device="cuda")
        at, slot = torch.tensor([0, N], dtype=torch.int32, device="cuda"), torch.tensor([0], dtype=torch.int32, device="cuda")
        kernels.gated_delta(x["qk"][:, :G * dk], x["qk"][:, G * dk:], x["v"], x["ba"][:, :H], x["ba"][:, H:], x["gate"], x["a_log"],
                            x["dt_bias"], x["gain"], st, out, at, slot, 1, H, G, dk, dv, 1e-6, 1e-5,
                            scratch=torch.zeros(floats, device="cuda") if floats else None, max_q_len=N)
        got.append((out.view(N, H, dv), st))
    return got


def test_a_decay_of_zero():
    """A log decay that overflows to minus infinity empties the state, and both forms go on from there."""
    H, G, dk, dv, N = 4, 2, 64, 64, 150
    x = inputs(H, G, dk, dv, N, 5)
    x["a_log"][1] = 100.0                         # its exp overflows: every token of the head
    x["ba"][[0, 40, 41, 130], H + 2] = 3e38       # the product with the rate overflows: these tokens
    (out, st), (want, want_st) = both_forms(x, H, G, dk, dv)
    assert bool(torch.isfinite(want).all()) and bool(torch.isfinite(out).all()) and bool(torch.isfinite(st).all())
    for h in range(H):                            # as far apart as the two orders of sums (see above)
        assert float((out[:, h] - want[:, h]).norm() / want[:, h].norm()) < 3e-6, h
        assert float((st[:, h] - want_st[:, h]).norm() / want_st[:, h].norm()) < 3e-6, h


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_token_that_is_no_number_spoils_no_earlier_one(value):
    H, G, dk, dv, N, at = 2, 1, 64, 64, 130, 100
    clean = inputs(H, G, dk, dv, N, 6)
    want = both_forms(clean, H, G, dk, dv)[1][0]
    x = dict(clean, v=clean["v"].clone())
    x["v"][at, 3] = value                         # one value channel of the first head, in the middle of a chunk
    out = both_forms(x, H, G, dk, dv)[0][0]
    assert bool(torch.isnan(out[at, 0, 3])) and bool(torch.isfinite(out[:at]).all()) and bool(torch.isfinite(out[:, 1]).all())
    assert float((out[:at] - want[:at]).norm() / want[:at].norm()) < 3e-6
    assert float((out[:, 1] - want[:, 1]).norm() / want[:, 1].norm()) < 3e-6
