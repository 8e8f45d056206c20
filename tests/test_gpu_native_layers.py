"""A step through all plain pre-norm layers issued natively gives the bits of the parts one by one: portions on each attention
kernel, mixed with decode tokens, below and above the tiles of the gated product, heads of 64 and 128, a window, untied heads."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BASE = {"architectures": ["LlamaForCausalLM"], "hidden_act": "silu", "rms_norm_eps": 1e-5, "max_position_embeddings": 1024, "vocab_size": 500,
        "rope_theta": 10000.0, "rope_scaling": None}


def runner(head_dim, heads, kv, tie, window=None, seed=0):
    import dataclasses
    from inf_engine_b200 import ModelRunner, parse_config_dict
    cfg = dict(BASE, num_hidden_layers=3, hidden_size=256, num_attention_heads=heads, num_key_value_heads=kv, head_dim=head_dim,
               intermediate_size=512, tie_word_embeddings=tie)
    g = torch.Generator("cuda").manual_seed(seed)
    w = lambda *s: (0.05 * torch.randn(*s, device="cuda", generator=g)).bfloat16()
    t = {"model.embed_tokens.weight": w(500, 256), "model.norm.weight": 1 + w(256)}
    if not tie:
        t["lm_head.weight"] = w(500, 256)
    for i in range(3):
        p = f"model.layers.{i}."
        for n, s in (("self_attn.q_proj", (heads * head_dim, 256)), ("self_attn.k_proj", (kv * head_dim, 256)), ("self_attn.v_proj", (kv * head_dim, 256)),
                     ("self_attn.o_proj", (256, heads * head_dim)), ("mlp.gate_proj", (512, 256)), ("mlp.up_proj", (512, 256)), ("mlp.down_proj", (256, 512))):
            t[p + n + ".weight"] = w(*s)
        t[p + "input_layernorm.weight"], t[p + "post_attention_layernorm.weight"] = 1 + w(256), 1 + w(256)
    cfg = parse_config_dict(cfg)
    spec = cfg.model_spec()
    spec = dataclasses.replace(spec, layers=tuple(dataclasses.replace(x, mixer=dataclasses.replace(x.mixer, window=window)) for x in spec.layers))
    return ModelRunner(cfg, t, "bfloat16", page_size=16, n_pages=128, max_requests=8, spec=spec)


@pytest.mark.parametrize("head_dim,heads,kv,tie,window", [(64, 4, 2, True, None), (128, 2, 1, False, None), (64, 4, 4, False, None),
                                                          (64, 4, 2, False, 70)])
def test_native_layers_give_the_same_bits(head_dim, heads, kv, tie, window, monkeypatch):
    from inf_engine_b200 import StepEntry, kernels
    from inf_engine_b200.parts import prenorm_layers
    runs = []
    for native in (True, False):
        r = runner(head_dim, heads, kv, tie, window)
        assert r.model._native is not None
        if not native:
            r.model._native = None
        # what the step through all layers would launch, as it deals the attention out
        kinds = []
        if native:
            issue = kernels.prenorm_layers

            def seen(layers, n, step):
                st = prenorm_layers._Step.from_address(step)
                kinds.append((bool(st.attn_small), bool(st.attn_tc), bool(st.attn_mma), bool(st.rotate_q), bool(st.gemm_silu)))
                issue(layers, n, step)

            monkeypatch.setattr(kernels, "prenorm_layers", seen)
        ids = torch.randint(0, 500, (900,), generator=torch.Generator().manual_seed(1)).tolist()
        for rid in "abcdef":
            r.open(rid)
        # a prompt below 128 rows (mma tiles), long ones alone (tcgen05 tiles, which rotate q themselves), one beside a portion of at
        # most 16 rows, a portion of few rows, portions beside decode tokens, portions of at most 16 rows alone
        steps = [[("a", 61)], [("e", 300)], [("e", 140), ("f", 200)], [("b", 200), ("c", 3)], [("a", 30)], [("a", 1), ("b", 90), ("c", 1), ("d", 17)],
                 [("a", 4), ("b", 4), ("c", 4), ("d", 5)]]
        out, at, launches = [], {}, []
        for step in steps:
            es = []
            for rid, n in step:
                k = at.get(rid, 0)
                es.append(StepEntry(rid, ids[k:k + n], [n - 1]))
                at[rid] = k + n
            before = kernels.LAUNCHES
            out.append(r.step(es).clone())
            launches.append(kernels.LAUNCHES - before)
        if native:
            monkeypatch.setattr(kernels, "prenorm_layers", issue)
            want = {(False, False, True), (False, True, False), (True, True, False), (True, False, False)} if window is None else \
                {(False, False, True), (True, False, True), (True, False, False)}
            assert want <= {k[:3] for k in kinds} and {k[3] for k in kinds} == ({True, False} if window is None else {True})
            assert {k[4] for k in kinds} == {True, False}
        runs.append((out, [v.k.clone() for v in r.model._views], [v.v.clone() for v in r.model._views], launches))
    for x, y in zip(*runs):
        for u, v in zip(x, y):
            assert torch.equal(u, v) if isinstance(u, torch.Tensor) else u == v
