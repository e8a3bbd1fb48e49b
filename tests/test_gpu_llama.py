"""The Llama-shaped decoder driver (full-decoder configuration) on a small shape: the AlignedKV cache on every layer
against the same weights with dense fp16 torch attention.  The aligned path is an approximation (skipped nibble planes,
fp16 accumulation in the reference's order), so logits are compared with a max-norm relative tolerance of 5e-2 and the
greedy tokens must agree for a clear majority of steps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kv_heads,v_mode", [(4, "exact"), (2, "order_free")])
def test_decoder_matches_dense_attention(akv_lib, kv_heads, v_mode):
    from alignedkv_b200.llama import LlamaConfig, LlamaDecoder
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=kv_heads, vocab_size=1000)
    B, S, new = 2, 150, 6
    ids = torch.randint(0, cfg.vocab_size, (B, S), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    a = LlamaDecoder(cfg, B, S + new + 1, "cuda:0", seed=1, v_mode=v_mode)
    d = LlamaDecoder(cfg, B, S + new + 1, "cuda:0", seed=1, attention="dense")
    la, ld = a.prefill(ids), d.prefill(ids)
    assert torch.equal(la, ld), "the prompt path is the same dense attention in both"
    agree, worst = 0, 0.0
    tok = ld.argmax(-1)
    for _ in range(new):
        la, ld = a.step(tok), d.step(tok)
        err = float((la.float() - ld.float()).abs().max() / ld.float().abs().max())
        worst = max(worst, err)
        agree += int(torch.equal(la.argmax(-1), ld.argmax(-1)))
        tok = ld.argmax(-1)
    print(f"decoder logits: worst max-norm relative error {worst:.2e}; greedy tokens agree in {agree}/{new} steps")
    assert worst <= 5e-2
    assert agree >= new - 2
    assert akv_lib.akv_device_error_flag() == 0


def test_decoder_graph_replay_matches_eager(akv_lib):
    """The decode step with its dense parts replayed from CUDA graphs gives the logits of the eager step."""
    from alignedkv_b200.llama import LlamaConfig, LlamaDecoder
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1024, num_hidden_layers=3, num_attention_heads=4,
                      num_key_value_heads=4, vocab_size=1000)
    B, S, new = 2, 100, 5
    ids = torch.randint(0, cfg.vocab_size, (B, S), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    a = LlamaDecoder(cfg, B, S + new + 1, "cuda:0", seed=2)
    b = LlamaDecoder(cfg, B, S + new + 1, "cuda:0", seed=2)
    tok = a.prefill(ids).argmax(-1)
    assert torch.equal(tok, b.prefill(ids).argmax(-1))
    b.capture_graphs()
    for _ in range(new):
        la, lb = a.step(tok), b.step(tok).clone()
        err = float((la.float() - lb.float()).abs().max() / la.float().abs().max())
        assert err <= 1e-3, err
        tok = la.argmax(-1)
    assert a.pos == b.pos and akv_lib.akv_device_error_flag() == 0


def tensor_step(dec, ids):
    """`LlamaDecoder.step` with torch's operations between the matrix products and the attention."""
    from alignedkv_b200.llama import _rms_norm, _rope, _rope_tables
    F, cfg, B = torch.nn.functional, dec.cfg, dec.B
    H, Hkv, D, eps = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.rms_norm_eps
    tables = _rope_tables(torch.tensor([dec.pos], device=dec.device), D, cfg.rope_theta)
    x = dec.embed[ids.view(B, 1)]
    for p, cache in zip(dec.layers, dec.caches):
        qkv = F.linear(_rms_norm(x, p["norm1"], eps), p["wqkv"]).view(B, 1, H + 2 * Hkv, D)
        qk = _rope(qkv[:, :, :H + Hkv], tables)
        o = cache.decode(qk[:, :, :H].contiguous(), qk[:, :, H:].contiguous(), qkv[:, :, H + Hkv:].contiguous())
        x = torch.addmm(x.view(B, -1), o.reshape(B, -1), p["wo"].t()).view(B, 1, -1)
        gate, up = F.linear(_rms_norm(x, p["norm2"], eps), p["w_gate_up"]).chunk(2, dim=-1)
        x = torch.addmm(x.view(B, -1), F.silu(gate).mul_(up).view(B, -1), p["w_down"].t()).view(B, 1, -1)
    dec.pos += 1
    return F.linear(_rms_norm(x, dec.final_norm, eps), dec.lm_head)[:, 0]


@pytest.mark.parametrize("E,Fi,H,Hkv,B", [(256, 512, 4, 4, 1), (512, 1032, 4, 2, 3), (768, 1000, 4, 4, 5), (1024, 2048, 4, 1, 2),
                                          (4096, 11008, 32, 8, 16)])
def test_step_is_that_of_tensor_operations(akv_lib, E, Fi, H, Hkv, B):
    """Bit for bit: the kernels between the matrix products round as the tensor operations do, in the same order of additions."""
    from alignedkv_b200.llama import LlamaConfig, LlamaDecoder
    cfg = LlamaConfig(hidden_size=E, intermediate_size=Fi, num_hidden_layers=2, num_attention_heads=H, num_key_value_heads=Hkv,
                      vocab_size=1000)
    g = torch.Generator(device="cuda").manual_seed(E)
    S, new = 100, 4
    ids = torch.randint(0, cfg.vocab_size, (B, S + new), device="cuda", generator=g)
    decs = [LlamaDecoder(cfg, B, S + new + 64, "cuda:0", seed=2) for _ in range(3)]
    norms = [(torch.randn(E, device="cuda", generator=g) * 0.3 + 1).half() for _ in range(5)]
    for dec in decs:
        for i, p in enumerate(dec.layers):
            p["norm1"], p["norm2"] = norms[2 * i], norms[2 * i + 1]
        dec.final_norm = norms[4]
        dec.prefill(ids[:, :S])
    decs[1].capture_graphs()
    with torch.no_grad():
        for t in range(new):
            want = tensor_step(decs[2], ids[:, S + t])
            for dec in decs[:2]:
                assert torch.equal(dec.step(ids[:, S + t]).view(torch.int16), want.view(torch.int16))


def test_step_under_autocast(akv_lib):
    """Autocast's type is what the products come out in: fp16 as without it, bf16 is refused by the cache, not misread."""
    from alignedkv_b200.llama import LlamaConfig, LlamaDecoder
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=4,
                      vocab_size=1000)
    ids = torch.randint(0, cfg.vocab_size, (2, 71), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9))
    a, b = (LlamaDecoder(cfg, 2, 128, "cuda:0", seed=4) for _ in range(2))
    for dec in (a, b):
        dec.prefill(ids[:, :70])
    with torch.no_grad(), torch.autocast("cuda", torch.float16):
        assert torch.equal(a.step(ids[:, 70]), tensor_step(b, ids[:, 70]))
    with torch.autocast("cuda", torch.bfloat16), pytest.raises(RuntimeError, match="fp16"):
        a.step(ids[:, 70])
