"""A decode step of a cache without a quantized block (one launch) against float64, and what it leaves behind."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,G,D,P", [(1, 1, 1, 64, 1), (2, 3, 1, 128, 28), (1, 4, 2, 128, 31), (3, 2, 4, 128, 32), (2, 2, 8, 256, 62),
                                       (1, 5, 1, 192, 33), (40, 32, 1, 128, 7)])
@pytest.mark.parametrize("append,packed,masked,mode", [(True, False, False, "exact"), (True, False, True, "exact"),
                                                       (False, True, False, "exact"), (True, True, False, "order_free")])
def test_small_step(akv_lib, B, H, G, D, P, append, packed, masked, mode):
    from alignedkv_b200.decode import DecodeLayer
    if mode == "order_free" and D != 128:
        pytest.skip("order-free P.V has head_dim 128")
    g = torch.Generator(device="cuda").manual_seed(P)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()  # noqa: E731
    k, v, q, k1, v1 = r(B, P, H, D), r(B, P, H, D), r(B, 1, H * G, D) * 2, r(B, 1, H, D) * 4, r(B, 1, H, D)
    layer = DecodeLayer(B, 128, H, D, "cuda:0", n_q_heads=H * G, v_mode=mode)
    layer.prefill(k, v)
    n = P + int(append)
    mask = None
    if masked:
        mask = torch.zeros(B, 1, 1, n, device="cuda", dtype=torch.half)
        mask[0, :, :, :n // 2] = torch.finfo(torch.half).min
    before = akv_lib.akv_launch_count()
    args = (q, k1, v1) if append else (q,)
    got = layer.decode(*args, append=append, packed=packed, mask=mask)
    assert akv_lib.akv_launch_count() - before == 1
    kk, vv = (torch.cat([a, b], 1) if append else a for a, b in ((k, k1), (v, v1)))
    assert torch.equal(layer.restk[:, :n], kk) and torch.equal(layer.restv[:, :n], vv)
    field = lambda t: (t.contiguous().view(torch.int16) >> 10).to(torch.uint8) & 0x1F  # noqa: E731
    for have, prompt, new in ((layer.k_exp_max, k, k1), (layer.v_exp_max, v, v1)):
        want = field(prompt.max(dim=1, keepdim=True).values)
        assert torch.equal(have, torch.maximum(want, field(new)) if append else want)
    kd, vd = (t.repeat_interleave(G, 2).double() for t in (kk, vv))
    s = torch.einsum("bhd,bnhd->bhn", q[:, 0].double(), kd) / math.sqrt(D)
    if masked:
        s = s + mask[:, 0].double()
    p = torch.softmax(s, -1)
    o = torch.einsum("bhn,bnhd->bhd", p, vd)
    # scores are rounded to fp16 up to three times (half a step of 2^-10 each), which moves exponents by d = 3 * 2^-11 |score|
    # and probabilities by 2.2 d relative; a probability is then rounded once (or to 2^-25), the output up to twice
    off = 2.2 * 3 * 2 ** -11 * torch.where(s < -1e4, 0.0, s).abs().amax(-1, keepdim=True)
    # (|score| up to 30 and more for the scaled keys: the bound is stated for the sum of |p v|)
    bound = (torch.expm1(off) + 2 ** -11) * torch.einsum("bhn,bnhd->bhd", p, vd.abs()) + n * 2 ** -25 * vd.abs().amax() + 2 ** -10 * o.abs() + 2 ** -20
    if packed:
        rec = got.view(B, H * G, D + 2).double()
        got = rec[..., 2:]
        assert bool(((rec[..., 0] - s.amax(-1)).abs() <= 2 * 2 ** -10 * s.abs().amax(-1) + 2 ** -14).all())
    else:
        got = got[:, 0].double()
    assert bool(((got - o).abs() <= bound).all())


@pytest.mark.parametrize("B,H,G,D,P", [(1, 1, 1, 64, 1), (2, 3, 1, 128, 28), (1, 4, 2, 128, 31), (3, 2, 4, 128, 32), (2, 2, 8, 256, 61),
                                       (1, 5, 1, 192, 33), (40, 32, 1, 128, 7)])
@pytest.mark.parametrize("append,packed,masked,mode", [(True, False, False, "exact"), (True, False, True, "exact"),
                                                       (False, False, True, "exact"), (False, True, False, "exact"),
                                                       (True, True, False, "exact"), (True, True, False, "order_free")])
def test_probabilities_of_a_small_step(akv_lib, B, H, G, D, P, append, packed, masked, mode):
    """Queries and keys of whole numbers: dot products are exact, and with them every rounding of a score.  Values that are unit vectors
    return the probabilities themselves; others are then held against the sum over these probabilities."""
    from alignedkv_b200.decode import DecodeLayer
    if mode == "order_free" and D != 128:
        pytest.skip("order-free P.V has head_dim 128")
    g = torch.Generator(device="cuda").manual_seed(1000 + P)
    whole = lambda *s: torch.randint(-3, 4, s, device="cuda", generator=g).half()  # noqa: E731
    n = P + int(append)
    k, q = whole(B, n, H, D), whole(B, 1, H * G, D)
    unit = torch.eye(n, D, device="cuda").half().view(1, n, 1, D).expand(B, n, H, D).contiguous()
    v = torch.randn(B, n, H, D, device="cuda", generator=g).half()
    mask = None
    if masked:
        mask = torch.zeros(B, 1, 1, n, device="cuda", dtype=torch.half)
        mask[0, :, :, :n // 2] = torch.finfo(torch.half).min
        mask[-1, :, :, n - 1] = 0.37

    def step(values):
        layer = DecodeLayer(B, 128, H, D, "cuda:0", n_q_heads=H * G, v_mode=mode)
        layer.prefill(k[:, :P].contiguous(), values[:, :P].contiguous())
        args = (q, k[:, P:].contiguous(), values[:, P:].contiguous()) if append else (q,)
        return layer.decode(*args, append=append, packed=packed, mask=mask).view(B, H * G, -1)

    dots = torch.einsum("bhd,bnhd->bhn", q[:, 0].double(), k.repeat_interleave(G, 2).double())
    s = (dots.half().float() / math.sqrt(D)).half()
    if masked:
        s = s + mask[:, 0]
    top = s.amax(-1, keepdim=True)
    e = torch.exp(s.double() - top.double())
    total = e.sum(-1, keepdim=True)
    exact = e / total
    one = step(unit)
    p = (one[..., 2:] if packed else one)[..., :n].double()
    # fp32 in front of the one rounding: the difference of two scores (up to 17.4, beyond that nothing is left: 2^-19.8), an
    # exponential (2 ulp), up to 64 additions and a quotient (2^-17)
    assert bool(((p - exact).abs() <= (2.0 ** -11 + 2.0 ** -16) * exact + 2.0 ** -25).all())
    if packed:
        assert torch.equal(one[..., 0], top[..., 0].float())
        assert bool(((one[..., 1].double() - total[..., 0]).abs() <= 2.0 ** -17 * total[..., 0]).all())
    got = step(v)
    got = (got[..., 2:] if packed else got).double()
    vd = v.repeat_interleave(G, 2).double()
    want, size = (torch.einsum("bhn,bnhd->bhd", p, t) for t in (vd, vd.abs()))
    # 64 fp32 additions, one rounding to fp16 (to 2^-25 at least; the order-free record stays in fp32)
    rounding = 0.0 if mode == "order_free" else 2.0 ** -11 * want.abs() + 2.0 ** -25
    assert bool(((got - want).abs() <= rounding + 65 * 2.0 ** -24 * size).all())
