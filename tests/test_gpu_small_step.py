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
