"""q.K^T in units of one 64-token block and of four, bit for bit against the oracle, and a decode step whose q.K^T makes its
alignment inputs itself (beside the append kernel) against the same step with launches that overlap nothing."""
import math

import numpy as np
import pytest
import torch

from helpers import exponent_field, k_planes_np, make_kvq
from test_gpu_ext import check, dev, stream, u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 4])
@pytest.mark.parametrize("B,H,G,D,nb", [(1, 1, 4, 128, 1), (2, 3, 4, 128, 5), (1, 8, 4, 256, 9), (1, 2, 8, 128, 3), (2, 4, 8, 128, 33),
                                        (1, 3, 8, 256, 2), (9, 8, 4, 128, 8), (1, 2, 4, 144, 7), (1, 2, 2, 128, 6)])
@pytest.mark.parametrize("reference", [False, True])
def test_forms(akv_lib, B, H, G, D, nb, tiles, reference):
    from oracle import akv_oracle as orc
    lib, Hq, L, nmb = akv_lib, H * G, nb * 64, nb + 1
    k, _, _ = make_kvq(81, B, L, H, D)
    _, _, q = make_kvq(82, B, 1, Hq, D)
    q = (q * 2.0 ** np.random.default_rng(83).integers(-7, 3, size=q.shape)).astype(np.float16)
    planes = k_planes_np(B, H, nmb, D)
    orc.k_cache_save(*planes, u8(k), B, H, nb, nmb, D, 64, 0, L)
    kexp = exponent_field(np.abs(k).max(axis=1, keepdims=True))
    kq = (exponent_field(q) + np.repeat(kexp, G, axis=2)).astype(np.uint8)
    kqmax = kq.max(axis=3, keepdims=True)
    rep = [np.ascontiguousarray(np.repeat(x, G, axis=1)) for x in planes]
    want, _ = orc.k_cache_compute(*rep, kq, kqmax, u8(q), B, Hq, nb, nmb, D, 64, L, 1 / math.sqrt(D), reference)
    dp, dkq, dkm, dq = [dev(x) for x in planes], dev(kq), dev(kqmax), dev(u8(q))
    s = torch.zeros((B, Hq, 1, (nb + 1) * 64), dtype=torch.half, device="cuda")
    assert lib.akv_set_tuning(b"k_tiles", tiles) == 0
    try:
        check(lib, lib.akv_k_cache_compute_gqa(dp[0].data_ptr(), dp[1].data_ptr(), dp[2].data_ptr(), dkq.data_ptr(),
                                               dkm.data_ptr(), dq.data_ptr(), s.data_ptr(), B, H, G, nb, nmb, D, 64, L,
                                               1 / math.sqrt(D), int(reference), stream()))
        torch.cuda.synchronize()
    finally:
        lib.akv_set_tuning(b"k_tiles", 0)
    got = s.cpu().numpy().view(np.uint16).reshape(B, Hq, -1)[..., :L]
    assert np.array_equal(got, want.view(np.uint16).reshape(B, Hq, -1)[..., :L])


@pytest.mark.parametrize("B,H,G,D,P,mode", [(1, 2, 1, 128, 64, "exact"), (3, 4, 1, 64, 100, "exact"), (2, 8, 4, 128, 700, "exact"),
                                            (1, 4, 8, 128, 190, "exact"), (2, 3, 2, 256, 130, "exact"),
                                            (1, 8, 1, 128, 1500, "order_free"), (2, 4, 4, 128, 600, "order_free"),
                                            (40, 8, 1, 128, 300, "exact")])
@pytest.mark.parametrize("append", [True, False])
def test_overlapped_steps(akv_lib, B, H, G, D, P, mode, append):
    """Steps that follow one another without a pause, one of them flushing a block, with and without overlapped launches."""
    from alignedkv_b200.decode import DecodeLayer
    g = torch.Generator(device="cuda").manual_seed(P)
    T = 66 - P % 64 if append and P % 64 else 4
    r = lambda n, h: torch.randn(n, B, 1, h, D, device="cuda", generator=g)  # noqa: E731
    k = torch.randn(B, P, H, D, device="cuda", generator=g)
    k[..., [3, 34]] *= 20
    k, v, q, k1, v1 = k.half(), torch.randn(B, P, H, D, device="cuda", generator=g).half(), r(T, H * G).half(), r(T, H) * 3, r(T, H).half()
    k1 = (k1 * torch.linspace(0.2, 9.0, T, device="cuda").view(T, 1, 1, 1, 1)).half()      # the maxima grow under way
    outs = []
    for pdl in (0, 1):
        assert akv_lib.akv_set_tuning(b"pdl", pdl) == 0
        try:
            layer = DecodeLayer(B, -(-(P + T) // 64) * 64, H, D, "cuda:0", n_q_heads=H * G, v_mode=mode)
            layer.prefill(k, v)
            o = [layer.decode(q[t], k1[t], v1[t]) if append else layer.decode(q[t], append=False) for t in range(T)]
            torch.cuda.synchronize()
        finally:
            akv_lib.akv_set_tuning(b"pdl", 1)
        outs.append(torch.stack(o + [layer.k_exp_max.float().mean().half().expand_as(o[0])]))
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert akv_lib.akv_device_error_flag() == 0


# rows of more than 17408 scores (few: the split softmax with P.V's first stages requested in front of its end; many: three passes
# and a probe of their own), a padded batch, a step that flushes among them
@pytest.mark.parametrize("B,H,G,P,T,mode,packed,masked", [(1, 3, 1, 17500, 4, "order_free", True, False),
                                                          (1, 3, 1, 17500, 38, "exact", False, False),
                                                          (2, 2, 4, 17470, 3, "exact", True, False),
                                                          (75, 1, 4, 24576, 2, "exact", False, False),
                                                          (75, 4, 1, 24570, 8, "order_free", True, False),
                                                          (5, 8, 4, 700, 6, "exact", False, True),
                                                          (3, 4, 1, 16440, 3, "exact", False, True)])
def test_overlapped_steps_leave_the_same(akv_lib, B, H, G, P, T, mode, packed, masked):
    """Everything that a run of steps returns and leaves behind, with and without overlapped launches."""
    from alignedkv_b200.decode import DecodeLayer
    D = 128
    g = torch.Generator(device="cuda").manual_seed(P + B)
    r = lambda *s: torch.randn(*s, D, device="cuda", generator=g).half()  # noqa: E731
    k, v, q, k1, v1 = r(B, P, H), r(B, P, H), r(T, B, 1, H * G), r(T, B, 1, H), r(T, B, 1, H)
    k[..., [3, 34]] *= 20
    k1 *= torch.linspace(0.2, 9.0, T, device="cuda").view(T, 1, 1, 1, 1)
    v1 *= torch.linspace(1.0, 30.0, T, device="cuda").view(T, 1, 1, 1, 1)                  # the maxima grow under way
    L = -(-(P + T) // 64) * 64
    mask = None
    if masked:
        mask = torch.zeros(B, 1, 1, L, device="cuda", dtype=torch.half)
        mask[0, ..., :P // 3] = torch.finfo(torch.half).min
    seen = []
    for pdl in (0, 1):
        assert akv_lib.akv_set_tuning(b"pdl", pdl) == 0
        try:
            layer = DecodeLayer(B, L, H, D, "cuda:0", n_q_heads=H * G, v_mode=mode)
            layer.prefill(k, v)
            out = [layer.decode(q[t], k1[t], v1[t], packed=packed, mask=mask) for t in range(T)]
            torch.cuda.synchronize()
        finally:
            akv_lib.akv_set_tuning(b"pdl", 1)
        n = layer.rest_len
        seen.append(out + [layer.restk[:, :n], layer.restv[:, :n], layer.k_exp_max, layer.v_exp_max, layer.k_first_8, layer.k_mid_4,
                           layer.k_last_4] + [t[:, :, :layer.rest_start] for t in (layer.v_first_8, layer.v_mid_4, layer.v_last_4)])
    for a, b in zip(*seen):
        assert torch.equal(a, b) and bool(a.count_nonzero() or not a.numel())
    assert akv_lib.akv_device_error_flag() == 0


@pytest.mark.parametrize("B,H,G,D,P", [(2, 3, 1, 128, 640), (1, 4, 1, 64, 192), (1, 2, 2, 128, 320), (2, 4, 4, 128, 3968), (40, 4, 4, 128, 1088),
                                       (1, 3, 4, 256, 64), (2, 2, 8, 128, 448), (1, 2, 1, 256, 320)])
@pytest.mark.parametrize("append", [True, False])
def test_own_alignment_inputs(akv_lib, B, H, G, D, P, append):
    """A step whose q.K^T makes its alignment inputs from query, exponent maxima and new token, against one that takes the append
    kernel's: K planes off a 16-byte boundary go to the kernel that has no form of its own for them."""
    from alignedkv_b200.decode import DecodeLayer
    g = torch.Generator(device="cuda").manual_seed(P + D)
    r = lambda *s: torch.randn(*s, D, device="cuda", generator=g)  # noqa: E731
    spread = 2.0 ** torch.randint(-7, 3, (H, D), device="cuda", generator=g)
    k, v, v1 = (r(B, P, H) * spread).half(), r(B, P, H).half(), r(B, 1, H).half()
    k1 = (r(B, 1, H) * spread * 2.0 ** torch.randint(-6, 7, (B, 1, H, D), device="cuda", generator=g)).half()   # some maxima are the token's
    q = (r(B, 1, H * G) * 2.0 ** torch.randint(-5, 3, (B, 1, H * G, D), device="cuda", generator=g)).half()
    outs = []
    for off in (0, 8):
        layer = DecodeLayer(B, P + 64, H, D, "cuda:0", n_q_heads=H * G)
        layer.prefill(k, v)
        if off:
            for name in ("k_first_8", "k_mid_4", "k_last_4"):
                t = getattr(layer, name)
                at = torch.empty(t.numel() + off, dtype=torch.uint8, device="cuda")[off:].view(t.shape)
                setattr(layer, name, at.copy_(t))
                assert at.data_ptr() % 16 == off
        o = layer.decode(q, k1, v1) if append else layer.decode(q, append=False)
        outs.append([o, layer.k_exp_max, layer.v_exp_max])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    assert bool(outs[0][0].count_nonzero())
