"""Exact P.V (the chain kernel) at the edges of its stages, its unit counts and its read codes, bit for bit against the
oracle.  A stage is 64 tokens, a ring up to 16 stages; one unit per SM up to 148 units, then two, then (one head per unit)
four; grouped queries take a unit per head while the heads fit one wave."""
import numpy as np
import pytest
import torch

from helpers import softmax_probs
from test_gpu_ext import check, dev, stream, u8, v_state

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("B,H,G,n,form", [
    (1, 4, 1, 1, 0), (1, 4, 1, 63, 0), (1, 4, 1, 64, 0), (1, 4, 1, 65, 0),       # fewer stages than helpers
    (2, 4, 1, 16 * 64 + 5, 0), (1, 4, 1, 40 * 64, 0),                            # ring wraps, with and without a tail
    (3, 52, 1, 321, 0),                                                          # 156 units: two per SM
    (10, 64, 1, 200, 0),                                                         # 640 units: four per SM, two rounds
    (2, 4, 2, 130, 0), (2, 4, 2, 130, 2), (40, 8, 2, 129, 0),                    # group of 2: unit per head, shared
    (1, 2, 4, 700, 0), (5, 16, 4, 300, 0), (5, 31, 4, 300, 0),                   # group of 4: per head, <= 148, > 148 units
    (1, 1, 8, 1000, 0), (6, 8, 8, 190, 0), (20, 8, 8, 190, 0),                   # group of 8: the same
    (1, 2, 8, 700, 2), (1, 1, 4, 65, 1),
])
@pytest.mark.parametrize("amin", [31, 9, 0])     # nothing flagged, a few tokens, every token
def test_exact_pv_edges(akv_lib, B, H, G, n, form, amin):
    from oracle import akv_oracle as orc
    lib, Hq, L = akv_lib, H * G, n + 64
    _, planes = v_state(61, B, H, n, L)
    pad = (-n) % 8
    p = softmax_probs(62, B, Hq, n, pad=pad)
    a = np.full((B, Hq, 1, 1), amin, np.uint8)
    a[0, 1] = max(amin - 1, 0)                   # the heads of a group decide differently
    want, _ = orc.v_cache_compute(*[np.ascontiguousarray(np.repeat(x, G, axis=1)) for x in planes], u8(p), a, B, Hq, L, D,
                                  n + pad, n, False)
    dp, ds, da = [dev(x) for x in planes], dev(u8(p)), dev(a)
    out = torch.empty((B, Hq, 1, D), dtype=torch.half, device="cuda")
    assert lib.akv_set_tuning(b"v_gqa_form", form) == 0
    try:
        check(lib, lib.akv_v_cache_compute_gqa(dp[0].data_ptr(), dp[1].data_ptr(), dp[2].data_ptr(), ds.data_ptr(),
                                               da.data_ptr(), out.data_ptr(), None, 0, B, H, G, L, D, n + pad, n, 0, stream()))
        torch.cuda.synchronize()
    finally:
        lib.akv_set_tuning(b"v_gqa_form", 0)
    assert np.array_equal(out.cpu().numpy().view(np.uint16).reshape(B, Hq, D), want.view(np.uint16).reshape(B, Hq, D))
    assert lib.akv_device_error_flag() == 0


def test_exact_pv_group_of_eight_all_planes(akv_lib):
    """reference mode with eight heads per KV head runs the same kernel with every token reading every plane."""
    from oracle import akv_oracle as orc
    B, H, G, n, L = 2, 2, 8, 333, 384
    _, planes = v_state(63, B, H, n, L)
    pad = (-n) % 8
    p = softmax_probs(64, B, H * G, n, pad=pad)
    a = np.full((B, H * G, 1, 1), 20, np.uint8)
    want, _ = orc.v_cache_compute(*[np.ascontiguousarray(np.repeat(x, G, axis=1)) for x in planes], u8(p), a, B, H * G, L, D,
                                  n + pad, n, True)
    dp, ds, da = [dev(x) for x in planes], dev(u8(p)), dev(a)
    out = torch.empty((B, H * G, 1, D), dtype=torch.half, device="cuda")
    check(akv_lib, akv_lib.akv_v_cache_compute_gqa(dp[0].data_ptr(), dp[1].data_ptr(), dp[2].data_ptr(), ds.data_ptr(),
                                                   da.data_ptr(), out.data_ptr(), None, 0, B, H, G, L, D, n + pad, n, 1, stream()))
    got = out.cpu().numpy().view(np.uint16).reshape(B, H * G, D)
    assert np.array_equal(got, want.view(np.uint16).reshape(B, H * G, D))


@pytest.mark.parametrize("B,H,G", [(10, 64, 1), (80, 4, 2), (80, 4, 4), (80, 4, 8)])    # 640 units of one head, 320 of several
def test_thresholds_of_every_round(akv_lib, B, H, G):
    """A decode step with more units than fit at once: the threshold bytes that the kernel derives for the units of its second
    round too, against the rule in integers, and the outputs against the operator with those bytes given."""
    from alignedkv_b200.decode import DecodeLayer
    Hq, n = H * G, 192
    rows, R = B * Hq, n + 64
    g = torch.Generator(device="cuda").manual_seed(B * H)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).half()  # noqa: E731
    layer = DecodeLayer(B, R, H, D, "cuda:0", n_q_heads=Hq)
    v = rnd(B, n, H, D) * torch.exp2(torch.randint(-6, 4, (B, 1, H, 1), device="cuda", generator=g).float()).half()
    layer.prefill(rnd(B, n, H, D), v)
    got = layer.decode(rnd(B, 1, Hq, D), append=False)
    at = {x: layer._scratch_offset(x) for x in ("test_o", "amin")}
    p = layer.scratch[:rows * R * 2].view(torch.half)
    amin = layer.scratch[at["amin"]:at["amin"] + rows].clone()
    exps = (layer.scratch[at["test_o"]:at["test_o"] + rows * D * 2].view(torch.int16).view(rows, D).to(torch.int32) >> 10) & 0x1E
    v_exp = layer.v_exp_max.view(B, H, D).repeat_interleave(G, 1).view(rows, D).to(torch.int32)
    # row b * Hq + h of the reference's [B, Hq, Hq] broadcast, read flat (extension/v_cache_file.py:142,156-160)
    i = torch.arange(rows, device="cuda")
    bb, hp, he = i // (Hq * Hq), i // Hq % Hq, i % Hq
    want = ((exps[bb * Hq + hp] + 15 - v_exp[bb * Hq + he]) & 0xFF).amin(dim=1).to(torch.uint8)
    assert torch.equal(amin, want)
    assert len(torch.unique(want)) > 2                       # (otherwise a wrong row's byte would pass)
    o = torch.empty_like(got)
    check(akv_lib, akv_lib.akv_v_cache_compute_gqa(layer.v_first_8.data_ptr(), layer.v_mid_4.data_ptr(), layer.v_last_4.data_ptr(),
                                                   p.data_ptr(), want.data_ptr(), o.data_ptr(), None, 0, B, H, G, R, D, R, n, 0,
                                                   stream()))
    assert torch.equal(got.view(torch.int16), o.view(torch.int16))
    assert akv_lib.akv_device_error_flag() == 0
