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
