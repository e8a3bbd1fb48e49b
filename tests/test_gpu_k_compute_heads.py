"""q.K^T where a warp goes from one (batch, KV head) to the next - its tables and plane masks change under way - bit for bit
against the oracle: few blocks per head and many heads per warp, at every group size, head sizes from 64 to 256, ring depths
from 3 to 5.  Queries are scaled by powers of two per (head, channel), so that neighbouring heads read different planes."""
import math

import numpy as np
import pytest
import torch

from helpers import exponent_field, k_planes_np, make_kvq
from test_gpu_ext import check, dev, stream, u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,G,D,nb,stages,wpc", [
    # one warp per SM: 320 (batch, KV head) pairs are 3 units (or, from five blocks on, 5) for each of 148 warps
    *[(40, 8, 1, 64, nb, stages, 1) for nb in (1, 3, 4, 5) for stages in (3, 4, 5)],
    (40, 8, 1, 128, 1, 3, 1), (40, 8, 1, 128, 5, 5, 1), (40, 8, 1, 80, 3, 5, 1), (40, 8, 1, 256, 3, 3, 1),
    (80, 4, 2, 64, 1, 3, 1), (80, 4, 2, 128, 5, 3, 1), (80, 4, 2, 192, 3, 3, 1),
    (80, 4, 4, 64, 3, 3, 1), (80, 4, 4, 128, 5, 3, 1), (80, 4, 4, 256, 1, 3, 1),
    (80, 4, 8, 64, 1, 3, 1), (80, 4, 8, 128, 3, 3, 1), (80, 4, 8, 256, 1, 3, 1),
    # as many warps as fit
    (94, 32, 1, 64, 1, 5, 0), (94, 32, 1, 64, 1, 3, 0), (160, 16, 1, 128, 1, 3, 0), (160, 16, 4, 64, 1, 3, 0),
])
@pytest.mark.parametrize("reference", [False, True])
def test_heads_of_a_warp(akv_lib, B, H, G, D, nb, stages, wpc, reference):
    from oracle import akv_oracle as orc
    lib, Hq, L = akv_lib, H * G, nb * 64
    k, _, _ = make_kvq(71, B, L, H, D)
    _, _, q = make_kvq(72, B, 1, Hq, D)
    q = (q * 2.0 ** np.random.default_rng(73).integers(-7, 3, size=q.shape)).astype(np.float16)
    planes = k_planes_np(B, H, nb, D)
    orc.k_cache_save(*planes, u8(k), B, H, nb, nb, D, 64, 0, L)
    kexp = exponent_field(np.abs(k).max(axis=1, keepdims=True))
    kq = (exponent_field(q) + np.repeat(kexp, G, axis=2)).astype(np.uint8)
    kqmax = kq.max(axis=3, keepdims=True)
    rep = [np.ascontiguousarray(np.repeat(x, G, axis=1)) for x in planes]
    want, _ = orc.k_cache_compute(*rep, kq, kqmax, u8(q), B, Hq, nb, nb, D, 64, L, 1 / math.sqrt(D), reference)
    dp, dkq, dkm, dq = [dev(x) for x in planes], dev(kq), dev(kqmax), dev(u8(q))
    s = torch.zeros((B, Hq, 1, (nb + 1) * 64), dtype=torch.half, device="cuda")
    assert lib.akv_set_tuning(b"k_stages", stages) == 0 and lib.akv_set_tuning(b"k_wpc", wpc) == 0
    try:
        check(lib, lib.akv_k_cache_compute_gqa(dp[0].data_ptr(), dp[1].data_ptr(), dp[2].data_ptr(), dkq.data_ptr(),
                                               dkm.data_ptr(), dq.data_ptr(), s.data_ptr(), B, H, G, nb, nb, D, 64, L,
                                               1 / math.sqrt(D), int(reference), stream()))
        torch.cuda.synchronize()
    finally:
        lib.akv_set_tuning(b"k_stages", 3)
        lib.akv_set_tuning(b"k_wpc", 0)
    got = s.cpu().numpy().view(np.uint16).reshape(B, Hq, -1)[..., :L]
    assert np.array_equal(got, want.view(np.uint16).reshape(B, Hq, -1)[..., :L])
