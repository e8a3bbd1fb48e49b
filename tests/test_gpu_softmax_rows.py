"""The softmax of a decode step at the row lengths where it changes form (thread counts and vectors per thread at 2048,
4096, 8192, 12288 scores, split and three-pass forms beyond): probabilities against float64 on the same scores, the
probe's class maxima against the probabilities."""
import math

import numpy as np
import pytest
import torch

from test_gpu_ext import check, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,G,D,qn,masked", [
    (1, 4, 1, 128, 64, False), (2, 4, 1, 128, 1984, True), (1, 4, 1, 128, 2048, False), (1, 2, 4, 128, 4032, False),
    (1, 4, 1, 128, 4096, True), (1, 4, 1, 128, 8128, False), (1, 4, 1, 128, 8192, False), (1, 4, 1, 128, 12224, False),
    (1, 4, 1, 128, 12288, True), (1, 4, 1, 128, 17344, False),               # 17408 scores: the longest unsplit row when few
    (1, 4, 1, 128, 17408, False),                                            # split across CTAs
    (75, 1, 4, 128, 24512, False), (75, 1, 4, 128, 24576, False),            # many rows: last one-CTA row, three passes
    (2, 4, 1, 64, 320, False), (1, 4, 1, 256, 320, True), (1, 4, 1, 512, 192, False),
])
def test_probabilities(akv_lib, B, H, G, D, qn, masked):
    from alignedkv_b200.decode import DecodeLayer
    Hq, R = H * G, qn + 64
    g = torch.Generator(device="cuda").manual_seed(qn + D)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).half()  # noqa: E731
    layer = DecodeLayer(B, qn + 64, H, D, "cuda:0", n_q_heads=Hq)
    layer.prefill(rnd(B, qn, H, D), rnd(B, qn, H, D))
    q = 3 * rnd(B, 1, Hq, D)
    mask = None
    if masked:
        mask = torch.zeros(B, 1, 1, R, device="cuda", dtype=torch.half)
        mask[..., :qn // 3] = -1.5
        mask[..., :7] = torch.finfo(torch.half).min
    layer.decode(q, append=False, mask=mask)
    at = {n: layer._scratch_offset(n) for n in ("kq", "kqmax", "pval", "pidx")}
    rows = B * Hq
    p = layer.scratch[:rows * R * 2].view(torch.half).view(rows, R).clone()
    s = torch.zeros(rows, R, dtype=torch.half, device="cuda")
    check(akv_lib, akv_lib.akv_k_cache_compute_gqa(
        layer.k_first_8.data_ptr(), layer.k_mid_4.data_ptr(), layer.k_last_4.data_ptr(), layer.scratch[at["kq"]:].data_ptr(),
        layer.scratch[at["kqmax"]:].data_ptr(), q.data_ptr(), s.data_ptr(), B, H, G, qn // 64, (qn + 64) // 64, D, 64, qn,
        1 / math.sqrt(D), 0, stream()))
    s = s[:, :qn]
    if masked:
        s = (s.view(B, Hq, qn) + mask[:, 0, :, :qn]).view(rows, qn)
    want = torch.softmax(s.double(), 1)
    # a probability is off by half an fp16 step (2^-11 relative, 2^-25 absolute below the normal range) plus the fp32
    # exponential, sum and division (a few 2^-24 relative)
    assert ((p[:, :qn].double() - want).abs() <= want * (2 ** -11 + 2 ** -20) + 2 ** -25).all()
    assert (p[:, qn:] == 0).all()
    classes = p[:, :qn].view(rows, qn // 32, 32).cpu().float().numpy()
    top, first = classes.max(axis=1), classes.argmax(axis=1)                 # (argmax: the first maximum)
    pval = layer.scratch[at["pval"]:at["pval"] + rows * 64].view(torch.half).view(rows, 32).cpu().float().numpy()
    pidx = layer.scratch[at["pidx"]:at["pidx"] + rows * 128].view(torch.int32).view(rows, 32).cpu().numpy()
    assert np.array_equal(pval, top) and np.array_equal(pidx, first)
