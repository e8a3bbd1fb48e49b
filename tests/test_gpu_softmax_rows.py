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


def _added_in_columns(e, cols):
    """Sums of fp32 rows in the order of the decode step's softmax: column t % cols takes its values in order, the columns of
    a warp are added as an xor tree, the warps in order."""
    rows, n = e.shape
    e = torch.nn.functional.pad(e, (0, -n % cols)).view(rows, -1, cols)
    x = torch.zeros(rows, cols, device=e.device)
    for k in range(e.shape[1]):
        x = x + e[:, k]
    x, lane = x.view(rows, cols // 32, 32), torch.arange(32, device=e.device)
    for o in (16, 8, 4, 2, 1):
        x = x + x[..., lane ^ o]
    total = torch.zeros(rows, device=e.device)
    for w in range(cols // 32):
        total = total + x[:, w, 0]
    return total


# (rows of at most 12288 scores in 256 and 512 threads, longer ones in 1024; few rows, and more than four per SM)
@pytest.mark.parametrize("B,H,G,qn", [
    (1, 4, 1, 0), (1, 4, 1, 448), (1, 4, 1, 1984), (1, 4, 1, 3968), (1, 4, 1, 8128), (1, 4, 1, 8192), (1, 4, 1, 12224),
    (1, 4, 1, 12288), (1, 4, 1, 17344), (75, 2, 4, 0), (75, 2, 4, 1024), (75, 2, 4, 4032), (75, 1, 4, 4096), (75, 1, 4, 10176),
    (75, 1, 4, 10240), (75, 1, 4, 12288), (75, 1, 4, 24512), (75, 1, 4, 24576),
])
def test_sum_of_exponentials(akv_lib, B, H, G, qn):
    """The order in which a row's exponentials are added is part of the result - through a model's layers one step of an fp16
    probability moves its logits - and does not depend on the form that runs: 256 columns, 512 for few rows of 8193 to 17408
    scores, whatever the threads hold.  Bit for bit, residual tokens (scores exactly 0) among them."""
    from alignedkv_b200.decode import DecodeLayer
    D, rest = 128, 7
    Hq, n, rows = H * G, qn + rest, B * H * G
    g = torch.Generator(device="cuda").manual_seed(qn + B)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).half()  # noqa: E731
    layer = DecodeLayer(B, qn + 64, H, D, "cuda:0", n_q_heads=Hq, v_mode="order_free")
    k = rnd(B, n, H, D)
    k[:, qn:] = 0
    layer.prefill(k, rnd(B, n, H, D))
    q = rnd(B, 1, Hq, D)
    rec = layer.decode(q, append=False, packed=True)
    at = {x: layer._scratch_offset(x) for x in ("kq", "kqmax")}
    s = torch.zeros(rows, qn + 64, dtype=torch.half, device="cuda")
    if qn:
        check(akv_lib, akv_lib.akv_k_cache_compute_gqa(
            layer.k_first_8.data_ptr(), layer.k_mid_4.data_ptr(), layer.k_last_4.data_ptr(), layer.scratch[at["kq"]:].data_ptr(),
            layer.scratch[at["kqmax"]:].data_ptr(), q.data_ptr(), s.data_ptr(), B, H, G, qn // 64, (qn + 127) // 64, D, 64, qn,
            1 / math.sqrt(D), 0, stream()))
    s = s[:, :n].float()
    m = s.amax(dim=1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cols = 512 if 8192 < qn + 64 <= 17408 and rows <= 2 * sms else 256
    assert torch.equal(rec[:, 0], m)
    assert torch.equal(rec[:, 1], _added_in_columns(torch.exp(s - m[:, None]), cols))


@pytest.mark.parametrize("B,H,G,qn,rest,masked", [
    (75, 1, 4, 2048, 1, False), (75, 1, 4, 4032, 7, True), (75, 1, 4, 4096, 63, False), (75, 1, 4, 10176, 8, True),
    (75, 1, 4, 10240, 7, False), (75, 1, 4, 12288, 63, True), (75, 1, 4, 24512, 8, False), (75, 1, 4, 24576, 1, False),
    (75, 2, 4, 1024, 63, False), (75, 2, 4, 8192, 7, False), (75, 2, 4, 0, 29, False), (2, 4, 1, 640, 63, True),
    (5, 2, 8, 320, 63, False), (5, 4, 2, 320, 29, False), (1, 4, 1, 4096, 8, False), (1, 4, 1, 8192, 7, True), (1, 4, 1, 17344, 63, False),
])
def test_residual_tokens(akv_lib, B, H, G, qn, rest, masked):
    """A step with residual tokens, at every form: their probabilities against float64, and the output bit for bit from the
    step's own probabilities: the exact P.V operator over the quantized tokens, the residual tokens in fp32 by shares of
    every third token (few rows, groups of up to four) or every fourth, each rounded to fp16 before they are added."""
    from alignedkv_b200.decode import DecodeLayer
    D = 128
    Hq, n, rows, R = H * G, qn + rest, B * H * G, qn + 64
    g = torch.Generator(device="cuda").manual_seed(qn + rest)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).half()  # noqa: E731
    layer = DecodeLayer(B, R, H, D, "cuda:0", n_q_heads=Hq)
    k, v = rnd(B, n, H, D), rnd(B, n, H, D)
    k[:, qn:] *= 4                                       # (the residual tokens take their part)
    layer.prefill(k, v)
    q = rnd(B, 1, Hq, D)
    mask = None
    if masked:
        mask = torch.zeros(B, 1, 1, R, device="cuda", dtype=torch.half)
        mask[..., :qn // 3] = -1.5
        mask[..., n - 1] = torch.finfo(torch.half).min
    got = layer.decode(q, append=False, mask=mask).view(rows, D)
    at = {x: layer._scratch_offset(x) for x in ("kq", "kqmax", "amin")}
    p = layer.scratch[:rows * R * 2].view(torch.half).view(rows, R).clone()
    s = torch.zeros(rows, R, dtype=torch.half, device="cuda")
    if qn:
        check(akv_lib, akv_lib.akv_k_cache_compute_gqa(
            layer.k_first_8.data_ptr(), layer.k_mid_4.data_ptr(), layer.k_last_4.data_ptr(), layer.scratch[at["kq"]:].data_ptr(),
            layer.scratch[at["kqmax"]:].data_ptr(), q.data_ptr(), s.data_ptr(), B, H, G, qn // 64, (R + 63) // 64, D, 64, qn,
            1 / math.sqrt(D), 0, stream()))
    kr = k[:, qn:].double().repeat_interleave(G, 2)                                          # [B, rest, Hq, D]
    sr = torch.einsum("bhd,brhd->bhr", q[:, 0].double(), kr).view(rows, rest) / math.sqrt(D)
    x = torch.cat([s[:, :qn].double(), sr], 1)
    if masked:
        x = (x.view(B, Hq, n) + mask[:, 0, :, :n].double()).view(rows, n)
    want = torch.softmax(x, 1)
    # a residual (or masked) score is rounded to fp16 up to three times, half a step of 2^-10 relative each: exponents are
    # off by up to d = 3 * 2^-11 * |score|, numerator and sum each by a factor of e^d, and e^(2d) - 1 <= 2.2 d below d = 0.09
    off = 3 * 2 ** -11 * torch.where(x < -1e4, 0.0, x).abs().amax(dim=1, keepdim=True)
    assert off.max() < 0.09
    assert ((p[:, :n].double() - want).abs() <= want * (2.2 * off + 2 ** -11 + 2 ** -20) + 2 ** -25).all()
    assert (p[:, n:] == 0).all()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shares = 3 if qn > 0 and G <= 4 and rows <= (4 if R <= 8192 else 2 if R <= 17408 else 0) * sms else 4
    pr, vr = p[:, qn:n].float(), v[:, qn:].float().repeat_interleave(G, 2).transpose(1, 2).reshape(rows, rest, D)
    part = torch.zeros(shares, rows, D, device="cuda")
    for r in range(rest):                                # (the product of two fp16 values is exact in fp32)
        part[r % shares] = part[r % shares] + pr[:, r:r + 1] * vr[:, r]
    res = part[0]
    for j in range(1, shares):
        res = res + part[j]
    o = torch.zeros(rows, D, dtype=torch.half, device="cuda")
    if qn:
        check(akv_lib, akv_lib.akv_v_cache_compute_gqa(
            layer.v_first_8.data_ptr(), layer.v_mid_4.data_ptr(), layer.v_last_4.data_ptr(), p.data_ptr(),
            layer.scratch[at["amin"]:].data_ptr(), o.data_ptr(), None, 0, B, H, G, R, D, R, qn, 0, stream()))
    assert torch.equal(got.view(torch.int16), (o.float() + res.half().float()).half().view(torch.int16))


def test_long_rows_on_two_threads(akv_lib):
    """Caches of different lengths on two host threads, each with its own stream: rows of 17408 and of 12352 scores, whose
    softmax asks for different amounts of shared memory of one kernel.  Every call succeeds and repeats its result."""
    import threading

    from alignedkv_b200.decode import DecodeLayer
    from alignedkv_b200 import _lib
    _lib.load()
    failed = []

    def work(qn):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                g = torch.Generator(device="cuda").manual_seed(qn)
                rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).half()  # noqa: E731
                layer = DecodeLayer(1, qn + 64, 1, 128, "cuda:0")
                layer.prefill(rnd(1, qn, 1, 128), rnd(1, qn, 1, 128))
                q = rnd(1, 1, 1, 128)
                first = layer.decode(q, append=False).clone()
                out = torch.empty_like(first)
                for _ in range(3000):
                    layer.decode(q, append=False, out=out)
                torch.cuda.current_stream().synchronize()
                if not torch.equal(out, first):
                    failed.append(f"{qn}: another result")
        except Exception as e:  # noqa: BLE001
            failed.append(f"{qn}: {e}")

    threads = [threading.Thread(target=work, args=(qn,)) for qn in (17344, 12288)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
