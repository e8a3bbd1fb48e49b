"""akv_prefill for head_dim 128 at the edges of its 64-token tiles against the operator-by-operator route, on planes that
already hold something (K nibbles are added onto them) and exponent tensors at odd addresses."""
import pytest
import torch

from test_gpu_ext import check, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 63, 64, 65, 127, 128, 1000])
@pytest.mark.parametrize("special", [False, True])
def test_prefill128(akv_lib, S, special):
    lib, (B, H, D, L) = akv_lib, (2, 3, 128, 1088)
    g = torch.Generator(device="cuda").manual_seed(S)
    k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).half() for _ in range(2))
    if special:      # infinities, NaNs, zeros of both signs, all-negative channels: bytes are bytes, and the maximum skips NaN
        for t in (k, v):
            flat = t.view(-1)
            flat[::37], flat[1::41], flat[2::43], flat[3::47] = float("inf"), float("-inf"), float("nan"), -0.0
            t[:, :, 1, 7] = -t[:, :, 1, 7].nan_to_num(1.0, 1.0, 1.0).abs()
    rnd = lambda *shape: torch.randint(0, 256, shape, device="cuda", dtype=torch.uint8, generator=g)  # noqa: E731
    planes = [rnd(B, H, L // 64, D, 64), rnd(B, H, L // 64, D, 32), rnd(B, H, L // 64, D, 32),
              rnd(B, H, L, D), rnd(B, H, L, D // 2), rnd(B, H, L, D // 2)]
    want = [x.clone() for x in planes]
    rest = [torch.zeros(B, 64, H, D, dtype=torch.half, device="cuda") for _ in range(2)]
    exps = [torch.zeros(B * H * D + 1, dtype=torch.uint8, device="cuda")[1:] for _ in range(2)]
    ws = torch.empty(lib.akv_prefill_scratch_bytes(B, H, D, S), dtype=torch.uint8, device="cuda")
    check(lib, lib.akv_prefill(*[x.data_ptr() for x in planes], exps[0].data_ptr(), exps[1].data_ptr(), rest[0].data_ptr(),
                               rest[1].data_ptr(), k.data_ptr(), v.data_ptr(), ws.data_ptr(), ws.numel(), B, H, D, L, S, stream()))
    full = S // 64 * 64
    check(lib, lib.akv_k_cache_save(*[x.data_ptr() for x in want[:3]], k.data_ptr(), B, H, S // 64, L // 64, D, 64, 0, S, stream()))
    if full:
        first = v[:, :full].contiguous()
        check(lib, lib.akv_v_cache_save(*[x.data_ptr() for x in want[3:]], first.data_ptr(), B, H, L, D, 0, full, full, stream()))
    for got, ref in zip(planes, want):
        assert torch.equal(got, ref)
    for got, src in zip(rest, (k, v)):
        assert torch.equal(got[:, :S - full].contiguous().view(torch.int16), src[:, full:].contiguous().view(torch.int16))
    for got, src in zip(exps, (k, v)):
        top = torch.where(src.isnan(), float("-inf"), src.float()).amax(dim=1).half()
        assert torch.equal(got.view(B, H, D), ((top.view(torch.int16) >> 10) & 0x1F).to(torch.uint8))
